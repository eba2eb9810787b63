"""An evaluation that has no room for its poses' order or for all of its atom sums does without the one and takes
the other in windows: the energies are those of a device with room.  The rest of the memory is taken up by
a buffer that nothing writes."""
import numpy as np
import pytest

from minibude_gb300.capi import BudeError
from minibude_gb300.deck import BatchDeck, DeckSpec, synthetic_deck, synthetic_ligand, synthetic_poses
from minibude_gb300.model import GpuContext

pytestmark = pytest.mark.gpu

MB = 1 << 20
DECK = DeckSpec("memory", 300, 9.0, 24, 12, 64)
NTILE = 62500


def leave(nbytes):
    """Take up the device memory but for nbytes."""
    import torch
    free, _ = torch.cuda.mem_get_info()
    return torch.empty(free - nbytes, dtype=torch.uint8, device="cuda")


def free_bytes():
    import torch
    return torch.cuda.mem_get_info()[0]


def give_back(held):
    import torch
    del held[:]
    torch.cuda.empty_cache()


def test_batch(built_library):
    deck = synthetic_deck(DECK, seed=1)
    rng = np.random.default_rng(2)
    tile = synthetic_poses(rng, NTILE)
    n, per = 8, np.ascontiguousarray(np.tile(tile, 6))  # 8 ligands of 375,000 poses
    ligands = [synthetic_ligand(rng, 24, 5.0, 12) for _ in range(n)]
    batch = BatchDeck(deck.protein, deck.forcefield, ligands, [per] * n, "memory")
    total = batch.total_poses
    with GpuContext(0) as roomy, GpuContext(0) as tight:
        cfg = roomy.default_cfg(8, 512)
        roomy.upload_batch(batch)
        roomy.run_batch(cfg)
        want = roomy.download_batch()
        tight.default_cfg(8, 512)
        held = [leave(76 * total + 110 * MB)]  # the order takes 56 bytes a pose, the sums 96
        try:
            tight.upload_batch(batch)
            assert free_bytes() < 56 * total
            tight.run_batch(cfg)
            got = tight.download_batch()
        finally:
            give_back(held)
    assert np.array_equal(got, want)


def test_deck(built_library):
    deck = synthetic_deck(DECK, seed=1)
    deck.poses = np.ascontiguousarray(np.tile(synthetic_poses(np.random.default_rng(3), NTILE), 64))
    n = deck.nposes
    with GpuContext(0) as roomy, GpuContext(0) as tight:
        want = roomy.energies(deck)
        held = [leave(77 * n + 24 * MB)]  # the order takes 8 bytes a pose, the sums 96
        try:
            tight.upload(deck)
            assert free_bytes() < 8 * n
            tight.run(tight.default_cfg(0, 0))
            got = tight.download()
        finally:
            give_back(held)
    assert np.array_equal(got, want)


def test_poses_that_do_not_fit_leave_no_deck(built_library):
    deck = synthetic_deck(DECK, seed=1)
    many = np.zeros((6, 4_000_000), np.float32)
    with GpuContext(0) as c:
        want = c.energies(deck)
        cfg = c.default_cfg(0, 0)
        held = [leave(64 * MB)]  # 76 bytes a pose are asked for
        try:
            with pytest.raises(BudeError, match="out of memory"):
                c.set_poses(many)
            for call in (lambda: c.run(cfg), lambda: c.set_poses(deck.poses), c.download):
                with pytest.raises(BudeError, match="no deck"):
                    call()
            assert np.array_equal(c.energies(deck), want)
        finally:
            give_back(held)
        assert np.array_equal(c.energies(deck), want)
