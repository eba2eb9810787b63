"""Which evaluations sort their poses first: many points near many protein atoms, and enough ligand atoms to a
pose.  Sorted, an evaluation of a deck makes five launches instead of three; its energies are the same."""
import numpy as np
import pytest

from minibude_gb300.deck import BatchDeck, DeckSpec, synthetic_deck, synthetic_poses
from minibude_gb300.model import GpuContext

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("natpro,natlig,nposes,sorts", [(400, 8, 131072, True), (400, 8, 65536, False),
                                                        (140, 2, 1_500_000, False), (400, 2, 300_000, True)])
def test_deck_and_batch(built_library, natpro, natlig, nposes, sorts):
    box = 0.5 * (natpro / 0.05) ** (1 / 3)
    deck = synthetic_deck(DeckSpec("order", natpro, box, natlig, 34, 64), seed=1)
    some = 50000
    tile = synthetic_poses(np.random.default_rng(1), some)
    deck.poses = np.ascontiguousarray(np.tile(tile, -(-nposes // some))[:, :nposes])
    with GpuContext(0) as c:
        c.upload(deck)
        cfg = c.default_cfg(8, 512)
        before = c.launch_count()
        c.run(cfg)
        assert c.launch_count() - before == (5 if sorts else 3)
        got = c.download()
        assert np.array_equal(got, np.tile(got[:some], -(-nposes // some))[:nposes])
        # The same, whole, as a batch of one ligand, whose own line lies elsewhere.
        c.upload_batch(BatchDeck(deck.protein, deck.forcefield, [deck.ligand], [deck.poses], "order"))
        c.run_batch(cfg)
        assert np.array_equal(c.download_batch(), got)
        c.run_batch(cfg, per_ligand=True)
        assert np.array_equal(c.download_batch(), got)
