"""Many poses against a protein of a few dozen atoms have every pair evaluated (csrc/direct_kernel.cuh).  The
energies are the bits of the culled kernel, which takes the same poses in pieces of fewer than 16,384; the
oracle bounds both.  Sizes lie on both sides of the rule's line (64 atoms, up to 128 for ligands of few)."""
import numpy as np
import pytest

import oracle
from minibude_gb300 import validate
from minibude_gb300.deck import BatchDeck, DeckSpec, synthetic_deck, synthetic_ligand, synthetic_poses
from minibude_gb300.model import GpuContext, launch_cfg

pytestmark = pytest.mark.gpu

SHAPES = [(1, 32), (1, 512), (2, 96), (4, 128), (4, 512), (8, 64), (16, 512)]


@pytest.fixture(scope="module")
def ctx(built_library):
    c = GpuContext(0)
    yield c
    c.close()


def deck_of(natpro, natlig, nposes, half_box=None, seed=0):
    box = half_box or 0.5 * (natpro / 0.05) ** (1 / 3)
    return synthetic_deck(DeckSpec("direct", natpro, box, natlig, 12, nposes), seed=seed)


def in_pieces(ctx, deck, piece=16000):
    """The energies of the uploaded deck's poses, in sets too small for direct_kernel."""
    out = []
    for p in range(0, deck.nposes, piece):
        ctx.set_poses(np.ascontiguousarray(deck.poses[:, p:p + piece]))
        ctx.run(ctx.default_cfg(0, 0))
        out.append(ctx.download())
    return np.concatenate(out)


def assert_parity(got, deck, n=512):
    head = synthetic_like(deck, n)
    e32, e64 = oracle.fasten_f32(head), oracle.fasten_f64(head)
    scale = np.maximum(np.abs(e64), 1.0)
    bound = max(2e-4, 4 * float((np.abs(e32 - e64) / scale).max()))
    max_diff, failed = validate(got[:n], e32)
    assert not failed and max_diff < 0.025, (max_diff, failed[:5])
    assert float((np.abs(got[:n] - e64) / scale).max()) < bound


def synthetic_like(deck, n):
    import dataclasses
    return dataclasses.replace(deck, poses=np.ascontiguousarray(deck.poses[:, :n]))


@pytest.mark.parametrize("natpro,natlig,nposes,half_box", [
    (1, 1, 16384, None), (1, 3, 16383, None), (8, 5, 20001, 1.0), (15, 2, 16384, None), (16, 26, 16385, None),
    (31, 4, 64 * 31 * 31, None), (32, 0, 70000, None), (32, 2, 65535, None), (32, 33, 65536, 2.0), (33, 1, 70001, None),
    (64, 3, 262143, None), (64, 2, 262144, 3.0), (65, 2, 300000, None), (128, 1, 1 << 20, None), (128, 4, 1 << 20, None),
    (96, 8, 589823, None), (96, 8, 589824, None), (96, 9, 589824, None)])
def test_sizes_around_the_line(ctx, natpro, natlig, nposes, half_box):
    deck = deck_of(natpro, natlig, nposes, half_box, seed=natpro)
    ctx.upload(deck)
    want = in_pieces(ctx, deck)
    ctx.upload(deck)
    for p, w in [(0, 0)] + SHAPES:
        ctx.run(ctx.default_cfg(p, w))
        assert np.array_equal(ctx.download(), want), (p, w)
    for u in (1, 2, 4):
        ctx.run(launch_cfg(2, 64, 1, 64, u))
        assert np.array_equal(ctx.download(), want), u
    out = np.empty(nposes, np.float32)
    for chunk in (1, 50000, 1 << 20):
        ctx.score_stream(ctx.default_cfg(4, 128), deck.poses, out, chunk=chunk)
        assert np.array_equal(out, want), chunk
    assert_parity(want, deck)


def test_the_pieces_take_the_other_kernel(ctx):
    """Above the line two launches (transforms, direct_kernel), below it three or more."""
    deck = deck_of(8, 4, 16384)
    ctx.upload(deck)
    for n, direct in ((16384, True), (16383, False)):
        ctx.set_poses(np.ascontiguousarray(deck.poses[:, :n]))
        before = ctx.launch_count()
        ctx.run(ctx.default_cfg(0, 0))
        assert (ctx.launch_count() - before == 2) == direct


def test_irregular_poses_and_decks(ctx):
    deck = deck_of(20, 6, 30001)
    rng = np.random.default_rng(1)
    for k, v in enumerate((np.nan, np.inf, -np.inf, 1e30, 3e11)):
        deck.poses[rng.integers(0, 6, 7), rng.integers(0, 30001, 7)] = v
        deck.poses[3 + k % 3, 31 + k] = v
    deck.poses[4, [0, 30000]] = np.nan
    wide = deck_of(20, 6, 30001)
    wide.forcefield["radius"][:] = 0.0  # every radius sum is 0: an irregular deck
    for d in (deck, wide):
        ctx.upload(d)
        want = in_pieces(ctx, d)
        ctx.upload(d)
        for p, w in SHAPES:
            ctx.run(ctx.default_cfg(p, w))
            assert np.array_equal(ctx.download(), want, equal_nan=True), (p, w)
    assert not np.isfinite(want).all() or d is wide


@pytest.mark.parametrize("natpro,counts", [(8, (1, 0, 30000, 257, 5000, 4096)), (32, (100000, 1, 40000, 33)),
                                           (20, (127, 128, 129) * 140)])
def test_batches(ctx, natpro, counts):
    """Ragged ligands, some without atoms or poses, an irregular pose and an irregular ligand; against one
    launch per ligand and single decks."""
    rng = np.random.default_rng(natpro)
    deck = deck_of(natpro, 1, 64)
    ligands = [synthetic_ligand(rng, int(rng.integers(0, 9)), 5.0, 12) for _ in counts]
    poses = [synthetic_poses(rng, n) for n in counts]
    ligands[0] = synthetic_ligand(rng, 4, 5.0, 12)
    ligands[-1]["x"][:1] = 1e30
    poses[2][3, -1] = np.nan
    batch = BatchDeck(deck.protein, deck.forcefield, ligands, poses, "direct")
    ctx.upload_batch(batch)
    assert sum(counts) >= 2 * max(16384, 64 * natpro ** 2)
    ctx.run_batch(ctx.default_cfg(4, 128))
    want = ctx.download_batch()
    for p, w in SHAPES:
        ctx.run_batch(ctx.default_cfg(p, w))
        assert np.array_equal(ctx.download_batch(), want, equal_nan=True), (p, w)
    ctx.run_batch(ctx.autotune_batch(50)[0])
    assert np.array_equal(ctx.download_batch(), want, equal_nan=True)
    ctx.run_batch(ctx.default_cfg(4, 128), per_ligand=True)
    assert np.array_equal(ctx.download_batch(), want, equal_nan=True)
    off = batch.pose_offsets()
    for l in (0, 2, len(counts) - 1):
        d = deck_of(natpro, 1, 64)
        d.protein, d.forcefield, d.ligand, d.poses = deck.protein, deck.forcefield, ligands[l], poses[l]
        ctx.upload(d)
        assert np.array_equal(in_pieces(ctx, d), want[off[l]:off[l + 1]], equal_nan=True), l
