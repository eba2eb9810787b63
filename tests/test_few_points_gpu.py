"""Few points (poses x ligand atoms) get a warp each (csrc/cull_kernel.cuh: point_kernel).  Their energies are
the bits that the same poses get among so many others that the culled kernel takes them, for proteins around
the sizes of a cluster, of a cluster block and of the 16-bit list indices, dense ones that overflow a list of
candidates, poses near and far apart, and point counts on both sides of the rule's line."""
import dataclasses

import numpy as np
import pytest

import oracle
from minibude_gb300 import validate
from minibude_gb300.deck import BatchDeck, DeckSpec, synthetic_deck, synthetic_ligand, synthetic_poses
from minibude_gb300.model import GpuContext, launch_cfg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(built_library):
    c = GpuContext(0)
    yield c
    c.close()


def line(natpro):
    return min(8192, 4096 + 4 * natpro)


def deck_of(natpro, natlig, nposes, half_box=None, trans=3.0):
    box = half_box or 0.5 * (natpro / 0.05) ** (1 / 3)
    return synthetic_deck(DeckSpec("few", natpro, box, natlig, 12, nposes, max_trans=trans), seed=natpro)


def head(deck, n):
    return dataclasses.replace(deck, poses=np.ascontiguousarray(deck.poses[:, :n]))


def run(ctx, deck, p, w, u=1):
    ctx.upload(deck)
    ctx.run(launch_cfg(p, w, 1, 64, u))
    return ctx.download()


@pytest.mark.parametrize("trans", [3.0, 40.0])
@pytest.mark.parametrize("natpro,half_box", [(65, None), (96, None), (1023, None), (1025, None), (2080, None),
                                             (3000, 7.0), (65500, None), (70000, None)])
def test_the_bits_of_the_culled_kernel(ctx, natpro, half_box, trans):
    natlig = 3
    deck = deck_of(natpro, natlig, 9001, half_box, trans)
    many = run(ctx, deck, 8, 512, 2)
    for p, w, u in ((1, 32, 1), (2, 96, 2), (16, 512, 4), (4, 128, 4)):
        assert np.array_equal(run(ctx, deck, p, w, u), many), (p, w, u)
    most = line(natpro) // natlig
    for n, w in ((1, 32), (31, 64), (257, 512), (most, 32), (most, 96), (most, 512)):
        assert np.array_equal(run(ctx, head(deck, n), 8, w), many[:n]), (n, w)
    few = head(deck, 64)
    e32, e64 = oracle.fasten_f32(few), oracle.fasten_f64(few)
    scale = np.maximum(np.abs(e64), 1.0)
    bound = max(2e-4, 4 * float((np.abs(e32 - e64) / scale).max()))
    max_diff, failed = validate(many[:64], e32)
    assert not failed and max_diff < 0.025, (max_diff, failed[:5])
    assert float((np.abs(many[:64] - e64) / scale).max()) < bound


@pytest.mark.parametrize("natlig", [0, 1, 7])
def test_both_sides_of_the_line(ctx, natlig):
    most = line(300) // max(natlig, 1)
    deck = deck_of(300, natlig, 3 * most)
    many = run(ctx, deck, 4, 128, 2)
    for n in (most - 1, most, most + 1):
        assert np.array_equal(run(ctx, head(deck, n), 1, 128), many[:n]), n


def test_irregular_poses_and_decks(ctx):
    deck = deck_of(200, 4, 6000)
    rng = np.random.default_rng(1)
    for k, v in enumerate((np.nan, np.inf, -np.inf, 1e30, 3e11)):
        deck.poses[rng.integers(0, 6, 5), rng.integers(0, 500, 5)] = v
        deck.poses[3 + k % 3, 31 + k] = v
    wide = deck_of(200, 4, 6000)
    wide.forcefield["radius"][:] = 0.0
    for d in (deck, wide):
        many = run(ctx, d, 4, 128, 2)
        for n in (500, 33):
            assert np.array_equal(run(ctx, head(d, n), 1, 64), many[:n], equal_nan=True), n


def test_batches(ctx):
    """A batch of few points, ligands without atoms or poses among them, against single decks and a batch that is
    large enough for the culled kernel."""
    rng = np.random.default_rng(3)
    deck = deck_of(700, 1, 64)
    counts = (40, 0, 1, 33, 100, 64)
    ligands = [synthetic_ligand(rng, n, 5.0, 12) for n in (5, 3, 0, 12, 1, 9)]
    poses = [synthetic_poses(rng, n, 30.0) for n in counts]
    poses[3][4, 7] = np.nan
    few = BatchDeck(deck.protein, deck.forcefield, ligands, poses, "few")
    assert sum(n * len(l) for n, l in zip(counts, ligands)) < line(700)
    more = BatchDeck(deck.protein, deck.forcefield, ligands + [synthetic_ligand(rng, 9, 5.0, 12)],
                     poses + [synthetic_poses(rng, 2000)], "more")
    ctx.upload_batch(few)
    got = []
    for p, w in ((1, 32), (8, 128), (1, 512)):
        ctx.run_batch(launch_cfg(p, w, 1, 64, 1))
        got.append(ctx.download_batch())
        assert np.array_equal(got[0], got[-1], equal_nan=True), (p, w)
    ctx.upload_batch(more)
    ctx.run_batch(launch_cfg(4, 128, 1, 64, 2))
    assert np.array_equal(ctx.download_batch()[:few.total_poses], got[0], equal_nan=True)
    off = few.pose_offsets()
    for l in (0, 3, 5):
        d = dataclasses.replace(deck, ligand=ligands[l], poses=poses[l])
        assert np.array_equal(run(ctx, d, 2, 64), got[0][off[l]:off[l + 1]], equal_nan=True), l


def test_many_poses_without_atoms_beside_few_points(ctx):
    rng = np.random.default_rng(4)
    deck = deck_of(700, 1, 64)
    ligands = [synthetic_ligand(rng, n, 5.0, 12) for n in (0, 6, 0, 2)]
    poses = [synthetic_poses(rng, n) for n in (400000, 300, 1, 513)]
    batch = BatchDeck(deck.protein, deck.forcefield, ligands, poses, "none")
    off = batch.pose_offsets()
    ctx.upload_batch(batch)
    for p, w in ((1, 32), (4, 128)):
        ctx.run_batch(launch_cfg(p, w, 1, 64, 1))
        got = ctx.download_batch()
        assert not got[:off[1]].any() and not got[off[2]:off[3]].any()
        for l in (1, 3):
            d = dataclasses.replace(deck, ligand=ligands[l], poses=poses[l])
            assert np.array_equal(run(ctx, d, 2, 64), got[off[l]:off[l + 1]]), (p, w, l)
        ctx.upload_batch(batch)
