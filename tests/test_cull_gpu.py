"""The exact kernel evaluates only the pairs that can interact (csrc/cull_kernel.cuh).  Its energies are
checked where finding those pairs can go wrong: clusters of 32 protein atoms and blocks of 32 clusters
that are just full, pose chunks and groups at their edges, a protein so dense that a list of candidates
overflows, proteins past the 16-bit list indices, poses far from the protein, and atom sums that take
several windows.  The oracle evaluates every pair; against FP64 the bound is the one of
test_forcefield_and_deck_sizes (4x the FP32 oracle's own error, at least 2e-4).  The order of a pose's sum
depends on nothing else, so every launch shape has to give the same bits."""
import numpy as np
import pytest

import oracle
from minibude_gb300 import validate
from minibude_gb300.deck import BatchDeck, DeckSpec, synthetic_deck, synthetic_ligand, synthetic_poses
from minibude_gb300.model import GpuContext, launch_cfg

pytestmark = pytest.mark.gpu

SHAPES = [(1, 32, 1), (2, 96, 2), (4, 128, 4), (8, 512, 2), (16, 512, 1), (16, 512, 4)]


@pytest.fixture(scope="module")
def ctx(built_library):
    c = GpuContext(0)
    yield c
    c.close()


def deck_of(natpro, half_box, natlig, nposes, seed=0, ntypes=12):
    return synthetic_deck(DeckSpec("cull", natpro, half_box, natlig, ntypes, nposes), seed=seed)


def energies(ctx, deck, shapes=SHAPES):
    ctx.upload(deck)
    ctx.run(ctx.default_cfg(8, 128))
    want = ctx.download()
    for p, w, u in shapes:
        ctx.run(launch_cfg(p, w, 1, 64, u))
        assert np.array_equal(ctx.download(), want), (p, w, u)
    return want


def assert_parity(got, deck):
    e32, e64 = oracle.fasten_f32(deck), oracle.fasten_f64(deck)
    scale = np.maximum(np.abs(e64), 1.0)
    bound = max(2e-4, 4 * float((np.abs(e32 - e64) / scale).max()))
    max_diff, failed = validate(got, e32)
    assert not failed and max_diff < 0.025, (max_diff, failed[:5])
    assert float((np.abs(got - e64) / scale).max()) < bound


@pytest.mark.parametrize("natpro", [1, 31, 32, 33, 1023, 1024, 1025, 2080])
def test_protein_sizes_around_clusters(ctx, natpro):
    deck = deck_of(natpro, 0.5 * (natpro / 0.05) ** (1 / 3), 5, 130, seed=natpro)
    assert_parity(energies(ctx, deck), deck)


@pytest.mark.parametrize("nposes", [1, 63, 64, 65, 255, 257, 4095, 4097, 8200])
def test_pose_counts_around_groups_and_chunks(ctx, nposes):
    deck = deck_of(400, 10.0, 3, nposes, seed=3)
    got = energies(ctx, deck)
    assert_parity(got[-256:], deck_tail(deck, 256))
    # a pose's energy is its own: the head of a longer run has the same bits
    assert np.array_equal(energies(ctx, deck_of(400, 10.0, 3, 9000, seed=3), [])[:nposes], got)


def deck_tail(deck, n):
    tail = deck.head(deck.nposes)
    tail.poses = np.ascontiguousarray(deck.poses[:, -n:])
    return tail


def test_more_candidates_than_a_list_holds(ctx):
    # 3,000 atoms within 6 A: every one is in reach of every group.
    deck = deck_of(3000, 6.0, 3, 600, seed=5)
    assert_parity(energies(ctx, deck), deck)


def test_more_atoms_than_the_list_indices_count(ctx):
    # 140,000 atoms: the pairs of a group lie on both sides of several 2,048-cluster blocks.
    deck = deck_of(140000, 65.0, 2, 48, seed=6, ntypes=3)
    assert_parity(energies(ctx, deck, [(1, 32, 1), (1, 64, 2), (8, 512, 4)]), deck)


def test_poses_far_from_the_protein(ctx):
    deck = deck_of(500, 11.0, 4, 700, seed=7)
    deck.poses = deck.poses.copy()
    deck.poses[3, ::7] += 40.0       # just out of reach
    deck.poses[4, 3::11] -= 1e6
    deck.poses[5, 5::13] = 2.0 ** 37  # the far end of what counts as regular
    got = energies(ctx, deck)
    assert_parity(got, deck)
    assert np.all(got[5::13] == 0.0)


def test_atom_sums_in_several_windows(ctx):
    # 2,000 ligand atoms x 300,000 poses: 2.4 GB of atom sums, three windows; the batch path cuts its
    # windows between chunks of poses.
    rng = np.random.default_rng(8)
    base = deck_of(40, 5.0, 4, 8, seed=8)
    ligand = synthetic_ligand(rng, 2000, 5.0, base.ntypes)
    poses = synthetic_poses(rng, 300000)
    deck = base.head(8)
    deck.ligand, deck.poses = ligand, poses
    ctx.upload(deck)
    cfg = launch_cfg(8, 512, 1, 64, 2)
    ctx.run(cfg)
    got = ctx.download()
    cut = 170001
    ctx.upload_batch(BatchDeck(deck.protein, deck.forcefield, [ligand, ligand],
                               [np.ascontiguousarray(poses[:, :cut]), np.ascontiguousarray(poses[:, cut:])]))
    ctx.run_batch(cfg)
    assert np.array_equal(ctx.download_batch(), got)
    few = deck.head(8)
    few.poses = np.ascontiguousarray(poses[:, [0, 1, 150000, 262143, 262144, 268287, 268288, 299999]])
    e64 = oracle.fasten_f64(few)
    e32 = oracle.fasten_f32(few)
    at = got[[0, 1, 150000, 262143, 262144, 268287, 268288, 299999]]
    scale = np.maximum(np.abs(e64), 1.0)
    assert (np.abs(at - e64) / scale).max() < max(2e-4, 4 * (np.abs(e32 - e64) / scale).max())


def evaluated(ctx, deck):
    """The deck's energies from the single-deck path, streamed in chunks, and as a batch of one ligand,
    which takes the poses as they come."""
    cfg = launch_cfg(4, 512, 1, 64, 2)
    ctx.upload(deck)
    ctx.run(cfg)
    got = ctx.download()
    streamed = np.full(deck.nposes, 7.0, np.float32)
    ctx.score_stream(cfg, deck.poses, streamed, 32768)
    ctx.upload_batch(BatchDeck(deck.protein, deck.forcefield, [deck.ligand], [deck.poses]))
    ctx.run_batch(cfg)
    return got, streamed, ctx.download_batch()


# On both sides of 4,096 poses, from which sets are sorted, of the line between 64 and 512 cells, and of a tile.
@pytest.mark.parametrize("natlig,nposes", [(200, 4095), (200, 4096), (91, 8193), (11, 68180), (11, 68182), (7, 131071),
                                           (3, 262144), (3, 262145), (2, 500001)])
def test_sorted_poses(ctx, natlig, nposes):
    deck = deck_of(300, 9.0, natlig, nposes, seed=nposes)
    got, streamed, plain = evaluated(ctx, deck)
    assert np.array_equal(got, plain)
    assert np.array_equal(streamed, plain)


@pytest.mark.parametrize("kind", ["one place", "a line", "two places", "far", "irregular"])
def test_sorted_poses_of_every_spread(ctx, kind):
    deck = deck_of(300, 9.0, 20, 40000, seed=9)
    t = deck.poses[3:]
    if kind == "one place":
        t[:] = 1.25
    elif kind == "a line":
        t[1:] = 0.0
    elif kind == "two places":
        t[:] = np.where(np.arange(40000) % 2, 4.0, -2.0)
    elif kind == "far":
        t[:, ::3] *= 1e30
        t[0, 1::3] -= 1e9
    else:
        t[0, 5::701] = np.nan
        t[2, 7::503] = np.inf
        deck.poses[1, 9::997] = np.inf
    got, streamed, plain = evaluated(ctx, deck)
    assert np.array_equal(got, plain, equal_nan=True)
    assert np.array_equal(streamed, plain, equal_nan=True)


@pytest.mark.parametrize("irregular", [False, True])
@pytest.mark.parametrize("ppwi,wgsize", [(2, 512), (4, 512), (1, 64)])
def test_batch_with_sorted_poses(ctx, ppwi, wgsize, irregular):
    # A dense protein, so that the batch's poses are sorted; one launch per ligand takes them as they come.
    rng = np.random.default_rng(11)
    base = deck_of(700, 6.0, 4, 8, seed=11)
    sizes = [(60, 1), (50, 5000), (20, 300), (64, 9001), (33, 257), (45, 4097)]
    ligands = [synthetic_ligand(rng, a, 5.0, base.ntypes) for a, _ in sizes]
    poses = [synthetic_poses(rng, n) for _, n in sizes]
    if irregular:
        ligands[4]["x"][3] = np.float32(1e30)
        poses[1][3, ::777] = np.nan
        poses[3][1, 5::901] = np.inf
        poses[5][4] = 0.5
    ctx.upload_batch(BatchDeck(base.protein, base.forcefield, ligands, poses))
    cfg = launch_cfg(ppwi, wgsize, 1, 64, 2)
    ctx.run_batch(cfg, per_ligand=True)
    want = ctx.download_batch()
    ctx.run_batch(cfg)
    assert np.array_equal(ctx.download_batch(), want, equal_nan=True)
    if not irregular:
        for l in (1, 3):
            deck = base.head(8)
            pick = np.arange(0, poses[l].shape[1], 97)
            deck.ligand, deck.poses = ligands[l], np.ascontiguousarray(poses[l][:, pick])
            first = sum(n for _, n in sizes[:l])
            assert_parity(want[first + pick], deck)


# Whole chunks and a remainder, of one and of many blocks of poses.
@pytest.mark.parametrize("natlig,nposes,ppwi", [(200, 60001, 2), (200, 120001, 8), (2432, 3000, 1), (40, 300007, 4)])
def test_streamed_chunks(ctx, natlig, nposes, ppwi):
    deck = deck_of(150, 7.0, natlig, nposes, seed=natlig)
    cfg = launch_cfg(ppwi, 512, 1, 64, 2)
    ctx.upload(deck)
    ctx.run(cfg)
    got = np.full(nposes, 7.0, np.float32)
    ctx.score_stream(cfg, deck.poses, got, 1)
    assert np.array_equal(got, ctx.download())


# One atom, about as many as are put in order, and more; an empty protein; atoms that are not numbers.
@pytest.mark.parametrize("natlig,nposes,odd", [(1, 100001, ""), (2, 50001, ""), (1023, 101, ""), (1024, 98, ""),
                                               (1025, 98, ""), (50, 2001, "nan"), (50, 2001, "empty")])
def test_atoms_longest_first(ctx, natlig, nposes, odd):
    deck = deck_of(200, 7.0, natlig, nposes, seed=natlig + nposes)
    if odd == "nan":
        deck.ligand["x"][[3, 40]] = np.nan
        deck.ligand["z"][7] = np.inf
    if odd == "empty":
        deck.protein = deck.protein[:0].copy()
    cfg = launch_cfg(4, 512, 1, 64, 2)
    ctx.upload(deck)
    ctx.run(cfg)
    got = ctx.download()
    ctx.upload_batch(BatchDeck(deck.protein, deck.forcefield, [deck.ligand], [deck.poses]))
    ctx.run_batch(cfg)
    assert np.array_equal(got, ctx.download_batch(), equal_nan=True)


# Plans of one block, around the ranking's tiles, of the most that are put in order and of one more; a protein
# shorter than the sample.
@pytest.mark.parametrize("atoms", [(1,), (1, 1), (100, 156), (100, 157), (8000, 8384), (8000, 8385)])
def test_batch_items_longest_first(ctx, atoms):
    rng = np.random.default_rng(len(atoms) + sum(atoms))
    base = deck_of(90, 6.0, 4, 8, seed=5)
    ligands = [synthetic_ligand(rng, a, 5.0, base.ntypes) for a in atoms]
    ligands[-1]["y"][0] = np.nan
    poses = [synthetic_poses(rng, 40 + 7 * l) for l in range(len(atoms))]
    ctx.upload_batch(BatchDeck(base.protein, base.forcefield, ligands, poses))
    cfg = launch_cfg(1, 64, 1, 64, 1)
    ctx.run_batch(cfg, per_ligand=True)
    want = ctx.download_batch()
    ctx.run_batch(cfg)
    assert np.array_equal(ctx.download_batch(), want, equal_nan=True)
