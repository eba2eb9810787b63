"""What the autotuners keep: a pick and its time hold for what was timed, and are measured again for another
protein, ligand or pose count."""
import pytest

from minibude_gb300.deck import BatchSpec, DeckSpec, synthetic_batch, synthetic_deck
from minibude_gb300.model import GpuContext

pytestmark = pytest.mark.gpu


def deck(half_box, seed=1, nposes=4096):
    return synthetic_deck(DeckSpec("tune", 700, half_box, 20, 12, nposes), seed=seed)


def timed(ctx):
    """Whether an autotune call ran kernels, and its predicted ms."""
    before = ctx.launch_count()
    _, ms = ctx.autotune(200)
    return ctx.launch_count() > before, ms


def test_pick_follows_the_deck(built_library):
    with GpuContext(0) as c:
        dense, sparse = deck(4.0), deck(40.0)
        c.upload(dense)
        measured, dense_ms = timed(c)
        assert measured
        assert timed(c) == (False, dense_ms)
        c.upload(dense)  # the same records again: kept
        assert timed(c) == (False, dense_ms)
        c.upload(sparse)  # the same sizes, a sixtieth of the pairs
        measured, sparse_ms = timed(c)
        assert measured and sparse_ms < dense_ms
        assert timed(c) == (False, sparse_ms)
        c.set_poses(sparse.poses, ligand=deck(40.0, seed=2).ligand)
        assert timed(c)[0]
        c.set_poses(sparse.poses[:, :4000])
        assert timed(c)[0]
        assert not timed(c)[0]


def batch(seed):
    """Batches of one shape; the seed gives the ligands' atoms."""
    d = deck(12.0)
    return synthetic_batch(BatchSpec("tune", 6, 20, 20, 200, 200), d.protein, d.forcefield, seed=seed)


def test_kept_batch_plan_follows_the_ligands(built_library):
    with GpuContext(0) as c, GpuContext(0) as alone:
        c.upload_batch(batch(1))
        cfg, ms = c.autotune_batch(200)
        c.run_batch(cfg)
        before = c.launch_count()
        c.upload_batch(batch(1))
        assert c.launch_count() == before  # nothing to rank anew
        assert c.autotune_batch(200)[1] == ms and c.launch_count() == before
        c.run_batch(cfg)
        before = c.launch_count()
        c.upload_batch(batch(2))  # the same shape, other atoms
        assert c.launch_count() == before + 2
        c.run_batch(cfg)
        alone.upload_batch(batch(2))
        alone.run_batch(cfg)
        assert (c.download_batch() == alone.download_batch()).all()
        before = c.launch_count()
        c.autotune_batch(200)
        assert c.launch_count() > before
