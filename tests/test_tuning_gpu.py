"""What the autotuners keep: a pick and its time hold for what was timed, and are measured again for another
protein, ligand or pose count."""
import pytest

from minibude_gb300.deck import DeckSpec, synthetic_deck
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
