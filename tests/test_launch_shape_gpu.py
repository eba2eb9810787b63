"""The launch shape that a caller asks for is the one that runs: bude_gpu_default_cfg, and with it the model's
fasten and the driver's sweep, takes the reference's (PPWI, wgsize) pair; what the pair leaves open is the
library's choice.  No shape changes an energy."""
import numpy as np
import pytest

from minibude_gb300.capi import BudeError
from minibude_gb300.deck import DeckSpec, synthetic_deck
from minibude_gb300.model import Gb300Bude, GpuContext, launch_cfg

pytestmark = pytest.mark.gpu

DECK = synthetic_deck(DeckSpec("shape", 300, 9.0, 7, 12, 5000), seed=2)


@pytest.fixture(scope="module")
def ctx(built_library):
    c = GpuContext(0)
    c.upload(DECK)
    yield c
    c.close()


@pytest.mark.parametrize("ppwi,wgsize,want", [
    (1, 32, (1, 32)), (1, 33, (1, 64)), (3, 64, (2, 64)), (8, 64, (8, 64)), (8, 128, (8, 128)), (16, 512, (16, 512)),
    (32, 128, (16, 128)), (128, 100, (16, 128)), (4, 1024, (4, 512)), (2, 2**31 - 1, (2, 512))])
def test_the_pair_asked_for(ctx, ppwi, wgsize, want):
    cfg = ctx.default_cfg(ppwi, wgsize)
    assert (cfg.ppwi, cfg.wgsize) == want
    assert 32 * cfg.unroll <= cfg.ppwi * cfg.wgsize
    own = ctx.energies(DECK)
    ctx.run(cfg)
    assert np.array_equal(ctx.download(), own)


@pytest.mark.parametrize("ppwi,wgsize", [(0, 0), (-1, 0), (0, 31), (1, 1), (16, 0), (128, -5), (0, 96), (0, 512)])
def test_what_the_pair_leaves_open(ctx, ppwi, wgsize):
    cfg = ctx.default_cfg(ppwi, wgsize)
    if ppwi >= 1:
        assert cfg.ppwi == min(ppwi, 16)
    if wgsize >= 32:
        assert cfg.wgsize == wgsize
    own = ctx.energies(DECK)
    ctx.run(cfg)
    assert np.array_equal(ctx.download(), own)


def test_model_without_a_deck_and_with_few_poses(built_library):
    c = GpuContext(0)
    assert (c.default_cfg(8, 64).ppwi, c.default_cfg(8, 64).wgsize) == (8, 64)
    c.close()
    few = synthetic_deck(DeckSpec("few", 70, 6.0, 3, 12, 33), seed=3)
    want = Gb300Bude(1).fasten(few, 1, 0, 1, 0).energies
    for ppwi, wgsize in ((1, 32), (16, 512), (8, 64), (64, 0)):
        assert np.array_equal(Gb300Bude(ppwi).fasten(few, wgsize, 0, 1, 0).energies, want)


@pytest.mark.parametrize("split,tile,cluster", [(1, 8, 0), (64, 512, 0), (1, 64, 1), (8, 128, 1), (5, 24, 1)])
def test_split_tile_and_cluster_are_checked_and_change_no_bit(ctx, split, tile, cluster):
    own = ctx.energies(DECK)
    before = ctx.launch_count()
    ctx.run(launch_cfg(4, 128, 1, 64, 2, 0))
    launches = ctx.launch_count() - before
    ctx.run(launch_cfg(4, 128, split, tile, 2, cluster))
    assert ctx.launch_count() - before == 2 * launches
    assert np.array_equal(ctx.download(), own)
    for bad in ((65, 64, 0), (9, 64, 1), (0, 64, 0), (1, 4, 0), (1, 520, 0), (1, 12, 0), (1, 64, 2)):
        with pytest.raises(BudeError):
            ctx.run(launch_cfg(4, 128, bad[0], bad[1], 2, bad[2]))
