"""The screen's exact energies are the batch's, whichever kernel its picks and its fallback take: a warp per point
for a few, every pair for many poses against a small protein, the culled kernel otherwise."""
import numpy as np
import pytest

from minibude_gb300.deck import BatchSpec, DeckSpec, synthetic_batch, synthetic_deck
from minibude_gb300.model import GpuContext, launch_cfg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("natpro", [20, 700])
def test_picks_and_fallback(built_library, natpro):
    deck = synthetic_deck(DeckSpec("s", natpro, 0.5 * (natpro / 0.05) ** (1 / 3), 4, 12, 4), seed=1)
    batch = synthetic_batch(BatchSpec("s", 6, 4, 9, 20000, 20000), deck.protein, deck.forcefield, 3)
    batch.poses[2][4, 17] = np.nan
    cfg = launch_cfg(4, 128, 1, 64, 2, cluster=0)
    with GpuContext(0) as c:
        c.upload_batch(batch)
        c.run_batch(cfg)
        exact = c.download_batch()
        c.surrogate_init(deck.protein, deck.forcefield, seed=2)
        c.surrogate_score()
        sur = c.surrogate_download()
        for top, chunks in ((0.5, 0), (0.5, 3), (0.05, 2), (0.0005, 0), (0.0005, 6)):
            c.screen(cfg, top_frac=top, audit_frac=top / 10, audit_tol=1e9, seed=5, chunks=chunks)
            final, rescored, _ = c.screen_download(batch.nligands)
            assert np.array_equal(final[rescored], exact[rescored], equal_nan=True), (top, chunks)
            assert np.array_equal(final[~rescored], sur[~rescored]), (top, chunks)
        st = c.screen(cfg, top_frac=0.01, audit_frac=0.01, audit_tol=-1.0)
        final, rescored, _ = c.screen_download(batch.nligands)
        assert st["fallback_ligands"] == batch.nligands and rescored.all()
        assert np.array_equal(final, exact, equal_nan=True)
