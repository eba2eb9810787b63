"""Poses that are scored by the reference's arithmetic (csrc/edge_pose.cuh) one after the other stay spread over
the warps when a large set is sorted by translation: those whose translation is the cause take no longer
than those whose angles are."""
import numpy as np
import pytest

from minibude_gb300.deck import BatchDeck, DeckSpec, synthetic_deck
from minibude_gb300.model import GpuContext

pytestmark = pytest.mark.gpu


def decks(nposes):
    out = []
    for field in (0, 3):  # an angle, a translation
        d = synthetic_deck(DeckSpec("irregular", 938, 13.3, 26, 34, nposes), seed=1)
        d.poses[field, ::10] = np.nan
        out.append(d)
    return out


def test_deck(built_library):
    times = []
    for d in decks(65536):
        with GpuContext(0) as c:
            c.upload(d)
            cfg = c.default_cfg(0, 0)
            c.run_many(cfg, 3, False)
            times.append(float(np.median(c.run_many(cfg, 9, False)[0])))
            e = c.download()
            assert np.isnan(e[::10]).all() and np.isfinite(np.delete(e, np.s_[::10])).all()
    assert times[1] < 1.2 * times[0], times


def test_batch(built_library):
    times = []
    for d in decks(60000):
        batch = BatchDeck(d.protein, d.forcefield, [d.ligand] * 2, [d.poses] * 2, "irregular")
        with GpuContext(0) as c:
            c.upload_batch(batch)
            cfg = c.default_cfg(8, 512)
            c.run_batch(cfg)
            times.append(float(np.median([c.run_batch(cfg) for _ in range(9)])))
            e = c.download_batch()
            assert np.isnan(e[::10]).all() and np.isfinite(np.delete(e, np.s_[::10])).all()
    assert times[1] < 1.2 * times[0], times
