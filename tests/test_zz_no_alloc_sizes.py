"""bude_gpu_fasten_noalloc over the decks that its tables lay out differently: below one cluster, at the
edges of the sort and of the record array, with sorted poses, and with more atom sums than the working memory holds."""
import numpy as np
import pytest

import oracle
from minibude_gb300.capi import check
from minibude_gb300.deck import DeckSpec, synthetic_deck
from test_zz_no_alloc import Caller, torch_cuda  # noqa: F401

pytestmark = pytest.mark.gpu

# (protein atoms, half box, types, ligand atoms, poses)
DECKS = [(1, 2.0, 3, 5, 100), (31, 5.0, 3, 5, 100), (32, 5.0, 3, 5, 100), (33, 5.0, 3, 5, 100),
         (1023, 14.0, 9, 26, 1000), (1025, 14.0, 9, 26, 1000),
         (16384, 34.0, 8, 9, 300), (16385, 34.0, 7, 9, 300),
         (131072, 68.0, 1, 4, 64), (8, 3.0, 16384, 4, 200),
         (300, 9.0, 5, 70, 65535),
         # poses sorted from 400,000 points on
         (500, 10.0, 5, 50, 7999), (500, 10.0, 5, 50, 8000), (500, 10.0, 5, 100, 4095), (500, 10.0, 5, 100, 4097),
         (500, 10.0, 5, 9, 65536)]


@pytest.mark.parametrize("natpro,half_box,ntypes,natlig,nposes", DECKS)
def test_noalloc_deck_sizes(built_library, torch_cuda, natpro, half_box, ntypes, natlig, nposes):  # noqa: F811
    deck = synthetic_deck(DeckSpec("na", natpro, half_box, natlig, ntypes, nposes), seed=natpro)
    c = Caller(torch_cuda, deck)
    check(c.call(built_library))
    got = c.result()
    sample = np.unique(np.r_[0, nposes - 1, np.arange(0, nposes, max(1, nposes // 200))])
    sub = deck.head(8)
    sub.poses = np.ascontiguousarray(deck.poses[:, sample])
    e32, e64 = oracle.fasten_f32(sub), oracle.fasten_f64(sub)
    scale = np.maximum(np.abs(e64), 1.0)
    # The reference's single-precision arithmetic on the same poses sets the scale of the rounding.
    bound = max(2e-4, 4 * float((np.abs(e32 - e64) / scale).max()))
    assert float((np.abs(got[sample] - e64) / scale).max()) < bound
    check(c.call(built_library))
    assert np.array_equal(c.result(), got)
