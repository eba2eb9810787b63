"""Device memory kept between uploads: a context that has held other decks and batches (its buffers parts
of one allocation, grown or larger than needed) gives the bits of a new one."""
import numpy as np
import pytest

from minibude_gb300.deck import BatchSpec, DeckSpec, synthetic_batch, synthetic_deck
from minibude_gb300.model import GpuContext

pytestmark = pytest.mark.gpu

ORDERS = [(0, 1, 2, 0), (2, 0, 1, 2), (1, 2, 0, 1)]


def decks():
    return [synthetic_deck(DeckSpec("r", n, 9.0, l, t, p), seed=n) for n, l, t, p in
            ((40, 3, 4, 33), (700, 40, 12, 1), (333, 17, 20, 5000))]


def batches(deck):
    return [synthetic_batch(BatchSpec("r", *s), deck.protein, deck.forcefield, i)
            for i, s in enumerate(((2, 5, 9, 40, 90), (9, 20, 40, 100, 900), (30, 3, 64, 1, 30)))]


@pytest.mark.parametrize("order", ORDERS)
def test_decks_in_one_context(built_library, order):
    all_decks = decks()

    def run(c, d):
        c.upload(d)
        c.run(c.default_cfg(8, 128))
        return c.download()

    with_others = GpuContext(0)
    for i in order:
        alone = GpuContext(0)
        assert np.array_equal(run(with_others, all_decks[i]), run(alone, all_decks[i])), i
        alone.close()
    with_others.close()


@pytest.mark.parametrize("order", ORDERS)
def test_batches_and_gradients_in_one_context(built_library, order):
    deck = decks()[2]
    all_batches = batches(deck)

    def run(c, b, i):
        c.upload_batch(b)
        c.run_batch(c.default_cfg(8, 128))
        out = [c.download_batch()]
        c.surrogate_init(deck.protein, deck.forcefield, seed=5)
        c.surrogate_train(2, 64, seed=i)
        rng = np.random.default_rng(i)
        poses = rng.permutation(b.total_poses)[:b.total_poses // 2 + 1].astype(np.int32)
        out += list(c.surrogate_gradient(poses, out[0]))
        c.surrogate_train(3, 33, labels=out[0], seed=i)
        c.surrogate_score()
        return out + [c.surrogate_params(), c.surrogate_download()]

    with_others = GpuContext(0)
    for i in order:
        alone = GpuContext(0)
        got, want = run(with_others, all_batches[i], i), run(alone, all_batches[i], i)
        for k, (g, w) in enumerate(zip(got, want)):
            assert np.array_equal(g, w), (i, k)
        alone.close()
    with_others.close()
