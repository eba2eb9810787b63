"""A call that returns an error has let go of its caller's buffers: nothing still copies from them."""
import ctypes

import numpy as np
import pytest

from minibude_gb300 import capi
from minibude_gb300.capi import fptr, ptr
from minibude_gb300.deck import DeckSpec, synthetic_deck, synthetic_poses
from minibude_gb300.model import GpuContext, PinnedBuffer, launch_cfg

pytestmark = pytest.mark.gpu

NPOSES = 2_000_000  # 48 MB: the copy outlasts the refusal by far
DECK = synthetic_deck(DeckSpec("failed", 40, 6.0, 2, 8, 64), seed=4)
BAD = launch_cfg(3, 128, 1, 64, 2)  # refused: 3 poses per thread


@pytest.fixture(scope="module")
def poses():
    return synthetic_poses(np.random.default_rng(5), NPOSES)


def test_score_host_with_a_refused_shape(built_library, poses):
    with GpuContext(0) as c:
        c.upload(DECK)
        want = c.score_host(c.default_cfg(0, 0), poses, np.empty(NPOSES, np.float32)).copy()
        c.upload(DECK)
        pinned, out = PinnedBuffer(poses.shape), np.empty(NPOSES, np.float32)
        pinned.array[...] = poses
        p = pinned.array
        rc = capi.lib().bude_gpu_score_host(c.handle, ctypes.byref(BAD), None, 0, ptr(p), NPOSES, NPOSES, fptr(out))
        p[5, -64:] = 100.0  # the caller has its buffer back; these bytes are copied last
        assert rc == capi.lib().bude_gpu_run(c.handle, ctypes.byref(BAD), None) != 0
        c.nposes = NPOSES
        c.run(c.default_cfg(0, 0))
        assert np.array_equal(c.download(), want)
        pinned.free()
