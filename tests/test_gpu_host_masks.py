"""PAWCS masks in pageable host memory: delivered by a frame that ends, left alone by one that fails, and no
reason for the host to wait while a frame is enqueued."""
import ctypes as C

import numpy as np
import pytest

from litiv_gb300 import BackgroundSubtractorPAWCS, BackgroundSubtractorSuBSENSE, LvException, SyntheticStream
from litiv_gb300 import _lib as L
from litiv_gb300 import batch_apply

pytestmark = pytest.mark.gpu

FAULT_PAWCS_ROUNDS = 3


def _frames(n, seed, channels, width=96, height=72):
    s = SyntheticStream(0, 0, seed, width=width, height=height, shape_min=10, shape_max=24, channels=channels)
    return [s.render(t) for t in range(n)]


def _initialized(cls, seed, frame):
    m = cls(seed=seed)
    m.initialize(frame)
    return m


def _frame_with_two_rounds(frames, seed):
    """index of the first frame whose fixed point takes more than one round"""
    twin = _initialized(BackgroundSubtractorPAWCS, seed, frames[0])
    for t in range(1, len(frames)):
        twin.apply(frames[t])
        if twin.scalars()["fixed_point_rounds"] > 1:
            return t
    raise AssertionError("every frame converges in one round")


@pytest.mark.parametrize("batched", [False, True])
@pytest.mark.parametrize("channels", [1, 3])
def test_a_failed_frame_leaves_the_mask(channels, batched):
    frames = _frames(9, 70, channels)
    k = _frame_with_two_rounds(frames, 7)
    m = _initialized(BackgroundSubtractorPAWCS, 7, frames[0])
    for f in frames[1:k]:
        m.apply(f)
    mask = np.full(frames[0].shape[:2], 77, np.uint8)
    assert L.lib().lvbgs_debug_inject_fault(m.handle, FAULT_PAWCS_ROUNDS) == L.OK
    with pytest.raises(LvException) as ei:
        batch_apply([m], [frames[k]], [mask]) if batched else m.apply(frames[k], mask)
    assert ei.value.status == L.DEVICE_ERROR
    assert (mask == 77).all()


def test_a_mixed_batch_delivers_pageable_masks():
    """Three PAWCS streams beside two of SuBSENSE, masks in numpy arrays: each equals the stream alone."""
    kinds = [(BackgroundSubtractorPAWCS, 3), (BackgroundSubtractorSuBSENSE, 3), (BackgroundSubtractorPAWCS, 1),
             (BackgroundSubtractorSuBSENSE, 1), (BackgroundSubtractorPAWCS, 3)]
    frames = [_frames(9, 80 + i, c) for i, (_, c) in enumerate(kinds)]
    mixed, alone = ([_initialized(cls, 40 + i, frames[i][0]) for i, (cls, _) in enumerate(kinds)] for _ in range(2))
    for t in range(1, 9):
        masks = batch_apply(mixed, [f[t] for f in frames])
        for i, m in enumerate(alone):
            assert np.array_equal(masks[i], m.apply(frames[i][t])), (t, i)


def test_the_host_enqueues_a_frame_without_waiting():
    """1280x720 BGR: the device takes milliseconds, a hundred launches a fraction of one. With a pageable mask too the
    host's time goes to the wait, not to the enqueueing."""
    frames = _frames(5, 90, 3, 1280, 720)
    m = _initialized(BackgroundSubtractorPAWCS, 9, frames[0])
    mask = np.zeros((720, 1280), np.uint8)
    for f in frames[1:]:
        m.apply(f, mask)
    parts = (C.c_double * 5)()
    assert L.lib().lvbgs_debug_pawcs_host_timing(m.handle, parts) == L.OK
    assert parts[1] > parts[0], list(parts)
