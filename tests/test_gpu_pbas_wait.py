"""A PBAS frame step is over, its frame-level mean included, when apply() returns."""
import time

import numpy as np
import pytest

from litiv_gb300 import BackgroundSubtractorPBAS, SyntheticStream

pytestmark = pytest.mark.gpu


def test_nothing_of_a_frame_step_is_left_when_apply_returns():
    """1920x1080 BGR: the mean's ordered sum is some 100 us of kernels. A wait for the device after apply() takes
    no longer than one for an idle device; 20 us are allowed for the scatter of host timers."""
    torch = pytest.importorskip("torch")
    stream = SyntheticStream(0, 0, 11, width=1920, height=1080, channels=3)
    frames = [torch.from_numpy(stream.render(t)).cuda() for t in range(4)]
    mask = torch.zeros((1080, 1920), dtype=torch.uint8, device="cuda")
    model = BackgroundSubtractorPBAS(seed=3)
    model.initialize(frames[0])
    after, idle = [], []
    for t in range(1, 25):
        model.apply(frames[t % 4], mask)
        t0 = time.perf_counter()
        torch.cuda.synchronize()
        t1 = time.perf_counter()
        torch.cuda.synchronize()
        after.append(t1 - t0)
        idle.append(time.perf_counter() - t1)
    assert np.median(after) < np.median(idle) + 20e-6, (np.median(after), np.median(idle))
