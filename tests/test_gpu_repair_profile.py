"""The repair kernel's phase profile: two durations and a pixel count for each round."""
import ctypes as C

import pytest

from litiv_gb300 import BackgroundSubtractorSuBSENSE, SyntheticStream
from litiv_gb300 import _lib as L

pytestmark = pytest.mark.gpu


def test_two_durations_a_round():
    """Learning rate 1: frames of a few rounds, most of which have nothing to resolve again. Up to 16 rounds fit the
    profile's counts."""
    s = SyntheticStream(0, 0, 51, width=96, height=72, shape_min=10, shape_max=24, channels=3)
    m = BackgroundSubtractorSuBSENSE(seed=5)
    m.initialize(s.render(0))
    out, seen = (C.c_double * 64)(), 0
    for t in range(1, 12):
        before = m.scalars()
        m.apply(s.render(t), learningRateOverride=1.0)
        after = m.scalars()
        rounds = after["stat_repair_rounds"] - before["stat_repair_rounds"]
        n = L.lib().lvbgs_debug_repair_phases(m.handle, 0, out, 64)
        assert rounds <= 16 and n == 3 * rounds, (t, rounds, n)
        if rounds:
            counts = list(out[2 * rounds:n])
            assert sum(counts) == after["stat_repair_rematched"] - before["stat_repair_rematched"] and min(counts) >= 1
            assert min(out[:2 * rounds]) >= 0.0
        seen += rounds
    assert seen > 0
