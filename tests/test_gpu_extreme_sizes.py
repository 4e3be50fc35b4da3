"""Frames of a few pixels and frames of a million rows, against the oracle (bit-exact)."""
import numpy as np
import pytest

import litiv_gb300 as lv
from oracle import pyoracle

pytestmark = pytest.mark.gpu

LOBSTER = (lv.BackgroundSubtractorLOBSTER, pyoracle.OracleLOBSTER, 2.0)
VIBE = (lv.BackgroundSubtractorViBe, pyoracle.OracleViBe, 2.0)
PBAS = (lv.BackgroundSubtractorPBAS, pyoracle.OraclePBAS, -1.0)
SUBSENSE = (lv.BackgroundSubtractorSuBSENSE, pyoracle.OracleSuBSENSE, 0.0)
PAWCS = (lv.BackgroundSubtractorPAWCS, pyoracle.OraclePAWCS, 0.0)


def _frames(W, H, channels, n, seed):
    rng = np.random.default_rng(seed)
    base = rng.integers(30, 120, (H, W, channels), dtype=np.uint8)
    out = []
    for t in range(n):
        f = base + rng.integers(0, 9, base.shape, dtype=np.uint8)
        f[t * H // (2 * n):t * H // (2 * n) + H // 3 + 1, :W // 2 + 1] = 230
        out.append(np.ascontiguousarray(f if channels == 3 else f[:, :, 0]))
    return out


def _run(algo, frames, gpu_args=None, oracle_args=None):
    cls, oracle, lr = algo
    gpu, ora = cls(seed=3, **(gpu_args or {})), oracle(seed=3, **(oracle_args or {}))
    gpu.initialize(frames[0])
    ora.initialize(frames[0])
    for t, f in enumerate(frames[1:], start=1):
        assert np.array_equal(gpu.apply(f, None, lr), ora.apply(f, lr)), t


@pytest.mark.parametrize("algo", [LOBSTER, PBAS], ids=["lobster", "pbas"])
def test_frames_of_more_tile_rows_than_a_grids_second_dimension(algo):
    """8 x 1,048,600: 65,538 rows of 16-pixel tiles (four samples a pixel keep the oracle to seconds)."""
    _run(algo, _frames(8, 1048600, 1, 3, 1), dict(nBGSamples=4, nRequiredBGSamples=1), dict(bg_samples=4, required_bg_samples=1))


@pytest.mark.parametrize("channels", [1, 3])
@pytest.mark.parametrize("algo,W,H", [(VIBE, 1, 1), (VIBE, 1, 7), (VIBE, 9, 1), (PBAS, 1, 1), (PBAS, 1, 7), (PBAS, 9, 1),
                                      (PBAS, 2, 2), (LOBSTER, 5, 5), (LOBSTER, 6, 40), (SUBSENSE, 5, 5), (SUBSENSE, 33, 5),
                                      (SUBSENSE, 5, 40), (PAWCS, 8, 8), (PAWCS, 9, 40)],
                         ids=lambda v: v if isinstance(v, int) else v[0].__name__[20:])
def test_frames_of_a_few_pixels(algo, W, H, channels):
    _run(algo, _frames(W, H, channels, 6, W + 7 * H))
