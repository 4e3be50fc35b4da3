"""Frames and masks on the device at any address: each algorithm's frame step against the oracle (bit-exact), with
the bytes around the masks left as they were. A frame of a contiguous clip of odd size starts at any byte, and the
kernels choose word loads and stores by the address."""
import numpy as np
import pytest

import litiv_gb300 as lv
from oracle import pyoracle
from tests.test_gpu_step_edges import hollow_frames

pytestmark = pytest.mark.gpu

CLASSES = {"subsense": (lv.BackgroundSubtractorSuBSENSE, pyoracle.OracleSuBSENSE, 0.0),
           "pawcs": (lv.BackgroundSubtractorPAWCS, pyoracle.OraclePAWCS, 0.0),
           "lobster": (lv.BackgroundSubtractorLOBSTER, pyoracle.OracleLOBSTER, 2.0),
           "vibe": (lv.BackgroundSubtractorViBe, pyoracle.OracleViBe, 2.0),
           "pbas": (lv.BackgroundSubtractorPBAS, pyoracle.OraclePBAS, -1.0)}
SIZES = {"subsense": [(61, 43), (64, 48), (320, 240)], "pawcs": [(61, 43), (64, 48)],
         "lobster": [(5, 5), (6, 5), (61, 43), (64, 48)], "vibe": [(2, 3), (61, 43)], "pbas": [(5, 5), (61, 43), (128, 32)]}
LAST_COLOR = ("subsense", "lobster")  # (PAWCS's is compared in its own tests' state)


@pytest.mark.parametrize("offset", [1, 2, 3, 4, 8, 16])
@pytest.mark.parametrize("channels", [1, 3])
@pytest.mark.parametrize("algo,W,H", [(a, w, h) for a in SIZES for w, h in SIZES[a]])
def test_device_frames_and_masks_at_any_address(algo, W, H, channels, offset):
    torch = pytest.importorskip("torch")
    cls, oracle, lr = CLASSES[algo]
    frames = hollow_frames(W, H, channels, 5, 13 * W + H)
    gpu, ora = cls(seed=offset), oracle(seed=offset)
    n = frames[0].size
    buf = torch.empty(len(frames) * n + offset, dtype=torch.uint8, device="cuda")
    clip = buf[offset:].view((len(frames),) + frames[0].shape)  # frame k: offset + k n
    clip.copy_(torch.from_numpy(np.stack(frames)))
    masks = torch.full((W * H + 64,), 77, dtype=torch.uint8, device="cuda")
    mask = masks[32 + offset:32 + offset + W * H].view(H, W)
    torch.cuda.synchronize()
    gpu.initialize(clip[0])
    ora.initialize(frames[0])
    for t in range(1, len(frames)):
        gpu.apply(clip[t], mask, lr)
        want = ora.apply(frames[t], lr)
        got = masks.cpu().numpy()
        assert np.array_equal(got[32 + offset:32 + offset + W * H].reshape(H, W), want), t
        assert (got[:32 + offset] == 77).all() and (got[32 + offset + W * H:] == 77).all(), t
    if algo in LAST_COLOR:
        assert np.array_equal(gpu.state_map("LAST_COLOR").ravel(), np.asarray(ora.state_map("LAST_COLOR")).ravel())
