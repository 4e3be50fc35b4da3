"""Dense LBSP descriptors of device buffers that the kernel cannot use where they are."""
import ctypes as C

import numpy as np
import pytest

from litiv_gb300 import _lib as L
from oracle import pyoracle

pytestmark = pytest.mark.gpu

W, H = 67, 41


def _case(channels, seed):
    rng = np.random.default_rng(seed)
    img = rng.integers(0, 256, (H, W, channels), dtype=np.uint8)
    want = pyoracle.lbsp_compute2(img if channels == 3 else img[:, :, 0], rel_threshold=0.333, offset=2)
    return img, want.reshape(H, W, channels)


def _compute(img_ptr, channels, desc_ptr):
    st = L.lib().lvbgs_lbsp_compute2(C.c_void_p(img_ptr), W, H, channels, -1, 0.333, 2, C.c_void_p(desc_ptr), 0)
    assert st == L.OK


def _check(buf, at, before, want, channels):
    """descriptors in the interior, the border and the bytes around as they were"""
    n = W * H * channels * 2
    got = buf[at:at + n].copy().view(np.uint16).reshape(H, W, channels)
    expect = before[at:at + n].copy().view(np.uint16).reshape(H, W, channels)
    expect[2:-2, 2:-2] = want[2:-2, 2:-2]
    assert np.array_equal(got, expect)
    assert np.array_equal(buf[:at], before[:at]) and np.array_equal(buf[at + n:], before[at + n:])


@pytest.mark.parametrize("where", ["host", "device"])
@pytest.mark.parametrize("channels", [1, 3])
def test_descriptors_at_an_odd_address(channels, where):
    torch = pytest.importorskip("torch")
    img, want = _case(channels, channels)
    before = np.random.default_rng(9).integers(0, 256, W * H * channels * 2 + 64, dtype=np.uint8)
    if where == "host":
        buf = before.copy()
        _compute(img.ctypes.data, channels, buf.ctypes.data + 33)
    else:
        di, do = torch.from_numpy(img).cuda(), torch.from_numpy(before).cuda()
        torch.cuda.synchronize()
        _compute(di.data_ptr(), channels, do.data_ptr() + 33)
        buf = do.cpu().numpy()
    _check(buf, 33, before, want, channels)


@pytest.mark.parametrize("at", ["start", "middle", "end", "before", "past"])
@pytest.mark.parametrize("channels", [1, 3])
def test_an_image_in_the_memory_of_its_descriptors(channels, at):
    """The image is read as it was before the call, wherever it lies in or beside the descriptors."""
    torch = pytest.importorskip("torch")
    img, want = _case(channels, 7 + channels)
    n, desc_at = W * H * channels, W * H * channels // 2 * 2 + 16
    img_at = {"start": desc_at, "middle": desc_at + n // 2, "end": desc_at + n, "before": desc_at - n // 2,
              "past": desc_at + 2 * n - n // 2}[at]
    before = np.random.default_rng(10).integers(0, 256, desc_at + 4 * n, dtype=np.uint8)
    before[img_at:img_at + n] = img.reshape(-1)
    buf = torch.from_numpy(before).cuda()
    torch.cuda.synchronize()
    _compute(buf.data_ptr() + img_at, channels, buf.data_ptr() + desc_at)
    _check(buf.cpu().numpy(), desc_at, before, want, channels)
