"""Batches around the sizes of the descriptor tables that travel as kernel arguments, and a captured batch."""
import ctypes as C

import numpy as np
import pytest

from litiv_gb300 import BackgroundSubtractorSuBSENSE, SyntheticStream, batch_apply
from litiv_gb300 import _lib as L

pytestmark = pytest.mark.gpu


def _frames(i, n, width=48, height=40):
    s = SyntheticStream(0, 0, 300 + i, width=width, height=height, shape_min=8, shape_max=16, channels=3 if i % 2 else 1)
    return [s.render(t) for t in range(n)]


def _models(frames):
    out = []
    for i, f in enumerate(frames):
        out.append(BackgroundSubtractorSuBSENSE(seed=i))
        out[-1].initialize(f[0])
    return out


@pytest.mark.parametrize("n", [1, 2, 16, 17, 64, 65, 129])
def test_batches_around_the_table_sizes(n):
    """One stream, tables of up to 16 and of 64, and one and two further tables: each stream as alone."""
    frames = [_frames(i, 4) for i in range(n)]
    batch, alone = _models(frames), _models(frames)
    for t in range(1, 4):
        masks = batch_apply(batch, [f[t] for f in frames])
        for i, m in enumerate(alone):
            assert np.array_equal(masks[i], m.apply(frames[i][t])), (t, i)


def test_a_captured_batch_replays():
    """The descriptors lie in the captured launches: frames put where the captured ones were give the masks of the
    streams alone."""
    torch = pytest.importorskip("torch")
    frames = [_frames(i, 6, 160, 120) for i in range(3)]
    batch, alone = _models(frames), _models(frames)
    image = [torch.from_numpy(f[1]).cuda() for f in frames]
    mask = [torch.zeros((120, 160), dtype=torch.uint8, device="cuda") for _ in frames]
    torch.cuda.synchronize()
    hs = (C.c_void_p * 3)(*[m.handle for m in batch])
    fr = (L.LvbgsFrame * 3)()
    for i in range(3):
        fr[i].image, fr[i].stride, fr[i].fgmask, fr[i].learning_rate = image[i].data_ptr(), 0, mask[i].data_ptr(), 0.0
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    sp = C.c_void_p(stream.cuda_stream)
    assert L.lib().lvbgs_batch_apply(hs, fr, 3, sp) == L.OK and L.lib().lvbgs_batch_wait(hs, 3, sp) == L.OK
    for m, f in zip(alone, frames):
        m.apply(f[1])
    with torch.cuda.stream(stream):
        graph.capture_begin(capture_error_mode="thread_local")
        status = L.lib().lvbgs_batch_apply(hs, fr, 3, sp)
        graph.capture_end()
    assert status == L.OK
    for t in range(2, 6):
        with torch.cuda.stream(stream):
            for i in range(3):
                image[i].copy_(torch.from_numpy(frames[i][t]))
            graph.replay()
        stream.synchronize()
        for i, m in enumerate(alone):
            assert np.array_equal(mask[i].cpu().numpy(), m.apply(frames[i][t])), (t, i)
