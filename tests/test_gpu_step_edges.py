"""Every algorithm's frame step at the edges of their kernels' tiles, words and chunks, against the oracle (bit-exact)."""
import ctypes as C

import numpy as np
import pytest

from litiv_gb300 import BackgroundSubtractorLOBSTER, _lib as L
from litiv_gb300.metrics import BinClassif
from oracle import metrics as oracle_metrics, pyoracle
from tests.test_gpu_lobster import run_pair as lobster_pair
from tests.test_gpu_parity import run_pair
from tests.test_gpu_pbas import run_pair as pbas_pair
from tests.test_gpu_pawcs import run_pair as pawcs_pair
from tests.test_gpu_vibe import run_pair as vibe_pair

pytestmark = pytest.mark.gpu


def hollow_frames(W, H, channels, n, seed):
    """A textured background with hollow rectangles (holes to fill), specks and a bar across the frame."""
    rng = np.random.default_rng(seed)
    base = rng.integers(40, 90, (H, W, 3)).astype(np.int16)
    frames = []
    for t in range(n):
        img = base + rng.integers(-3, 4, base.shape)
        for _ in range(6 if t else 0):
            w, h = int(rng.integers(6, max(7, W // 2))), int(rng.integers(6, max(7, H - 2)))
            x, y = int(rng.integers(0, max(1, W - 4))), int(rng.integers(0, max(1, H - 4)))
            keep = img[y + 2:y + h - 2, x + 2:x + w - 2].copy()
            img[y:y + h, x:x + w] = rng.integers(150, 255, 3)
            img[y + 2:y + 2 + keep.shape[0], x + 2:x + 2 + keep.shape[1]] = keep
        speck = rng.random((H, W)) < 0.01
        img[speck & (t > 0)] = 250
        if t % 3 == 2:
            img[H // 2:H // 2 + 2] = 200
        img = np.clip(img, 0, 255).astype(np.uint8)
        frames.append(img if channels == 3 else np.ascontiguousarray(img[:, :, 0]))
    return frames


@pytest.mark.parametrize("W,H,k,channels", [(31, 9, 1, 1), (32, 8, 3, 3), (33, 17, 15, 3), (127, 23, 17, 1),
                                            (128, 24, 31, 3), (130, 25, 9, 1), (1024, 16, 13, 1), (1061, 19, 9, 3),
                                            (2053, 11, 5, 1)])
def test_post_processing_at_word_tile_and_chunk_edges(W, H, k, channels):
    """Hole filling over rows of one word up to three 32-word chunks, every median width class (window counts
    of four and of five bit planes), frames that end inside a word, a tile and a quad of pixels."""
    run_pair(hollow_frames(W, H, channels, 7, W * 31 + H), seed=W, nDefaultMedianBlurKernelSize=k)


@pytest.mark.parametrize("channels", [1, 3])
@pytest.mark.parametrize("N,nreq", [(1, 1), (5, 2), (8, 3), (9, 2), (17, 1), (50, 4), (64, 2), (50, 0)])
def test_ordered_scans_by_groups_and_by_lanes(N, nreq, channels):
    """Sample counts around the evaluation's cap and the groups' steps of eight, and one to four required
    matches: the scans' stops and minima, with dense overwrites (learning rate 1) and foreground shares from
    a few pixels (one item a group) to most of the frame (every lane its own)."""
    frames = hollow_frames(96, 64, channels, 9, 100 * N + nreq)
    rng = np.random.default_rng(N)
    frames[5] = rng.integers(0, 256, frames[5].shape, dtype=np.uint8)
    lrs = [1.0 if t in (2, 3, 4, 6, 7) else 0.0 for t in range(len(frames))]
    run_pair(frames, seed=nreq + 3, lrs=lrs, nBGSamples=N, nRequiredBGSamples=nreq)


@pytest.mark.parametrize("W,H,channels", [(641, 243, 3), (328, 241, 1), (329, 240, 3), (320, 248, 1), (15, 5200, 1),
                                          (15, 5201, 3)])
def test_area_down_sampling_at_ragged_sizes(W, H, channels):
    """The frame-level down-sampling by groups of lanes: integral scales (8 and 15) with and without aligned
    rows, fractional scales in one or both directions (the averages are part of the compared state)."""
    run_pair(hollow_frames(W, H, channels, 3, W + H), seed=2)


@pytest.mark.parametrize("channels", [1, 3])
@pytest.mark.parametrize("words", [2, 3, 7, 50])
def test_pawcs_word_streams(words, channels):
    """Dictionaries of one word (the held word alone) up to the full count, through the local pass's bubble
    order, the updaters' loops at the last word and the later updaters, on a frame of partial tiles with border
    pixels that update themselves."""
    roi = np.zeros((43, 61), np.uint8)
    roi[3:40, 4:58] = 255
    frames = hollow_frames(61, 43, channels, 9, 7 * words)
    lrs = [1.0 if t in (3, 4, 7) else 0.0 for t in range(len(frames))]
    pawcs_pair(frames, seed=words, lrs=lrs, roi=roi, nMaxNbWords=words)


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("n", [1, 15, 16, 17, 4095, 4097, 70001])
def test_classification_counters_at_packed_byte_edges(n, offset):
    """Sizes around the 16-pixel packs and the 4,096-pixel blocks, images at and off 16-byte boundaries, with
    and without a region of interest, against the restatement."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    codes = np.array([0, 50, 85, 170, 255, 17], np.uint8)
    mask, gt = (rng.choice(codes, n) for _ in range(2))
    roi = rng.choice(np.array([0, 255], np.uint8), n)

    def on_device(a):
        buf = torch.zeros(n + offset, dtype=torch.uint8, device="cuda")
        buf[offset:] = torch.from_numpy(a).cuda()
        return buf[offset:].view(1, n)

    for r in (None, roi):
        got = BinClassif().accumulate(on_device(mask), on_device(gt), None if r is None else on_device(r))
        assert list(got.counts) == oracle_metrics.accumulate(mask[None], gt[None], None if r is None else r[None])


@pytest.mark.parametrize("where", ["host", "device"])
@pytest.mark.parametrize("W,H,channels", [(3, 9, 1), (4, 4, 3), (5, 5, 3), (61, 3, 1), (67, 53, 3), (640, 360, 1)])
def test_lbsp_descriptors_keep_the_border(W, H, channels, where):
    """Dense descriptors into host and device buffers: the interior against the oracle, the 2-pixel border as the
    caller left it."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(W * H)
    img = rng.integers(0, 256, (H, W, channels), dtype=np.uint8)
    mark = rng.integers(0, 65536, (H, W, channels), dtype=np.uint16)
    want = mark.copy()
    if W > 4 and H > 4:
        want[2:-2, 2:-2] = pyoracle.lbsp_compute2(img if channels == 3 else img[:, :, 0], rel_threshold=0.333,
                                                  offset=2).reshape(H, W, channels)[2:-2, 2:-2]
    if where == "host":
        out = mark.copy()
        ptrs = (img.ctypes.data, out.ctypes.data)
    else:
        di = torch.from_numpy(img).cuda()
        do = torch.from_numpy(mark.view(np.uint8).reshape(-1).copy()).cuda()
        torch.cuda.synchronize()
        ptrs = (di.data_ptr(), do.data_ptr())
    st = L.lib().lvbgs_lbsp_compute2(C.c_void_p(ptrs[0]), W, H, channels, -1, 0.333, 2, C.c_void_p(ptrs[1]), 0)
    assert st == L.OK
    if where == "device":
        out = do.cpu().numpy().view(np.uint16).reshape(H, W, channels)
    assert np.array_equal(out, want)


@pytest.mark.parametrize("channels", [1, 3])
@pytest.mark.parametrize("W,H,N,nreq", [(96, 64, 4, 1), (97, 61, 5, 2), (65, 33, 8, 3), (64, 17, 9, 2), (130, 16, 20, 1),
                                        (33, 47, 35, 4), (129, 79, 63, 2)])
def test_sample_scans_of_the_consensus_models(W, H, N, nreq, channels):
    """LOBSTER, ViBe and PBAS with sample counts around the lane scans' caps and the groups' steps of eight, frames
    of ragged gradient tiles and sum chunks, few repairs a block (one a group) and, at learning rate 1, most of a
    block's pixels (every lane its own)."""
    frames = hollow_frames(W, H, channels, 8, W * 7 + N)
    rng = np.random.default_rng(N)
    frames[5] = rng.integers(0, 256, frames[5].shape, dtype=np.uint8)
    lrs = [16.0, 1.0, 1.0, 2.0, 16.0, 1.0, 1.0, 3.0]
    args = dict(nBGSamples=N, nRequiredBGSamples=nreq)
    lobster_pair(frames, seed=N, lrs=lrs, **args)
    vibe_pair(frames, N + 1, lrs, **args)
    pbas_pair(frames, N + 2, lrs, **args)
    pbas_pair(frames, N + 3, [-1.0] * len(frames), **args)


@pytest.mark.parametrize("W,H,k,channels", [(31, 33, 3, 1), (128, 16, 9, 3), (129, 17, 15, 1), (255, 31, 17, 3), (300, 20, 31, 1),
                                            (67, 53, 1, 3), (640, 35, 9, 1)])
def test_median_of_bits_and_gradient_tiles(W, H, k, channels):
    """LOBSTER's median over windows of four and of five bit planes and PBAS's gradient, on frames that end inside a
    word, a tile and eight pixels, with rows at and off the alignment of the word loads."""
    frames = hollow_frames(W, H, channels, 5, W * 5 + k)
    gpu = BackgroundSubtractorLOBSTER(seed=k, nDefaultMedianBlurKernelSize=k)
    ora = pyoracle.OracleLOBSTER(seed=k, default_median_blur_kernel_size=k)
    gpu.initialize(frames[0])
    ora.initialize(frames[0])
    for f in frames[1:]:
        assert np.array_equal(gpu.apply(f, learningRate=16.0), ora.apply(f, 16.0))
    pbas_pair(frames, k + 1, [-1.0] * len(frames))
