"""Scoring calls from several threads at once, and calls that cannot be served."""
import threading

import numpy as np
import pytest

from litiv_gb300.metrics import BinClassif
from oracle import metrics as oracle_metrics

pytestmark = pytest.mark.gpu


def _images(n, seed):
    rng = np.random.default_rng(seed)
    codes = np.array([0, 50, 85, 170, 255, 17], np.uint8)
    return rng.choice(codes, (1, n)), rng.choice(codes, (1, n))


def test_threads_score_different_sizes_at_once():
    """Twelve threads, grids of one block up to hundreds, each on a stream of its own and more calls than places."""
    torch = pytest.importorskip("torch")
    wrong = []

    def work(i):
        n = 1 + 4096 * (i * i) + 37 * i
        mask, gt = _images(n, i)
        want = oracle_metrics.accumulate(mask, gt, None)
        dm, dg = torch.from_numpy(mask).cuda(), torch.from_numpy(gt).cuda()
        torch.cuda.synchronize()
        stream = torch.cuda.Stream()
        for k in range(40):
            a, b = (mask, gt) if k % 8 == 0 else (dm, dg)
            got = list(BinClassif().accumulate(a, b, cuda_stream=stream.cuda_stream).counts)
            if got != want:
                wrong.append((i, k, got, want))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(12)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong[:3]


def test_a_captured_stream_is_refused_and_nothing_is_lost():
    """A call waits for its result, so it cannot be captured; more refused calls than there are places leave the
    capture and the calls after it as they should be."""
    torch = pytest.importorskip("torch")
    mask, gt = _images(70001, 5)
    dm, dg = torch.from_numpy(mask).cuda(), torch.from_numpy(gt).cuda()
    x = torch.zeros(8, device="cuda")
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        graph.capture_begin()
        x += 1
        for _ in range(70):
            with pytest.raises(RuntimeError):
                BinClassif().accumulate(dm, dg, cuda_stream=stream.cuda_stream)
        graph.capture_end()
    graph.replay()
    torch.cuda.synchronize()
    assert x.sum().item() == 8
    assert list(BinClassif().accumulate(dm, dg).counts) == oracle_metrics.accumulate(mask, gt, None)
