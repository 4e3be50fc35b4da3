"""lvbgs_device_bytes against what a SuBSENSE handle allocates."""
import os
import subprocess

import pytest

from litiv_gb300 import _lib as L

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.mark.parametrize("W,H,C", [(320, 240, 3), (357, 288, 1), (1920, 1080, 3)])
def test_the_workspace_is_counted_as_it_is_allocated(product_lib, tmp_path, W, H, C):
    """The model is a multiple of 256 bytes; what is left is the work area, eight stream descriptors and four lists of
    one 8-byte entry a pixel."""
    if not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("no CUDA headers")
    src, exe = tmp_path / "sizes.cpp", tmp_path / "sizes"
    src.write_text('#include <cuda_runtime.h>\n#include <stdio.h>\n#include "lvbgs_internal.h"\n'
                   'int main() { printf("%zu %zu", sizeof(lvbgs::TickWork), sizeof(lvbgs::StreamDev)); }\n')
    subprocess.run(["g++", "-std=c++17"] + ["-I" + d for d in (os.path.join(CUDA, "include"), os.path.join(ROOT, "include"),
                                                                os.path.join(ROOT, "litiv_gb300", "csrc"))]
                   + [str(src), "-o", str(exe)], check=True)
    work, descriptor = (int(v) for v in subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split())
    total = product_lib.lvbgs_device_bytes(L.ALGO_SUBSENSE, W, H, C, 50)
    assert (total - work - 8 * descriptor - 32 * W * H) % 256 == 0
