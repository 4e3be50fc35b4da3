"""Which buffers a kernel may use where they are (litiv_gb300/csrc/staging.h), compiled for the host."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

PROGRAM = r"""
#include "staging.h"
#include <stdio.h>
using namespace lvbgs;
static int bad = 0;
#define CHECK(c) do { if (!(c)) { printf("%d: %s\n", __LINE__, #c); ++bad; } } while (0)
int main() {
    cudaPointerAttributes a = {};
    alignas(16) static unsigned char buf[64];
    a.type = cudaMemoryTypeDevice;
    a.device = 1;
    CHECK(usable_in_place(a, 1, buf, 2));
    CHECK(!usable_in_place(a, 0, buf, 2));      // another device's memory
    CHECK(!usable_in_place(a, 1, buf + 1, 2));  // an odd address
    CHECK(usable_in_place(a, 1, buf + 1, 1));
    a.type = cudaMemoryTypeManaged;
    CHECK(usable_in_place(a, 0, buf, 2));
    CHECK(!usable_in_place(a, 0, buf + 3, 2));
    a.type = cudaMemoryTypeHost;
    CHECK(!usable_in_place(a, 1, buf, 1));
    a.type = cudaMemoryTypeUnregistered;
    CHECK(!usable_in_place(a, 1, buf, 1));
    CHECK(ranges_overlap(buf, 8, buf + 7, 8) && ranges_overlap(buf + 7, 8, buf, 8) && ranges_overlap(buf, 64, buf + 8, 2));
    CHECK(!ranges_overlap(buf, 8, buf + 8, 8) && !ranges_overlap(buf + 8, 8, buf, 8));
    return bad;
}
"""


def test_buffers_that_kernels_may_use_in_place(tmp_path):
    if not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("no CUDA headers")
    src, exe = tmp_path / "staging_test.cpp", tmp_path / "staging_test"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I" + os.path.join(CUDA, "include"), "-I" + os.path.join(ROOT, "litiv_gb300", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
