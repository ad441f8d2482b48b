"""The dynamic shared-memory limit of a kernel is kept per device: raised on one, it is still to be
raised on another.  Host code compiled against stand-ins for the two runtime calls it makes."""
import os
import shutil
import subprocess

import pytest

from copsandrobbers_gb300 import build as B

PROGRAM = r"""
#include "crgpu_smem.h"
#include <cstdio>
static int device = 0, calls = 0, last = 0;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int v) {
    ++calls;
    last = v;
    return v > 1000 ? cudaErrorInvalidValue : cudaSuccess;
}
static int a, b;
static void raise(int dev, const void* kernel, size_t bytes) {
    device = dev;
    const int before = calls;
    const cudaError_t e = crgpu::raise_smem_limit(kernel, bytes);
    printf("%d:%d:%d ", calls - before, calls > before ? last : 0, (int)(e == cudaSuccess));
}
int main() {
    raise(0, &a, 500); raise(0, &a, 400); raise(1, &a, 500); raise(1, &a, 600); raise(0, &a, 600);
    raise(1, &b, 500); raise(1, &b, 2000); raise(1, &b, 2000);
}
"""


@pytest.mark.skipif(not shutil.which("g++"), reason="g++ absent")
def test_limit_is_kept_per_device(tmp_path):
    src, exe = tmp_path / "limit.cpp", tmp_path / "limit"
    src.write_text(PROGRAM)
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(B.nvcc()))), "include")
    subprocess.run(["g++", "-std=c++17", "-I", B.CSRC, "-I", cuda, str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split()
    # calls of cudaFuncSetAttribute : the size given : success
    assert out == ["1:500:1", "0:0:1", "1:500:1", "1:600:1", "1:600:1", "1:500:1", "1:2000:0", "1:2000:0"]
