"""The bisection of the Ising acceptance limits needs a logarithm that does not decrease from one
uniform to the next: logf over all 2^23 of them, compiled with the library's flags."""
import ctypes as C
import subprocess

import pytest

from nanomagmc_gb300 import build as B

pytestmark = pytest.mark.gpu

SRC = r"""
#include "philox.h"
__global__ void falls(unsigned* n, unsigned* equal) {
    const unsigned k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k + 1 >= 1u << 23) return;
    const float a = logf(nmmc_u01f(k << 9)), b = logf(nmmc_u01f((k + 1) << 9));
    if (!(b >= a)) atomicAdd(n, 1u);
    if (b == a) atomicAdd(equal, 1u);
}
extern "C" int count(unsigned* out) {
    unsigned* d = nullptr;
    if (cudaMalloc(&d, 8) != cudaSuccess || cudaMemset(d, 0, 8) != cudaSuccess) return 1;
    falls<<<(1 << 23) / 256, 256>>>(d, d + 1);
    const int rc = cudaMemcpy(out, d, 8, cudaMemcpyDeviceToHost) != cudaSuccess;
    cudaFree(d);
    return rc;
}
"""


def test_logf_does_not_fall_between_neighbouring_uniforms(tmp_path):
    src, lib = tmp_path / "falls.cu", tmp_path / "falls.so"
    src.write_text(SRC)
    subprocess.run([B._nvcc(), *B.ARCH, "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-I", B.CSRC, "-shared", str(src), "-o",
                    str(lib)], check=True, capture_output=True)
    out = (C.c_uint * 2)(7, 7)
    assert C.CDLL(str(lib)).count(out) == 0
    assert out[0] == 0
    assert out[1] < 1 << 23   # it was evaluated: not the same value everywhere
