"""rcp_newton is the correctly rounded reciprocal that div_exact asks for, over all
2^23 mantissas (the all-ones one among them, which no proof covers), and the
quotients that the kernels form with it are the correctly rounded ones."""
import ctypes as C
import subprocess

import pytest

from voxelmapping_b200 import build as B

pytestmark = pytest.mark.gpu
SRC = r"""
#include "vmap_internal.cuh"
using namespace vmapb;
// a thread per mantissa of b, at one exponent; a: powers of two, all-ones and scattered mantissas
__global__ void check(int exp, unsigned* bad)
{
    const unsigned m = blockIdx.x * blockDim.x + threadIdx.x;
    const float b = __uint_as_float((unsigned)exp << 23 | m), y = rcp_newton(b);
    if (y != __frcp_rn(b)) atomicAdd(bad, 1u);
    unsigned a = m * 2654435761u;
    for (int k = 0; k < 8; ++k) {
        const unsigned am = k == 0 ? 0u : k == 1 ? 0x7fffffu : k == 2 ? m : a >> 9;
        const float x = __uint_as_float((unsigned)(127 + k) << 23 | am);
        if (div_exact(x, b, y) != __fdiv_rn(x, b) || div_exact(-x, b, y) != __fdiv_rn(-x, b)) atomicAdd(bad + 1, 1u);
        a = a * 1664525u + 1013904223u;
    }
}
extern "C" int run(int exp, unsigned* out)
{
    unsigned* d = nullptr;
    cudaError_t e = cudaMalloc(&d, 8);
    if (e == cudaSuccess) e = cudaMemset(d, 0, 8);
    if (e == cudaSuccess) {
        check<<<(1 << 23) / 256, 256>>>(exp, d);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, d, 8, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return (int)e;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("rcp")
    (d / "rcp.cu").write_text(SRC)
    cmd = [B.nvcc(), *B.NVCC_FLAGS, "-I" + str(B.CSRC), "-shared", str(d / "rcp.cu"), "-o", str(d / "rcp.so")]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return C.CDLL(str(d / "rcp.so"))


# divisors from 2^-20 (a depth just over 1e-6 m) over 1 (weights) to 2^22 (ray lengths), and the ends of the range
@pytest.mark.parametrize("exp", [60, 107, 126, 127, 128, 134, 149, 190])
def test_all_mantissas(lib, exp):
    bad = (C.c_uint * 2)(1, 1)
    assert lib.run(exp, bad) == 0
    assert list(bad) == [0, 0]
