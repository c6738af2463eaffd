"""csrc/softdbl.h on the device, bit for bit the IEEE operators for every leading significand
its first approximations see."""
import ctypes as C
import subprocess

import numpy as np
import pytest

from ebbcfd_gb300 import build as B

pytestmark = pytest.mark.gpu

PROBE = r"""
#include "softdbl.h"
typedef unsigned long long u64;

// a value for every index, the same in each launch
__device__ u64 mix(u64 z)
{
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}
__device__ double from(u64 exponent, u64 mantissa) { return __longlong_as_double((long long)((exponent << 52) | mantissa)); }

// i < 2^23: the leading 23 bits of the divisor's and the radicand's significand, all the seeds
// are made of; `low` fills the rest.  Counts results that differ from the IEEE operators'.
__global__ void soft_sweep(u64 low, u64 salt, unsigned *wrong)
{
    const u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (1ull << 23)) return;
    const u64 m = (i << 29) | (low & 0x1fffffffull), r = mix(i + salt);
    const double b = from(1023, m), a = from(1023 + (r >> 52) % 9 - 4, r & 0xfffffffffffffull);
    bool bad = !ebbsoft::divisor_ok(b);
    const double q = ebbsoft::div(a, ebbsoft::recip(b)), p = ebbsoft::mul(a, b);
    if (bad || __double_as_longlong(q) != __double_as_longlong(__ddiv_rn(a, b))) atomicAdd(wrong, 1u);
    if (__double_as_longlong(p) != __double_as_longlong(__dmul_rn(a, b))) atomicAdd(wrong + 1, 1u);
    for (int e = 0; e < 2; e++) {
        const double x = from(1023 + e, m), s = ebbsoft::root(x, bad);
        if (bad || __double_as_longlong(s) != __double_as_longlong(__dsqrt_rn(x))) atomicAdd(wrong + 2, 1u);
    }
}

extern "C" int run_soft(u64 low, u64 salt, unsigned *out)
{
    unsigned *d = nullptr;
    cudaError_t e = cudaMalloc(&d, 3 * sizeof(unsigned));
    if (e == cudaSuccess) e = cudaMemset(d, 0, 3 * sizeof(unsigned));
    if (e == cudaSuccess) {
        soft_sweep<<<(1 << 23) / 256, 256>>>(low, salt, d);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, d, 3 * sizeof(unsigned), cudaMemcpyDeviceToHost);
    cudaFree(d);
    return (int)e;
}
"""


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    d = tmp_path_factory.mktemp("softdbl")
    (d / "probe.cu").write_text(PROBE)
    subprocess.run([B._nvcc()] + B.ARCH + B.CU["k_fp64.cu"] +
                   ["-O3", "-std=c++17", "-shared", "-cudart", "static", "-Xcompiler", "-fPIC", "-I", B.CSRC,
                    str(d / "probe.cu"), "-o", str(d / "probe.so")], check=True)
    lib = C.CDLL(str(d / "probe.so"))
    lib.run_soft.argtypes = [C.c_uint64, C.c_uint64, C.c_void_p]
    return lib


@pytest.mark.parametrize("low", [0, 0x1fffffff, 0x10000000, 0x0badcafe])
def test_integer_quotients_and_roots_for_every_seed(probe, low):
    for salt in (1, 1 << 40):
        wrong = np.zeros(3, dtype=np.uint32)
        assert probe.run_soft(low, salt, wrong.ctypes.data) == 0
        assert list(wrong) == [0, 0, 0]
