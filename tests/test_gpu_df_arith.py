"""The double-float arithmetic (csrc/dfloat.h, csrc/dfpair.cuh) on the device, whose first
approximations the host tests can only stand in for, over FP32's whole range."""
import ctypes as C
import subprocess

import numpy as np
import pytest

from ebbcfd_gb300 import build as B

pytestmark = pytest.mark.gpu

PROBE = r"""
#include "dfpair.cuh"
using namespace ebbdev;

// a / b and sqrt(a) singly, and both in pairs of neighbouring elements (n even)
__global__ void df_ops(int n, const float2 *a, const float2 *b, float2 *div1, float2 *root1, float2 *recip2, float2 *root2,
                       float2 *div2, float2 *sums1, float2 *sums2)
{
    const int i = 2 * (blockIdx.x * blockDim.x + threadIdx.x);
    if (i + 1 >= n) return;
    df x[2], y[2], o[2];
    for (int k = 0; k < 2; k++) {
        x[k] = df(a[i + k].x, a[i + k].y);
        y[k] = df(b[i + k].x, b[i + k].y);
        const df q = x[k] / y[k], s = sqrt(x[k]);
        div1[i + k] = make_float2(q.hi, q.lo);
        root1[i + k] = make_float2(s.hi, s.lo);
    }
    split(recip(pair(y[0], y[1])), o[0], o[1]);
    for (int k = 0; k < 2; k++) recip2[i + k] = make_float2(o[k].hi, o[k].lo);
    split(pair(x[0], x[1]) / pair(y[0], y[1]), o[0], o[1]);
    for (int k = 0; k < 2; k++) div2[i + k] = make_float2(o[k].hi, o[k].lo);
    // products under sums and differences, of like and unlike sign
    const dfp X = pair(x[0], x[1]), Y = pair(y[0], y[1]);
    split((X * Y + X) * Y - (X * X - Y * Y), o[0], o[1]);
    for (int k = 0; k < 2; k++) {
        const df s = (x[k] * y[k] + x[k]) * y[k] - (x[k] * x[k] - y[k] * y[k]);
        sums1[i + k] = make_float2(s.hi, s.lo);
        sums2[i + k] = make_float2(o[k].hi, o[k].lo);
    }
    split(root(pair(x[0], x[1])), o[0], o[1]);
    for (int k = 0; k < 2; k++) root2[i + k] = make_float2(o[k].hi, o[k].lo);
}

extern "C" int run_df(int n, const float *a, const float *b, float *out)
{
    float2 *d = nullptr;
    const size_t s = (size_t)n * sizeof(float2);
    cudaError_t e = cudaMalloc(&d, 9 * s);
    if (e == cudaSuccess) e = cudaMemcpy(d, a, s, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(d + n, b, s, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        df_ops<<<(n / 2 + 127) / 128, 128>>>(n, d, d + n, d + 2 * (size_t)n, d + 3 * (size_t)n, d + 4 * (size_t)n,
                                             d + 5 * (size_t)n, d + 6 * (size_t)n, d + 7 * (size_t)n, d + 8 * (size_t)n);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, d + 2 * (size_t)n, 7 * s, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return (int)e;
}
"""


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    d = tmp_path_factory.mktemp("arith")
    (d / "probe.cu").write_text(PROBE)
    subprocess.run([B._nvcc()] + B.ARCH + B.CU["k_df.cu"] +
                   ["-O3", "-std=c++17", "-shared", "-cudart", "static", "-Xcompiler", "-fPIC", "-I", B.CSRC,
                    str(d / "probe.cu"), "-o", str(d / "probe.so")], check=True)
    lib = C.CDLL(str(d / "probe.so"))
    lib.run_df.argtypes = [C.c_int, C.c_void_p, C.c_void_p, C.c_void_p]
    return lib


def pairs(rng, n, e0, e1):
    """n double-floats of exponents e0..e1"""
    x = np.ldexp(1.0 + rng.random(n), rng.integers(e0, e1 + 1, n))
    hi = x.astype(np.float32)
    return np.stack([hi, (x - hi).astype(np.float32)], axis=1)


def value(p):
    return p[:, 0].astype(np.longdouble) + p[:, 1].astype(np.longdouble)


def ops(probe, a, b):
    out = np.zeros((7, len(a), 2), dtype=np.float32)
    a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
    assert probe.run_df(len(a), a.ctypes.data, b.ctypes.data, out.ctypes.data) == 0
    return out


@pytest.mark.parametrize("e0,e1,tol", [(-149, -101, 2.0 ** -22), (-100, -60, 2.0 ** -44), (-20, 20, 2.0 ** -44),
                                       (60, 126, 2.0 ** -44)])
def test_double_float_roots_over_the_range(probe, e0, e1, tol):
    """Within 2^-44 where the remainder of the FP32 root is an FP32 number, within 2^-22
    below.  The packed root is the single one's bit for bit, also beside a zero."""
    a = pairs(np.random.default_rng(200 + e0), 1 << 18, e0, e1)
    a[::101] = 0.0
    out = ops(probe, a, pairs(np.random.default_rng(2), len(a), -20, 20))
    pos = a[:, 0] > 0
    exact = np.sqrt(value(a))
    for r in (out[1], out[3]):
        assert (r[~pos] == 0.0).all()
        err = np.abs(value(r)[pos] / exact[pos] - 1)
        assert np.isfinite(err).all() and err.max() <= tol
    assert np.array_equal(out[1].view(np.uint32), out[3].view(np.uint32))


@pytest.mark.parametrize("e0,e1,f0,f1", [(-127, -127, 30, 60), (-126, -100, 26, 60), (-20, 20, -20, 20), (100, 126, -60, 0),
                                         (127, 127, -60, -1)])
def test_double_float_quotients_over_the_range(probe, e0, e1, f0, f1):
    """Divisors of exponents e0..e1 -- from half the smallest normal number to the largest
    exponent, where a reciprocal or a divisor is subnormal -- and quotients of exponents
    f0..f1, which keep every remainder an FP32 number: within 2^-44, in pairs the same bits.
    Reciprocals in pairs, within that and a unit of the smallest subnormal."""
    rng = np.random.default_rng(400 + e0)
    b = pairs(rng, 1 << 18, e0, e1)
    q = value(pairs(rng, len(b), f0, f1)).astype(np.float64)
    x = q * value(b).astype(np.float64)
    hi = x.astype(np.float32)
    a = np.stack([hi, (x - hi).astype(np.float32)], axis=1)
    out = ops(probe, a, b)
    err = np.abs(value(out[0]) / (value(a) / value(b)) - 1)
    assert np.isfinite(err).all() and err.max() <= 2.0 ** -44
    assert np.array_equal(out[0].view(np.uint32), out[4].view(np.uint32))
    inv = 1 / value(b)
    err = np.abs(value(out[2]) - inv)
    assert np.isfinite(err).all() and (err <= 2.0 ** -44 * inv + 2.0 ** -148).all()


def test_packed_sums_of_products_are_the_single_ones(probe):
    """Bit for bit: a product contracted with the sum that takes it would not be."""
    rng = np.random.default_rng(6)
    out = ops(probe, pairs(rng, 1 << 18, -3, 3), -pairs(rng, 1 << 18, -3, 3))
    assert np.array_equal(out[5].view(np.uint32), out[6].view(np.uint32))
