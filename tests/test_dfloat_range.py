"""csrc/dfloat.h over FP32's whole range, with first approximations as the device's
instructions give them: off by up to 2^-22.9, that of the root flushing what is not a normal
number."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHECK = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <random>
static std::mt19937_64 g(3);
static double u01() { return (double)(g() >> 11) * 0x1p-53; }
static float off(double y) { return (float)(y * (1.0 + (2.0 * u01() - 1.0) * 0x1.12p-23)); }
static float flush(float x) { return std::fabs(x) < 0x1p-126f ? std::copysign(0.0f, x) : x; }
#define EBB_HOST_RCP(x) off(1.0 / (double)(x))
#define EBB_HOST_RSQRT(x) flush(off(1.0 / std::sqrt((double)flush(x))))
#include "dfloat.h"
using ebbdf::df;
typedef long double L;
static L val(df a) { return (L)a.hi + (L)a.lo; }
static df rnd(int e0, int e1)
{
    return df(std::ldexp(1.0 + u01(), e0 + (int)(g() % (uint64_t)(e1 - e0 + 1))));
}
int main()
{
    double low = 0, high = 0;
    long odd = 0;
    for (int k = 0; k < 1000000; k++) {
        const df a = rnd(-149, 126);
        const L r = std::sqrt(val(a));
        const double e = (double)(std::fabs(val(ebbdf::sqrt(a)) - r) / r);
        if (!(e < 1.0)) odd++;  // NaN too
        double &m = a.hi < 0x1p-100f ? low : high;
        m = std::fmax(m, e);
    }
    const df z = ebbdf::sqrt(df(0.0f)), n = ebbdf::sqrt(df(-1.0f)), t = ebbdf::sqrt(df(-0x1p-140f));
    odd += z.hi != 0.0f || z.lo != 0.0f || n.hi == n.hi || t.hi == t.hi;
    std::printf("%ld %g %g\n", odd, low * 0x1p22, high * 0x1p44);
    return 0;
}
"""


def build(tmp_path, text, name):
    src, exe = tmp_path / (name + ".cpp"), tmp_path / name
    src.write_text(text)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, "ebbcfd_gb300", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    return str(exe)


def test_square_root_down_to_the_smallest_subnormal(tmp_path):
    """Within 2^-44 where the remainder of the FP32 root is an FP32 number (from 2^-100 on),
    within 2^-22 -- FP32's own precision and a unit -- below; zero gives zero, a negative
    number NaN."""
    odd, low, high = (float(x) for x in subprocess.run([build(tmp_path, CHECK, "root")], capture_output=True, text=True,
                                                       check=True).stdout.split())
    assert odd == 0 and low <= 1.0 and high <= 1.0, (odd, low, high)


PRECISION = CHECK[:CHECK.index("static df rnd")] + r"""
// the long division and the root from IEEE FP32 operations that the short forms replace
static df div_ieee(df a, df b)
{
    const float y = 1.0f / b.hi, q1 = a.hi * y;
    const df r = a - ebbdf::mul_f(b, q1);
    const float q2 = r.hi * y;
    const df r2 = r - ebbdf::mul_f(b, q2);
    const df q = ebbdf::fast_two_sum(q1, q2);
    return ebbdf::fast_two_sum(q.hi, q.lo + r2.hi * y);
}
static df root_ieee(df a)
{
    const float s = sqrtf(a.hi);
    const df e = a - ebbdf::two_prod(s, s);
    return ebbdf::fast_two_sum(s, e.hi / (2.0f * s));
}
static df rnd(bool product)
{
    const df a = df(std::ldexp(1.0 + u01(), (int)(g() % 41) - 20));
    return product ? a * df(1.0 + u01()) : a;  // a product's low word is not renormalised
}
struct Err {
    double max = 0, sum = 0;
    void add(df x, L r)
    {
        const double e = (double)(std::fabs(val(x) - r) / std::fabs(r)) * 0x1p48;
        max = std::fmax(max, e);
        sum += e * e;
    }
};
int main(int argc, char **argv)
{
    const int N = 4000000;
    Err q, q0, i, i0, s, s0;
    for (int k = 0; k < N; k++) {
        const df a = rnd(argc > 1), b = rnd(argc > 1), one = df(1.0f);
        q.add(a / b, val(a) / val(b));
        q0.add(div_ieee(a, b), val(a) / val(b));
        i.add(one / b, 1 / val(b));
        i0.add(div_ieee(one, b), 1 / val(b));
        s.add(ebbdf::sqrt(a), std::sqrt(val(a)));
        s0.add(root_ieee(a), std::sqrt(val(a)));
    }
    for (const Err *e : {&q, &q0, &i, &i0, &s, &s0}) std::printf("%.3f %.4f ", e->max, std::sqrt(e->sum / N));
    return 0;
}
"""


@pytest.mark.parametrize("product", [False, True])
def test_quotient_and_root_as_near_as_from_ieee_operations(tmp_path, product):
    """The short quotient and root, from approximate FP32 reciprocals, against the ones from
    IEEE FP32 operations on the same operands: the same largest error, to the 10% that the
    largest of 4,000,000 is uncertain by, and no larger an rms error."""
    out = subprocess.run([build(tmp_path, PRECISION, "precision")] + ["product"] * product, capture_output=True, text=True,
                         check=True).stdout.split()
    q, q0, inv, inv0, s, s0 = [(float(out[k]), float(out[k + 1])) for k in range(0, 12, 2)]
    for name, now, ieee in (("quotient", q, q0), ("reciprocal", inv, inv0), ("root", s, s0)):
        assert now[0] <= 1.1 * ieee[0] and now[1] <= ieee[1], (name, now, ieee)
