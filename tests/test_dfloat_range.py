"""csrc/dfloat.h over FP32's whole range, with first approximations as the device's
instructions give them: off by up to 2^-22.9, that of the root flushing what is not a normal
number."""
import os
import subprocess

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
