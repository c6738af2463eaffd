"""csrc/softdbl.h: IEEE double products, quotients and square roots from integer
instructions, compared with the host's operators bit for bit."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHECK = r"""
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>
#include "softdbl.h"
using namespace ebbsoft;
static double from(uint64_t u) { double x; memcpy(&x, &u, 8); return x; }
static uint64_t bits(double x) { uint64_t u; memcpy(&u, &x, 8); return u; }
int main(int argc, char **argv) {
    const long N = atol(argv[1]);
    const int lo = atoi(argv[2]), hi = atoi(argv[3]);  // exponents of the operands
    std::mt19937_64 g(20260 + lo);
    auto val = [&](int e0, int e1, long i) {
        uint64_t m = g() & 0xfffffffffffffull;
        if (i % 5 == 0) m &= ~((1ull << (g() % 53)) - 1);    // trailing zeros: exact results and ties
        if (i % 11 == 0) m = 0xfffffffffffffull - (g() % 64);  // just below a power of two
        if (i % 13 == 0) m = g() % 64;                         // just above one
        const double x = from(((uint64_t)(e0 + (int)(g() % (e1 - e0 + 1)) + 1023) << 52) | m);
        if (i % 31 == 0) return (g() & 1) ? 0.0 : -0.0;
        return (g() & 1) ? -x : x;
    };
    long bad[3] = {0, 0, 0}, out = 0;
    for (long i = 0; i < N; i++) {
        double a = val(lo, hi, i + g() % 7), b = val(lo, hi, i + g() % 7);
        bool f = false;
        check<200>(a, f);
        check<200>(b, f);
        out += f;
        bad[0] += bits(mul(a, b)) != bits(a * b);
        const long pat[4] = {1, 5, 11, 13};
        b = val(lo < -125 ? -125 : lo, hi > 125 ? 125 : hi, pat[g() & 3]);
        if (i % 17 == 0) a = b * from(((uint64_t)(1023 + (int)(g() % 9) - 4) << 52) | (g() % 4096));
        if (i % 19 == 0) a = nextafter(b, (g() & 1) ? 1e300 : -1e300);
        f = !divisor_ok(b);
        check<200>(a, f);
        if (!f) bad[1] += bits(div(a, recip(b))) != bits(a / b);
        double x = fabs(val(2 * lo, 2 * hi - 2, i + g() % 7));
        if (i % 19 == 0) { const double t = (float)fabs(val(-60, 60, 1)); x = t * t; }
        if (i % 23 == 0 && x != 0.0) x = nextafter(x, (g() & 1) ? 1e300 : 1.0);
        f = false;
        const double r = root(x, f);
        out += f;
        if (!f) bad[2] += bits(r) != bits(sqrt(x));
    }
    // outside the ranges: reported
    long missed = 0;
    const double odd[6] = {0x1p-1030, -0x1p-201, 0x1p200, INFINITY, -INFINITY, NAN};
    for (double x : odd) {
        bool f = false;
        check<200>(x, f);
        missed += !f;
    }
    const double neg[4] = {-1.0, 0x1p-1030, INFINITY, NAN};
    for (double x : neg) {
        bool f = false;
        (void)root(x, f);
        missed += !f;
    }
    missed += divisor_ok(0.0) + divisor_ok(0x1p-126) + divisor_ok(0x1p126) + divisor_ok(NAN) + divisor_ok(INFINITY);
    printf("%ld %ld %ld %ld %ld\n", bad[0], bad[1], bad[2], out, missed);
    return 0;
}
"""


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    d = tmp_path_factory.mktemp("softdbl")
    (d / "check.cpp").write_text(CHECK)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, "ebbcfd_gb300", "csrc"),
                    str(d / "check.cpp"), "-o", str(d / "check")], check=True)
    return str(d / "check")


@pytest.mark.parametrize("lo,hi", [(-200, 199), (-10, 10), (-1, 1)])
def test_integer_products_quotients_and_roots_are_ieee(exe, lo, hi):
    out = subprocess.run([exe, "2000000", str(lo), str(hi)], capture_output=True, text=True, check=True).stdout
    assert [int(x) for x in out.split()] == [0, 0, 0, 0, 0]
