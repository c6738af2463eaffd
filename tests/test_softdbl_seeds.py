"""csrc/softdbl.h with first approximations as far off as its header allows the device's
instructions to be (2^-22.9, relative), to either side: still the IEEE operators' bits.  A
seed of a value just above 0.5 may then lie below it."""
import os
import subprocess

import pytest

from tests.test_softdbl import CHECK, ROOT

SEEDS = r"""
#include <cmath>
#include <random>
static std::mt19937 seed_rng(9);
static float seed_off(double y)
{
    const double u = (double)seed_rng() * 0x1p-32;
    return (float)(y * (1.0 + OFF * 0x1.12p-23));
}
#define EBB_HOST_RCP(x) seed_off(1.0 / (double)(x))
#define EBB_HOST_RSQRT(x) seed_off(1.0 / std::sqrt((double)(x)))
"""


@pytest.mark.parametrize("lo,hi", [(-200, 199), (-1, 1)])
@pytest.mark.parametrize("off", ["-1.0", "1.0", "(2.0 * u - 1.0)"])
def test_integer_arithmetic_with_seeds_off_by_their_bound(tmp_path, off, lo, hi):
    (tmp_path / "check.cpp").write_text(SEEDS.replace("OFF", off) + CHECK)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, "ebbcfd_gb300", "csrc"),
                    str(tmp_path / "check.cpp"), "-o", str(tmp_path / "check")], check=True)
    out = subprocess.run([str(tmp_path / "check"), "2000000", str(lo), str(hi)], capture_output=True, text=True,
                         check=True).stdout
    assert [int(x) for x in out.split()] == [0, 0, 0, 0, 0]
