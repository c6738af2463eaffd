"""The autotuner searches the launch shapes of the kernels that run, the shipped ones among
them: a re-run times what is there and can keep it."""
import os
import re

from ebbcfd_gb300 import autotune

CSRC = os.path.join(os.path.dirname(os.path.abspath(autotune.__file__)), "csrc")


def defines(name):
    return {m[0]: int(m[1]) for m in re.findall(r"^#define (EBB_\w+) (\d+)$", open(os.path.join(CSRC, name)).read(), re.M)}


def test_shipped_shapes_are_candidates():
    tuned = defines("tuned.h")
    rows = [autotune.setting(r) for r in range(autotune.N_ROWS)]
    assert set(tuned) == {m for pair in autotune.MACRO.values() for m in pair}
    for (form, kernel), (threads, blocks) in autotune.MACRO.items():
        assert (tuned[threads], tuned[blocks]) in [r[form][kernel] for r in rows], (form, kernel)


def test_second_order_cell_kernel_of_fp64_and_double_float_is_searched():
    text = open(os.path.join(CSRC, "kernels.cuh")).read()
    shapes = {f: re.search(r"constexpr int cell4_%s\(\) \{ return is_fp64<T> \? (\w+) : (\w+); \}" % f, text).groups()
              for f in ("threads", "minb")}
    for k, form in enumerate(("fp64", "df")):
        assert autotune.MACRO[(form, "cell")] == (shapes["threads"][k], shapes["minb"][k])


def test_every_variant_defines_every_shape():
    macros = sorted({m for pair in autotune.MACRO.values() for m in pair})
    for r in range(autotune.N_ROWS):
        assert sorted(d[2:].split("=")[0] for d in autotune.defines(r)) == macros
