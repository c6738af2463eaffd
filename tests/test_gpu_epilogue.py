"""The step epilogue's sums (residual norms and forces) against sums made independently, on
meshes whose block partial sums it adds in several parts: n x n quads, one update block per
256 cells, one part per 256 blocks and 16 at most.

  257: 259 blocks in parts of 130 and 129;  400: 625 in parts of 209, 209 and 207;
  1000: 3,907 in 15 parts of 245 and one of 232.

All 4 n boundary edges are in the force group.  A sum that leaves out or repeats a block is
off by 1/3,907 at least, one force edge by 1/4,000.

Tolerances.  FP64 and double-float: any order of these additions takes a value through fewer
than 256 of them, 2^-53 of the summed magnitudes each.  Split precision: squares and sums
within a block are FP32, fewer than 16 roundings of 2^-24 each.  The forces are the oracle's
within the accuracy of a step of the form (tests/test_gpu_small_meshes.py)."""
import functools

import numpy as np
import pytest

import ebbcfd_gb300 as E
from ebbcfd_gb300 import meshgen
from oracle import gmsh_ref, ref
from tests.test_gpu_small_meshes import text

pytestmark = pytest.mark.gpu


@functools.lru_cache(maxsize=None)
def oracle_step(n):
    mesh = meshgen.uniform_quads(n)
    cfg = text("rusanovFlux", "Euler", False)
    om = ref.OracleMesh(mesh.as_reader_dict(), gmsh_ref.load_config(cfg))
    host = mesh.to_solver_mesh()
    xy = host.centroids()
    q = om.state()
    q *= 1 + 0.05 * np.sin(9 * xy[:, :1] + 5 * xy[:, 1:] + np.arange(4))
    q[:, 2] = 0.2 + 0.05 * np.cos(7 * xy[:, 1])
    om.set_state(q)
    return host, E.load_config(cfg), q, om.run(1)[0]


@pytest.mark.parametrize("form", ["fp64", "df", "split"])
@pytest.mark.parametrize("n", [257, 400, 1000])
def test_sums_of_the_epilogue(n, form):
    host, cfg, q, rec = oracle_step(n)
    s = E.UfvmSolver(host, cfg, form)
    s.set_state(q)
    got = s.run(1)[0]
    new = s.state
    s.close()
    want = np.sqrt(n * n * np.sum((new - q) ** 2, axis=0, dtype=np.longdouble)) / np.sum(new, axis=0, dtype=np.longdouble)
    tol = 2.0 ** -20 if form == "split" else 2.0 ** -44
    assert np.abs(got[3:7] / want - 1).max() <= tol
    force = 4 * 4.0  # perimeter times p + rho |u|^2, and some
    assert np.abs(got[1:3] - rec[1:3]).max() <= force * {"fp64": 2.0 ** -44, "df": 3e-11, "split": 1e-5}[form]
