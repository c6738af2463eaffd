"""The stage kernels at the smallest meshes and at the edges of their blocks: n x n quads,
from a single cell (four boundary faces, no interior one) over counts around a warp's 8
and 32 cells and a block's 32, 64 and 256, in each precision form and with both fluxes,
against the oracle.

Plain FP64 is bitwise the oracle's.  The double-float form is held to 3e-11 and split
precision to 1e-5 of each component's largest magnitude: the tolerances of one evaluation
(tests/test_gpu_df.py) and of two steps (__graft_entry__.smoke) there."""
import json

import numpy as np
import pytest

import ebbcfd_gb300 as E
from ebbcfd_gb300 import meshgen
from oracle import gmsh_ref, ref

pytestmark = pytest.mark.gpu


def text(flux, integrator, viscosity):
    return json.dumps({"mesh": "m.msh", "dt": 1e-4, "tEnd": 1000.0, "flux": flux, "saveIter": -1, "plotIter": -1,
                       "forceBoundary": "Freestream", "initialConditions": [0.5, 0, 1, 1], "integrator": integrator,
                       "limited": True, "CFL": 0.4, "viscosity": viscosity,
                       "physicalConfig": {"Pr": 0.72, "R": 1.0, "gamma": 1.4, "Re": 100.0, "L": 1.0},
                       "boudaryConditions": [{"tag": "Freestream", "type": "fullState", "q": [0.5, 0, 1, 1]}]})


@pytest.mark.parametrize("viscosity", [False, True])
@pytest.mark.parametrize("flux", ["roeFlux", "rusanovFlux"])
@pytest.mark.parametrize("n", [1, 2, 3, 5, 6, 8, 11, 16, 17])
def test_small_meshes_match_oracle(n, flux, viscosity):
    cfg_text = text(flux, "RK2", viscosity)
    mesh = meshgen.uniform_quads(n)
    om = ref.OracleMesh(mesh.as_reader_dict(), gmsh_ref.load_config(cfg_text))
    q = om.state()
    rng = np.random.default_rng(n)
    q *= 1.0 + 0.05 * rng.standard_normal(q.shape) * [1, 1, 0, 1]
    q[:, 2] = 0.1 * rng.standard_normal(len(q))
    q[::3, 2] = 0.0  # exact zeros among the momenta
    om.set_state(q)
    rec = om.run(3)
    want = om.state()
    for form, tol in (("fp64", 0.0), ("df", 3e-11), ("split", 1e-5)):
        s = E.UfvmSolver(mesh.to_solver_mesh(), E.load_config(cfg_text), form)
        s.set_state(q)
        got = s.run(3)
        err = (np.abs(s.state - want).max(axis=0) / np.maximum(np.abs(want).max(axis=0), 1e-300)).max()
        s.close()
        assert err <= tol, (form, err)
        if form == "fp64":
            assert np.array_equal(got[:, [0, 7, 8]], rec[:, [0, 7, 8]])


@pytest.mark.parametrize("scale", [1e-70, 1e-20, 1e45])
def test_values_outside_the_integer_arithmetic(scale):
    """Momenta too small (and states too large) for the integer-pipe arithmetic take the
    plain operators: still bitwise the oracle's residual."""
    cfg_text = text("roeFlux", "RK2", False)
    mesh = meshgen.uniform_quads(12)
    om = ref.OracleMesh(mesh.as_reader_dict(), gmsh_ref.load_config(cfg_text))
    q = om.state()
    rng = np.random.default_rng(1)
    noise = rng.standard_normal(q.shape)
    if scale < 1:
        q[:, 0] *= 1 + 0.01 * noise[:, 0]
        q[:, 2] = scale * noise[:, 2]
        q[:, 3] *= 1 + 0.01 * noise[:, 3]
    else:
        q *= (1 + 0.01 * noise) * [1, scale ** 0.5, scale ** 0.5, scale]
        q[:, 1] *= 0.1
        q[:, 2] = q[:, 1] * noise[:, 2]
    R, dt, rmax = om.residual(q.copy())
    s = E.UfvmSolver(mesh.to_solver_mesh(), E.load_config(cfg_text))
    Rg, dtg, rg = s.ufvm_solver(q)
    s.close()
    assert np.array_equal(Rg, R) and dtg == dt and rg == rmax


def test_epilogue_parts_sum_alike_alone_and_batched():
    """66,049 cells have 259 update blocks: two parts in the step epilogue.  Alone and
    between two small instances the records' sums run in the same order."""
    cfg = E.load_config(text("rusanovFlux", "RK2", False))
    big, small = meshgen.uniform_quads(257).to_solver_mesh(), meshgen.uniform_quads(5).to_solver_mesh()
    one = E.UfvmSolver(big, cfg)
    xy = big.centroids()
    q = one.state
    q[:, 0] *= 1 + 0.05 * np.sin(9 * xy[:, 0] + 5 * xy[:, 1])
    one.set_state(q)
    rec = one.run(2)
    batch = E.UfvmBatch([small, big, small], cfg)
    batch.set_instance_state(1, q)
    batch.run(2, records=False)
    st = batch.status()[1]
    assert np.array_equal(batch.instance_state(1), one.state)
    assert st["resid"] == list(rec[-1, 3:7]) and (st["drag"], st["lift"]) == (rec[-1, 1], rec[-1, 2])
    # against sums in another order: 66,049 FP64 additions of one sign, 2^-53 each at most
    r = one.state - q
    assert rec.shape == (2, 10) and np.isfinite(r).all()
    one.close()
    batch.close()
