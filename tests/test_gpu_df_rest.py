"""Double-float solves of gas at or near rest against the oracle: speeds whose squares lie
below FP32's smallest normal number (2^-126, a speed of 1.1e-19) are ordinary values ahead
of a spreading disturbance, and the Roe flux and the wall take the root of u^2 + v^2.

Tolerances: those of tests/test_gpu_df.py, one evaluation and 100 steps."""
import json

import numpy as np
import pytest

import ebbcfd_gb300 as E
from ebbcfd_gb300 import meshgen
from oracle import gmsh_ref, ref
from tests.test_gpu_df import DF_RES_TOL, DF_STATE_TOL
from tests.test_gpu_parity import rel_err

pytestmark = pytest.mark.gpu


def box(flux):
    return json.dumps({"mesh": "m.msh", "dt": 1e-4, "tEnd": 1000.0, "flux": flux, "saveIter": -1, "plotIter": -1,
                       "forceBoundary": "Freestream", "initialConditions": [0.5, 0, 1, 1], "integrator": "RK2",
                       "limited": True, "CFL": 0.4,
                       "physicalConfig": {"Pr": 0.72, "R": 1.0, "gamma": 1.4, "Re": 100.0, "L": 1.0},
                       "boudaryConditions": [{"tag": "Freestream", "type": "inviscidWall", "q": [0.5, 0, 1, 1]}]})


def both(flux, n):
    mesh = meshgen.uniform_quads(n)
    om = ref.OracleMesh(mesh.as_reader_dict(), gmsh_ref.load_config(box(flux)))
    return E.UfvmSolver(mesh.to_solver_mesh(), E.load_config(box(flux)), "df"), om


def at_rest(om):
    q = om.state()
    q[:, 3] -= 0.5 * (q[:, 1] ** 2 + q[:, 2] ** 2) / q[:, 0]
    q[:, 1:3] = 0.0
    return q


@pytest.mark.parametrize("flux", ["roeFlux", "rusanovFlux"])
@pytest.mark.parametrize("speed", [1e-15, 1e-19, 1e-20, 1e-22, 1e-24])
def test_speeds_below_the_root_of_the_smallest_normal(speed, flux):
    s, om = both(flux, 12)
    q = at_rest(om)
    rng = np.random.default_rng(7)
    q[:, 0] *= 1 + 0.01 * rng.standard_normal(len(q))
    q[:, 1:3] = speed * rng.standard_normal((len(q), 2))
    q[:, 3] *= 1 + 0.01 * rng.standard_normal(len(q))
    R, dt, rmax = om.residual(q.copy())
    Rd, dtd, rd = s.ufvm_solver(q)
    s.close()
    assert rel_err(Rd, R) <= DF_RES_TOL
    assert abs(dtd - dt) <= 1e-12 * dt and abs(rd - rmax) <= 1e-11 * rmax


@pytest.mark.parametrize("flux", ["roeFlux", "rusanovFlux"])
def test_pressure_bump_in_a_closed_box(flux):
    s, om = both(flux, 64)
    q = at_rest(om)
    xy = s.mesh.centroids()
    q[:, 3] *= 1 + 0.1 * np.exp(-((xy[:, 0] - 0.4) ** 2 + (xy[:, 1] - 0.55) ** 2) / 0.003)
    om.set_state(q)
    s.set_state(q)
    for _ in range(3):
        om.run(4)
        s.run(4)
        assert rel_err(s.state, om.state()) <= DF_STATE_TOL
    s.close()
