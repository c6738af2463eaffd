"""Split solves of inviscid meshes beyond the size where the stage kernels change their
launch shape and load order (2.5M cells): an arena of three instances that together lie
beyond it gives bitwise the states and records of single solves, which lie below."""
import functools
import json

import numpy as np
import pytest

import ebbcfd_gb300 as E
from ebbcfd_gb300 import meshgen

pytestmark = pytest.mark.gpu

MESHES = {"quads": lambda: meshgen.uniform_quads(921), "polygons": lambda: meshgen.hanging_quads(514),
          "triangles": lambda: meshgen.wedge(850000, seed=0)}


@functools.lru_cache(maxsize=1)
def host_mesh(kind):
    return MESHES[kind]().to_solver_mesh()


def config(kind, integrator, mesh):
    q = [2.5, 0, 1, 1] if kind == "triangles" else [0.5, 0, 1, 1]
    bcs = [{"tag": t, "type": {"Symmetry": "symmetry", "Ramp": "inviscidWall"}.get(t, "fullState"), "q": q}
           for t in mesh.tags]
    return E.load_config(json.dumps({
        "mesh": "m.msh", "dt": 1e-4, "tEnd": 1000.0, "flux": "rusanovFlux" if kind == "triangles" else "roeFlux",
        "saveIter": -1, "plotIter": -1, "forceBoundary": mesh.tags[0], "initialConditions": q, "integrator": integrator,
        "limited": True, "CFL": 0.4, "boudaryConditions": bcs}))


@pytest.mark.parametrize("integrator", ["Euler", "RK2", "RK2_TVD", "RK4"])
@pytest.mark.parametrize("kind", list(MESHES))
def test_arena_beyond_the_line_equals_single_solves_below_it(kind, integrator):
    mesh = host_mesh(kind)
    assert mesh.n_cells < 2500000 < 3 * mesh.n_cells
    cfg = config(kind, integrator, mesh)
    xy = mesh.centroids()
    batch = E.UfvmBatch([mesh] * 3, cfg, "split")
    one = E.UfvmSolver(mesh, cfg, "split")
    q0 = one.state
    q = [q0 * (1 + 0.01 * np.sin(3 * (k + 1) * xy[:, :1] + 5 * xy[:, 1:] + np.arange(4))) for k in range(3)]
    for k in range(3):
        batch.set_instance_state(k, q[k])
    batch.run(3, records=False)
    for k in (0, 2):
        one.close()
        one = E.UfvmSolver(mesh, cfg, "split")
        one.set_state(q[k])
        rec = one.run(3)[-1]
        st = batch.status(k, 1)[0]
        assert np.array_equal(batch.instance_state(k), one.state)
        assert st["resid"] == list(rec[3:7]) and (st["drag"], st["lift"]) == (rec[1], rec[2])
    one.close()
    batch.close()
