"""More instances in one arena than a launch grid has rows (65,535): the step epilogue has
one block at least per instance."""
import numpy as np
import pytest

import ebbcfd_gb300 as E
from ebbcfd_gb300 import meshgen
from tests.test_gpu_small_meshes import text

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [65535, 65536])
def test_many_single_cells_in_one_arena(n):
    cfg = E.load_config(text("rusanovFlux", "RK2", False))
    mesh = meshgen.uniform_quads(1).to_solver_mesh()
    batch = E.UfvmBatch([mesh] * n, cfg)
    q = np.array([[1.0, 0.6, 0.1, 8.0]])
    for k in (0, n - 1):
        batch.set_instance_state(k, q * (1 + 0.01 * (k > 0)))
    batch.run(2, records=False)
    for k, given in ((0, True), (1, False), (n - 1, True)):
        one = E.UfvmSolver(mesh, cfg)
        if given:
            one.set_state(q * (1 + 0.01 * (k > 0)))
        rec = one.run(2)[-1]
        st = batch.status(k, 1)[0]
        assert np.array_equal(batch.instance_state(k), one.state), k
        assert st["iterations"] == 2 and (st["drag"], st["lift"]) == (rec[1], rec[2])
        assert np.array_equal(st["resid"], rec[3:7], equal_nan=True)  # 0 / 0 where no momentum is
        one.close()
    batch.close()
