"""2D SOR as one thread-block cluster (grids without solid or outlet cells
between the block counts and the cells per thread that its rule names) against
the grid form: the same sweeps, at the cap and at convergence."""
import numpy as np
import pytest

from flursys_b200 import _abi
from flursys_b200.solver import _Handle

from .test_gpu_cavity2d import cfg2d

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(127, 64), (128, 64), (97, 101), (128, 128), (224, 128), (225, 128), (60, 400)])
@pytest.mark.parametrize("iters,tol", [(1, 1e-300), (40, 1e-300), (3000, 2.0)])
def test_cluster_sor_equals_the_grid_form(oracle, monkeypatch, shape, iters, tol):
    runs = []
    for env in ("1", "0"):
        monkeypatch.setenv("FLURSYS_2D_CLUSTER", env)
        c = cfg2d(oracle, *shape, tol=tol, dt=1e-4)
        c.pressure_solver = _abi.PRESSURE_SOR
        c.pressure_max_iters = iters
        h = _Handle(c)
        rng = np.random.default_rng(4)
        h.upload(_abi.FIELD_U, 0.1 * rng.standard_normal((shape[0] + 1) * shape[1]))
        runs.append((h.step(1), h.download(_abi.FIELD_PRESSURE)))
    (r1, p1), (r0, p0) = runs
    assert r1.pressure_iterations == r0.pressure_iterations and r1.pressure_status == r0.pressure_status
    # one program's operations in one order; a fused product may differ
    assert np.max(np.abs(p1 - p0)) <= 1e-12 * np.max(np.abs(p0))
    assert abs(r1.pressure_residual - r0.pressure_residual) <= 1e-9 * r0.pressure_residual + 1e-9
