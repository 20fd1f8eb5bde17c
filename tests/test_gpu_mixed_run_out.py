"""MIXED solves with a tolerance that cannot be met, on grids so small that the
FP32 recurrence reaches numbers whose products vanish before its next
replacement: the residual is replaced and the solve goes on to its cap, as the
forms without a state on the chip do."""
import numpy as np
import pytest

from flursys_b200 import _abi
from flursys_b200.solver import _Handle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("env", [{}, {"FLURSYS_2D_CLUSTER": "0", "FLURSYS_PCG_RESIDENT": "grid"}, {"FLURSYS_PCG_RESIDENT": "stream"}])
@pytest.mark.parametrize("shape,iters", [((12, 12), 200), ((12, 12), 2000), ((24, 24), 2000), ((4, 4, 4), 200), ((6, 5, 4), 2000),
                                         ((12, 12, 12), 2000), ((20, 20, 20), 2000)])
def test_an_unreachable_tolerance_ends_at_the_cap(oracle, monkeypatch, env, shape, iters):
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    c = oracle.default_config(len(shape))
    c.nx, c.ny = shape[:2]
    if len(shape) == 3:
        c.nz = shape[2]
    c.dt = 1e-3
    c.pressure_solver, c.stop_rule, c.precision = _abi.PRESSURE_PCG, _abi.STOP_REL_L2, _abi.PRECISION_MIXED
    c.pressure_rtol, c.pressure_atol, c.pressure_max_iters = 1e-30, 0.0, iters
    c.residual_replacement_every = 50
    h = _Handle(c)
    h.upload(_abi.FIELD_U, 0.1 * np.random.default_rng(1).standard_normal(h.download(_abi.FIELD_U).size))
    rep = h.step(1)
    assert rep.pressure_status == _abi.LINEAR_MAX_ITERATIONS and rep.pressure_iterations <= iters
    # the FP64 residual of an FP64 pressure: its rounding, 2^-53 of |A| |p|, is
    # a few times 1e-16 of the right-hand side times the condition of the grid
    assert rep.pressure_true_relative_residual <= 1e-12
