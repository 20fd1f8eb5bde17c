"""2D PCG on rows of a few cells: where a block's passes over many short rows
would take longer than an iteration of the streaming kernel that one serves (its
results, bit by bit), elsewhere the chip does."""
import numpy as np
import pytest

from flursys_b200 import _abi
from flursys_b200.solver import _Handle

from .test_gpu_cavity2d import cfg2d

pytestmark = pytest.mark.gpu

F64, MIXED = _abi.PRECISION_F64, _abi.PRECISION_MIXED


def _iterate(oracle, monkeypatch, env, shape, precision, iters):
    monkeypatch.setenv("FLURSYS_2D_RESIDENT", env)
    c = cfg2d(oracle, *shape, dt=1e-9, precision=precision)
    c.stop_rule, c.pressure_atol, c.pressure_rtol, c.pressure_max_iters = _abi.STOP_REL_L2, 0.0, 1e-30, iters
    c.residual_replacement_every = 50
    h = _Handle(c)
    h.upload(_abi.FIELD_U, 0.1 * np.random.default_rng(2).standard_normal((shape[0] + 1) * shape[1]))
    assert h.step(1).pressure_iterations == iters
    return h.download(_abi.FIELD_PRESSURE)


@pytest.mark.parametrize("shape,precision", [((4, 100000), F64), ((4, 100000), MIXED), ((6, 100000), F64), ((6, 60000), MIXED),
                                             ((4, 40000), MIXED)])
def test_long_runs_of_short_rows_stream(oracle, monkeypatch, shape, precision):
    assert np.array_equal(_iterate(oracle, monkeypatch, "1", shape, precision, 20),
                          _iterate(oracle, monkeypatch, "0", shape, precision, 20))


@pytest.mark.parametrize("shape", [(4, 700), (4, 2000), (4, 5000), (4, 10000), (5, 6001), (16, 20000), (33, 10000)])
def test_short_rows_on_the_chip(oracle, monkeypatch, shape):
    a, b = (_iterate(oracle, monkeypatch, env, shape, F64, 20) for env in ("1", "0"))
    assert not np.array_equal(a, b)  # another form
    # 20 iterations of FP64 rounding (1e-16 of terms that cancel by the grid's weights, at most 1e4)
    assert np.linalg.norm(a - b) <= 1e-10 * np.linalg.norm(b)
