"""Handles of different sizes that run the same kernel with different amounts
of shared memory: one after another, and on two threads at a time (the API
allows handles to run concurrently). A launch must not depend on what another
handle planned or launched in between."""
import threading

import numpy as np
import pytest

from flursys_b200 import _abi
from flursys_b200.solver import BatchedIncompressibleSolver, _Handle

from .test_gpu_cavity2d import cfg2d
from .test_gpu_cavity3d import cfg3d
from .test_gpu_csr_band import _poisson
from .test_gpu_linear import gpu_solve

pytestmark = pytest.mark.gpu

# name: environment, precision, large and small grid
FORMS = {
    "2d cluster f64": ({}, _abi.PRECISION_F64, (128, 128), (96, 80)),
    "2d grid mixed": ({"FLURSYS_2D_CLUSTER": "0"}, _abi.PRECISION_MIXED, (400, 300), (320, 200)),
    "3d rows cluster": ({}, _abi.PRECISION_F64, (30, 30, 32), (20, 24, 16)),
    "3d rows grid": ({"FLURSYS_PCG_RESIDENT": "grid"}, _abi.PRECISION_F64, (75, 62, 51), (60, 40, 30)),
    "3d tiles": ({"FLURSYS_PCG_RESIDENT": "2"}, _abi.PRECISION_MIXED, (64, 96, 100), (64, 64, 20)),
    "3d streaming": ({"FLURSYS_PCG_RESIDENT": "stream"}, _abi.PRECISION_F64, (64, 60, 50), (40, 30, 24)),
    "3d sor cluster": ({}, None, (32, 32, 32), (16, 12, 20)),
    "3d sor grid": ({"FLURSYS_SOR_RESIDENT": "grid"}, None, (32, 32, 32), (16, 12, 20)),
}


def _cfg(oracle, precision, shape, iters):
    if precision is None:
        c = oracle.default_config(3)
        c.nx, c.ny, c.nz = shape
        c.pressure_tolerance = 1e-300
    elif len(shape) == 2:
        c = cfg2d(oracle, *shape, precision=precision)
        c.stop_rule = _abi.STOP_REL_L2
        c.pressure_atol, c.pressure_rtol = 0.0, 1e-30
    else:
        c = cfg3d(oracle, *shape, rtol=1e-30, precision=precision)
    c.pressure_max_iters = iters
    c.max_steps = c.minimum_steps = 1 << 40
    c.t_end = 1e9
    return c


@pytest.mark.parametrize("name", list(FORMS))
def test_a_smaller_handle_does_not_stop_a_larger_one(oracle, monkeypatch, name):
    env, precision, large, small = FORMS[name]
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    a = _Handle(_cfg(oracle, precision, large, 7))
    b = _Handle(_cfg(oracle, precision, small, 7))
    for h in (a, b, a, b, a):
        assert h.step(1).pressure_iterations == 7
    one = a.download(_abi.FIELD_PRESSURE)
    c = _Handle(_cfg(oracle, precision, large, 7))
    c.step(3)
    assert np.array_equal(one, c.download(_abi.FIELD_PRESSURE))


@pytest.mark.parametrize("name", list(FORMS))
def test_two_threads_step_handles_of_different_sizes(oracle, monkeypatch, name):
    env, precision, large, small = FORMS[name]
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    steps, errors = 200, []

    def work(shape):
        try:
            h = _Handle(_cfg(oracle, precision, shape, 2))
            fields = [(f, np.zeros_like(h.download(f)))
                      for f in (_abi.FIELD_U, _abi.FIELD_V, _abi.FIELD_PRESSURE) + ((_abi.FIELD_W,) if len(shape) == 3 else ())]
            for _ in range(steps):
                for f, zero in fields:  # two iterations do not keep a flow stable: each step starts at rest
                    h.upload(f, zero)
                assert h.step(1).pressure_iterations == 2
            h.close()
        except Exception as e:  # noqa: BLE001 - reported by the main thread
            errors.append((shape, repr(e)))

    threads = [threading.Thread(target=work, args=(s,)) for s in (large, small)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors


def test_a_smaller_batch_does_not_stop_a_larger_one(oracle):
    def batch(side):
        return BatchedIncompressibleSolver([_cfg(oracle, _abi.PRECISION_F64, (side, side), 7)], autotune=False)

    a, b = batch(160), batch(24)
    for s in (a, b, a):
        s.advance(1)
    assert a.report(0).pressure_iterations == b.report(0).pressure_iterations == 7


def test_two_threads_solve_banded_matrices(oracle, cudalib):
    opts = _abi.LinearSolverOptions(0.0, 1e-15, 3)
    cases = []
    for nx, ny in ((300, 200), (40, 30)):
        cases.append((_poisson(oracle, nx, ny, 0.01), np.random.default_rng(nx).standard_normal(nx * ny)))
    errors = []

    def work(mat, rhs):
        try:
            for _ in range(60):
                st, _, rep = gpu_solve(cudalib, "cg", *mat, rhs, np.zeros_like(rhs), opts)
                assert st == 0 and rep.iterations == 3
        except Exception as e:  # noqa: BLE001
            errors.append((rhs.size, repr(e)))

    threads = [threading.Thread(target=work, args=c) for c in cases]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
