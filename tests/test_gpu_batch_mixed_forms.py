"""A batch whose instances are solved in different ways (resident queue,
cooperative launch of PCG, of SOR) against a handle per instance, whichever of
those that fit the queue are left in it."""
import time

import numpy as np
import pytest

from flursys_b200 import _abi
from flursys_b200.solver import BatchedIncompressibleSolver, _Handle

from .test_gpu_cavity2d import cfg2d

pytestmark = pytest.mark.gpu

STEPS = 2


def _cfg(oracle, nx, ny, solver=_abi.PRESSURE_PCG):
    c = cfg2d(oracle, nx, ny, dt=1e-4)
    c.pressure_solver = solver
    c.max_steps = c.minimum_steps = 1 << 40
    if solver == _abi.PRESSURE_SOR:
        c.pressure_max_iters = 60
    else:
        c.stop_rule = _abi.STOP_REL_L2
        c.pressure_atol, c.pressure_rtol = 0.0, 1e-12
    return c


@pytest.mark.parametrize("sizes", [
    [(344, 350), (40, 40)],                          # too large for the queue, and one that would fit
    [(330, 330), (16, 24), (344, 350), (96, 8)],     # the largest that fits, small ones, odd ones
    [(24, 20, "sor"), (30, 30), (64, 48)],           # SOR is never queued
    [(344, 350), (20, 20), (24, 20, "sor")] + [(64, 64)] * 9,
    [(16, 16)] * 40,                                 # many small ones
    [(200, 200)] * 2 + [(16, 16)] * 40 + [(4, 300)] * 3,
])
def test_batch_of_queued_and_shared_instances(oracle, sizes):
    cfgs = [_cfg(oracle, s[0], s[1], _abi.PRESSURE_SOR if len(s) == 3 else _abi.PRESSURE_PCG) for s in sizes]
    b = BatchedIncompressibleSolver(cfgs, autotune=False)
    b.advance(STEPS)
    for i, c in enumerate(cfgs):
        assert b.status(i) == _abi.OK
        h = _Handle(c)
        rep = h.step(STEPS)
        assert b.report(i).pressure_status == rep.pressure_status
        u, v = h.download(_abi.FIELD_U), h.download(_abi.FIELD_V)
        # a projection whose residual is 1e-12 of rhs = div u* / dt leaves the
        # velocity off by at most 1e-12 |div u*| / pi with |div u*| <= 2 n |u*|:
        # 2.3e-10 of |u| at n = 350, for two solves and two steps 1e-9
        scale = max(np.linalg.norm(u), np.linalg.norm(v))
        assert np.linalg.norm(b.field(i, "u") - u) <= 1e-9 * scale
        assert np.linalg.norm(b.field(i, "v") - v) <= 1e-9 * scale
        h.close()


def test_many_small_instances_run_at_a_time(oracle):
    # each instance has little work and many barriers, and all fit the chip
    # together: eight times as many may not take three times as long (one after
    # another on a few clusters they took six times as long)
    def step_seconds(count):
        cfgs = [_cfg(oracle, 16, 16) for _ in range(count)]
        for c in cfgs:
            c.dt, c.pressure_rtol = 1e-3, 1e-8
        b = BatchedIncompressibleSolver(cfgs, autotune=False)
        seconds = []
        for _ in range(8):
            start = time.perf_counter()
            b.advance(1)
            seconds.append(time.perf_counter() - start)
            assert b.status(count - 1) == _abi.OK and b.report(count - 1).pressure_iterations > 20
        return min(seconds)

    assert step_seconds(128) <= 3.0 * step_seconds(16)
