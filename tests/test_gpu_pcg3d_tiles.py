"""The tile-resident 3D PCG (pcg3d_res.cu, MIXED), which small grids reach by
FLURSYS_PCG_RESIDENT=tiles and grids between the row form and one tile per SM by
default: against the FP64 oracle, single- against two-reduction form, FP32
column sums, the maximum norm, the iteration cap and an injected fault. Only the
single-reduction tile kernel reports the time that block 0 waits inside grid
barriers, which shows that it is the one that ran."""
import ctypes as C

import numpy as np
import pytest

from flursys_b200 import _abi
from flursys_b200.solver import SolverError, _Handle

from .test_gpu_cavity3d import FIELDS, MIXED_TOL, cfg3d
from .test_gpu_pcg3d_variants import _vel_rel

pytestmark = pytest.mark.gpu


def _runs_tiles(h, single=True):
    ph = (C.c_double * 6)()
    h.lib.flursys_cuda_solver_profile(h.h, ph, 6)
    return h.solve_kind() == _abi.SOLVE_RESIDENT and (ph[4] > 0.0) == single


def _run(oracle, monkeypatch, form, shape, steps, rtol=1e-8, max_iters=20000, rule=_abi.STOP_REL_L2):
    if form is None:
        monkeypatch.delenv("FLURSYS_PCG_RESIDENT", raising=False)
    else:
        monkeypatch.setenv("FLURSYS_PCG_RESIDENT", form)
    cfg = cfg3d(oracle, *shape, rtol=rtol, precision=_abi.PRECISION_MIXED, rule=rule)
    cfg.pressure_max_iters = max_iters
    if rule != _abi.STOP_REL_L2:
        cfg.pressure_tolerance = rtol
    h = _Handle(cfg)
    reps = [h.step(1) for _ in range(steps)]
    return reps, {fid: h.download(fid) for fid, _ in FIELDS}, h


def _close(a, b):
    """Counts of two MIXED solves that differ in rounding (see test_gpu_pcg3d_resident)."""
    return abs(a - b) <= 3 + max(a, b) // 25


@pytest.mark.parametrize("shape,dots", [((32, 32, 32), "64"), ((48, 40, 36), "64"), ((20, 70, 9), "64"),
                                        ((64, 96, 50), "64"), ((33, 65, 31), "64"), ((33, 65, 31), "32")])
def test_tiles_against_fp64_oracle(oracle, monkeypatch, shape, dots):
    monkeypatch.setenv("FLURSYS_PCG_RES_DOTS", dots)
    ref = oracle.OracleSolver(cfg3d(oracle, *shape, rtol=1e-8))
    ref_reps = [ref.step(1) for _ in range(4)]
    reps, fields, h = _run(oracle, monkeypatch, "tiles", shape, 4)
    assert _runs_tiles(h)
    for a, b in zip(reps, ref_reps):
        assert a.pressure_status == _abi.LINEAR_CONVERGED
        assert a.pressure_true_relative_residual <= 1.0e-8 * 1.0001
        assert b.pressure_iterations - 3 <= a.pressure_iterations
        assert a.pressure_iterations <= b.pressure_iterations + 50 + b.pressure_iterations // 4
    assert _vel_rel(fields, {fid: ref.get(fid) for fid, _ in FIELDS[:3]}) <= MIXED_TOL


@pytest.mark.parametrize("shape", [(48, 40, 32), (64, 96, 50)])
def test_single_and_two_reduction_tiles_agree(oracle, monkeypatch, shape):
    one, f1, g1 = _run(oracle, monkeypatch, "tiles", shape, 3)
    two, f2, g2 = _run(oracle, monkeypatch, "2", shape, 3)
    assert _runs_tiles(g1) and _runs_tiles(g2, single=False)
    for a, b in zip(one, two):
        assert a.pressure_status == b.pressure_status == _abi.LINEAR_CONVERGED
        assert a.pressure_true_relative_residual <= 1.0e-8 * 1.0001
        assert _close(a.pressure_iterations, b.pressure_iterations)
    assert _vel_rel(f1, f2) <= MIXED_TOL


def test_tiles_stop_by_the_maximum_norm(oracle, monkeypatch):
    shape = (40, 36, 28)
    cfg = cfg3d(oracle, *shape, rule=_abi.STOP_ABS_INF)
    cfg.pressure_tolerance = 1e-7
    ref = oracle.OracleSolver(cfg)
    ref_reps = [ref.step(1) for _ in range(3)]
    reps, fields, h = _run(oracle, monkeypatch, "tiles", shape, 3, rtol=1e-7, rule=_abi.STOP_ABS_INF)
    assert _runs_tiles(h, single=False)
    for a, b in zip(reps, ref_reps):
        assert a.pressure_status == _abi.LINEAR_CONVERGED
        assert b.pressure_iterations - 3 <= a.pressure_iterations <= b.pressure_iterations + 50 + b.pressure_iterations // 4
    assert _vel_rel(fields, {fid: ref.get(fid) for fid, _ in FIELDS[:3]}) <= MIXED_TOL


@pytest.mark.parametrize("form", ["tiles", "2"])
def test_tiles_at_the_iteration_cap(oracle, monkeypatch, form):
    reps, fields, h = _run(oracle, monkeypatch, form, (32, 32, 32), 1, rtol=1e-12, max_iters=37)
    assert _runs_tiles(h, single=form == "tiles")
    assert reps[0].pressure_status == _abi.LINEAR_MAX_ITERATIONS
    assert reps[0].pressure_iterations == 37
    assert all(np.isfinite(v).all() for v in fields.values())


@pytest.mark.parametrize("form", ["tiles", "2"])
def test_tiles_report_a_barrier_timeout(oracle, monkeypatch, cudalib, form):
    _, _, h = _run(oracle, monkeypatch, form, (32, 32, 32), 1)
    assert _runs_tiles(h, single=form == "tiles")
    assert cudalib.flursys_cuda_debug_inject_barrier_fault(1) == 0
    with pytest.raises(SolverError) as e:
        h.step(1)
    assert e.value.status == _abi.ERR_TIMEOUT and "timed out" in str(e.value)
    assert h.step(1).pressure_status == _abi.LINEAR_CONVERGED


def test_tiles_are_the_default_between_rows_and_streaming(oracle, monkeypatch):
    shape = (192, 128, 96)
    reps, fields, h = _run(oracle, monkeypatch, None, shape, 1)
    assert _runs_tiles(h)
    other, ref, g = _run(oracle, monkeypatch, "stream", shape, 1)
    assert g.solve_kind() == _abi.SOLVE_PERSISTENT
    for r in (reps[0], other[0]):
        assert r.pressure_status == _abi.LINEAR_CONVERGED
        assert r.pressure_true_relative_residual <= 1.0e-8 * 1.0001
    assert _close(reps[0].pressure_iterations, other[0].pressure_iterations)
    assert _vel_rel(fields, ref) <= MIXED_TOL
