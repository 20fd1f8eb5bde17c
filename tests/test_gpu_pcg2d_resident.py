"""Chip-resident 2D PCG (pcg2d_res.cu) at the edges of its tiles: rows of one and
of several vectors with every remainder, one row and many per block, cluster
and grid form, with and without solid cells, both stop rules, against the FP64
oracle and against the kernel that streams its state."""
import ctypes as C

import numpy as np
import pytest

from flursys_b200 import _abi
from flursys_b200.solver import _Handle

from .paritylib import rel_l2
from .test_gpu_cavity2d import cfg2d
from .test_oracle_solver import case_cfg

pytestmark = pytest.mark.gpu

# 2D: nx over vector remainders and strip edges, ny below, at and above the
# block counts; 300 x 150 and 700 x 90 use the grid form in FP64
SHAPES = [(4, 4), (5, 67), (67, 5), (33, 31), (129, 6), (31, 17), (66, 130), (256, 9), (300, 150), (700, 90)]


def _stencil(cudalib, nx, ny, precision, rtol, max_iters=20000):
    rng = np.random.default_rng(nx * 1000 + ny)
    rhs = rng.standard_normal(nx * ny)
    rhs -= rhs.mean()
    x = np.zeros(nx * ny)
    rep = _abi.LinearSolveReport()
    opts = _abi.LinearSolverOptions(0.0, rtol, max_iters)
    st = cudalib.flursys_cuda_stencil_pcg(nx, ny, 1, 1.0 / nx, 1.0 / ny, 1.0, _abi.dptr(rhs), _abi.dptr(x), precision,
                                          C.byref(opts), C.byref(rep))
    assert st == 0
    return x, rep


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("precision", [_abi.PRECISION_F64, _abi.PRECISION_MIXED], ids=["f64", "mixed"])
def test_resident_pcg2d_forms_agree_with_the_streaming_kernel(cudalib, monkeypatch, shape, precision):
    rtol = 1e-12 if precision == _abi.PRECISION_F64 else 1e-10
    runs = {}
    for name, env in (("auto", {}), ("grid", {"FLURSYS_2D_CLUSTER": "0"}), ("stream", {"FLURSYS_2D_RESIDENT": "0"})):
        for k, v in env.items():
            monkeypatch.setenv(k, v)
        runs[name] = _stencil(cudalib, *shape, precision, rtol)
        for k in env:
            monkeypatch.delenv(k)
    ref, rep = runs["stream"]
    # ||x - x_ref|| <= 2 rtol cond(A); cond(A) of the Neumann operator is below 4 max(nx, ny)^2
    tol = 2.0 * rtol * 4.0 * max(shape) ** 2
    for name in ("auto", "grid"):
        x, r = runs[name]
        assert r.status == _abi.LINEAR_CONVERGED
        if rep.status != _abi.LINEAR_CONVERGED:
            continue  # CG ends exactly on the smallest grid; the streaming form stops there on r.z = 0 unconverged
        assert rel_l2(x, ref) <= tol, name
        if precision == _abi.PRECISION_F64:
            assert abs(r.iterations - rep.iterations) <= 2 + rep.iterations // 100


@pytest.mark.parametrize("iters", [1, 2, 7, 50, 51])
def test_resident_pcg2d_iterate_at_the_cap(cudalib, monkeypatch, iters):
    # the k-th iterate itself, not only the converged solution
    x, r = _stencil(cudalib, 37, 29, _abi.PRECISION_F64, 0.0, iters)
    monkeypatch.setenv("FLURSYS_2D_RESIDENT", "0")
    ref, q = _stencil(cudalib, 37, 29, _abi.PRECISION_F64, 0.0, iters)
    assert r.iterations == q.iterations == iters and r.status == q.status
    # both forms carry FP64 rounding of a few hundred operations per iteration
    assert rel_l2(x, ref) <= 1e-12 * (1 + iters)


@pytest.mark.parametrize("rule", [_abi.STOP_ABS_INF, _abi.STOP_REL_L2])
@pytest.mark.parametrize("kind,nx,ny", [(_abi.CASE_CYLINDER, 80, 32), (_abi.CASE_BACKWARD_STEP, 70, 17),
                                        (_abi.CASE_CYLINDER, 203, 81), (_abi.CASE_CHANNEL, 45, 19)])
def test_resident_pcg2d_masked_cases_match_oracle(oracle, monkeypatch, kind, nx, ny, rule):
    cfg = case_cfg(oracle, kind, nx, ny)
    cfg.pressure_max_iters = 20000
    cfg.t_end = 100.0
    cfg.stop_rule = rule
    # the absolute part ends steps whose right-hand side is rounding (the oracle
    # breaks down on those)
    cfg.pressure_tolerance, cfg.pressure_atol, cfg.pressure_rtol = 1e-12, 1e-12, 1e-13
    ref = oracle.OracleSolver(cfg)
    ref.step(2)
    for env in ("1", "0"):
        monkeypatch.setenv("FLURSYS_2D_CLUSTER", env)
        g = _Handle(cfg)
        rep = g.step(2)
        assert rep.pressure_status == _abi.LINEAR_CONVERGED
        for fid in (_abi.FIELD_U, _abi.FIELD_V, _abi.FIELD_PRESSURE):
            # the badly conditioned step needs 1e-8, as its other parity test does
            assert rel_l2(g.download(fid), ref.get(fid)) <= (1e-8 if kind == _abi.CASE_BACKWARD_STEP else 1e-10)
