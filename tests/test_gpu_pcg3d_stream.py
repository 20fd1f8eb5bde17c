"""3D PCG that streams its vectors once per iteration (pcg3d_stream.cu) at the
edges of its blocks: rows of one and of several vectors with every remainder,
one and two vector columns per thread, one block and many on each axis, both
precisions and stop rules, against the FP64 oracle and the graph-driven PCG."""
import numpy as np
import pytest

from flursys_b200 import _abi
from flursys_b200.solver import SolverError, _Handle

from .paritylib import rel_l2
from .test_gpu_cavity3d import FIELDS, MIXED_TOL, cfg3d
from .test_gpu_pcg3d_rows import _pressure_tolerance
from .test_gpu_pcg3d_variants import _vel_rel

pytestmark = pytest.mark.gpu

F64, MIXED = _abi.PRECISION_F64, _abi.PRECISION_MIXED
SHAPES = [(5, 7, 4), (6, 67, 4), (66, 5, 33), (33, 31, 17), (17, 40, 48), (131, 20, 24), (258, 33, 9), (63, 64, 65)]
FORMS = ("stream", "0")  # 0: graph-driven


def _step(oracle, monkeypatch, form, shape, precision, rtol, max_iters=20000, rule=_abi.STOP_REL_L2):
    monkeypatch.setenv("FLURSYS_PCG_RESIDENT", form)
    cfg = cfg3d(oracle, *shape, rtol=rtol, precision=precision, rule=rule)
    cfg.pressure_max_iters = max_iters
    if rule != _abi.STOP_REL_L2:
        cfg.pressure_tolerance = rtol
    g = _Handle(cfg)
    nx, ny, nz = shape
    g.upload(_abi.FIELD_U, 0.1 * np.random.default_rng(5).standard_normal((nx + 1) * ny * nz))
    rep = g.step(1)
    assert g.solve_kind() == (_abi.SOLVE_GRAPH if form == "0" else _abi.SOLVE_PERSISTENT)
    return {fid: g.download(fid) for fid, _ in FIELDS}, rep


@pytest.mark.parametrize("shape", SHAPES)
def test_streaming_f64_agrees_with_the_graph_driven_solve(oracle, monkeypatch, shape):
    (f, rep), (ref, q) = [_step(oracle, monkeypatch, form, shape, F64, 1e-12) for form in FORMS]
    p, ref = f[_abi.FIELD_PRESSURE], ref[_abi.FIELD_PRESSURE]
    assert rep.pressure_status == q.pressure_status == _abi.LINEAR_CONVERGED
    assert abs(rep.pressure_iterations - q.pressure_iterations) <= 2 + q.pressure_iterations // 100
    assert rel_l2(p - p.mean(), ref - ref.mean()) <= _pressure_tolerance(shape, 1e-12)


@pytest.mark.parametrize("shape", SHAPES + [(150, 137, 141)])  # the last by the size rule
def test_streaming_mixed_agrees_with_the_graph_driven_solve(oracle, monkeypatch, shape):
    form = "1" if shape[0] == 150 else "stream"
    (f, rep), (ref, q) = [_step(oracle, monkeypatch, m, shape, MIXED, 1e-8) for m in (form, "0")]
    assert rep.pressure_status == q.pressure_status == _abi.LINEAR_CONVERGED
    assert rep.pressure_true_relative_residual <= 1.0e-8 * 1.0001
    # accepted at a replacement, at most one interval later but for rounding
    assert rep.pressure_iterations <= q.pressure_iterations + 50 + q.pressure_iterations // 25
    assert _vel_rel(f, ref) <= MIXED_TOL


@pytest.mark.parametrize("iters", [1, 2, 3, 50, 51])
@pytest.mark.parametrize("shape", [(29, 13, 11), (112, 115, 117)])
def test_streaming_iterate_at_the_cap(oracle, monkeypatch, shape, iters):
    # the k-th iterate itself, not only the converged solution
    (f, rep), (ref, q) = [_step(oracle, monkeypatch, form, shape, F64, 1e-300, iters) for form in FORMS]
    assert rep.pressure_iterations == q.pressure_iterations == iters
    assert rep.pressure_status == q.pressure_status == _abi.LINEAR_MAX_ITERATIONS
    # both forms carry FP64 rounding of a few hundred operations per iteration
    assert rel_l2(f[_abi.FIELD_PRESSURE], ref[_abi.FIELD_PRESSURE]) <= 1e-12 * (1 + iters)


@pytest.mark.parametrize("precision", [F64, MIXED], ids=["f64", "mixed"])
@pytest.mark.parametrize("shape", [(18, 21, 9), (37, 30, 41)])
def test_streaming_max_norm_rule_matches_oracle(oracle, monkeypatch, shape, precision):
    cfg = cfg3d(oracle, *shape, rule=_abi.STOP_ABS_INF)
    cfg.pressure_tolerance = 1e-7
    ref = oracle.OracleSolver(cfg)
    nx, ny, nz = shape
    ref.set(_abi.FIELD_U, 0.1 * np.random.default_rng(5).standard_normal((nx + 1) * ny * nz))
    ref.step(1)
    f, rep = _step(oracle, monkeypatch, "stream", shape, precision, 1e-7, rule=_abi.STOP_ABS_INF)
    assert rep.pressure_status == _abi.LINEAR_CONVERGED and rep.pressure_residual <= 1e-7
    assert _vel_rel(f, {fid: ref.get(fid) for fid, _ in FIELDS[:3]}) <= MIXED_TOL


def test_streaming_timeout_is_reported(oracle, monkeypatch, cudalib):
    monkeypatch.setenv("FLURSYS_PCG_RESIDENT", "stream")
    g = _Handle(cfg3d(oracle, 20, 18, 16, rtol=1e-8, precision=F64))
    assert cudalib.flursys_cuda_debug_inject_barrier_fault(1) == 0
    with pytest.raises(SolverError) as e:
        g.step(1)
    assert e.value.status == _abi.ERR_TIMEOUT
    assert g.step(1).pressure_status == _abi.LINEAR_CONVERGED
