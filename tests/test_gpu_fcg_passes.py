"""The FCG's smoothing and operator passes (fcg3d.cu) on grids of two vectors
per row, of one and of several blocks, and of plane counts that end inside a
block's march: a step against the FP64 oracle."""
import numpy as np
import pytest

from flursys_b200 import _abi
from flursys_b200.learned import DEFAULT_WEIGHTS
from flursys_b200.solver import _Handle

from .test_gpu_cavity3d import FIELDS, MIXED_TOL, cfg3d
from .test_gpu_pcg3d_variants import _vel_rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(8, 8, 8), (8, 40, 24), (72, 8, 16), (16, 24, 136), (40, 48, 56)])
def test_fcg_step_matches_the_fp64_oracle(oracle, shape):
    nx, ny, nz = shape
    u = 0.1 * np.random.default_rng(5).standard_normal((nx + 1) * ny * nz)
    ref = oracle.OracleSolver(cfg3d(oracle, *shape, rtol=1e-12))
    ref.set(_abi.FIELD_U, u)
    ref.step(1)
    cfg = cfg3d(oracle, *shape, solver=_abi.PRESSURE_FCG, rtol=1e-8, precision=_abi.PRECISION_MIXED)
    cfg.fcg_weights_path = str(DEFAULT_WEIGHTS).encode()
    g = _Handle(cfg)
    g.upload(_abi.FIELD_U, u)
    rep = g.step(1)
    assert rep.pressure_status == _abi.LINEAR_CONVERGED
    assert rep.pressure_true_relative_residual <= 1.0e-8 * 1.0001
    assert _vel_rel({fid: g.download(fid) for fid, _ in FIELDS[:3]}, {fid: ref.get(fid) for fid, _ in FIELDS[:3]}) <= MIXED_TOL
