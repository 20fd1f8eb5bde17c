"""Chip-resident 3D SOR (sor.cu) against the streaming sweeps: rows of odd and
even length, one plane and several per block, cluster and grid form, at its
sweep cap and at convergence."""
import numpy as np
import pytest

from flursys_b200 import _abi
from flursys_b200.solver import _Handle

pytestmark = pytest.mark.gpu


def _sor(oracle, shape, iters, tol):
    cfg = oracle.default_config(3)
    cfg.nx, cfg.ny, cfg.nz = shape
    cfg.pressure_max_iters = iters
    cfg.pressure_tolerance = tol
    g = _Handle(cfg)
    rng = np.random.default_rng(3)
    nx, ny, nz = shape
    g.upload(_abi.FIELD_U, 0.1 * rng.standard_normal((nx + 1) * ny * nz))
    rep = g.step(1)
    return g.download(_abi.FIELD_PRESSURE), rep


@pytest.mark.parametrize("shape", [(4, 4, 4), (5, 7, 4), (8, 5, 17), (33, 6, 16), (12, 31, 40), (32, 32, 32)])
@pytest.mark.parametrize("iters,tol", [(1, 1e-300), (2, 1e-300), (60, 1e-300), (4000, 1e-4)])
def test_resident_sor_equals_the_streaming_sweeps(oracle, monkeypatch, shape, iters, tol):
    runs = []
    for env in ("0", "1", "grid"):
        monkeypatch.setenv("FLURSYS_SOR_RESIDENT", env)
        runs.append(_sor(oracle, shape, iters, tol))
    (p0, r0) = runs[0]
    for p, r in runs[1:]:
        assert r.pressure_iterations == r0.pressure_iterations and r.pressure_status == r0.pressure_status
        # the same sweeps; a quotient may round the other way now and then
        assert np.max(np.abs(p - p0)) <= 1e-12 * np.max(np.abs(p0))
        assert abs(r.pressure_residual - r0.pressure_residual) <= 1e-9 * max(r0.pressure_residual, 1e-300) + 1e-9
