"""Chip-resident 3D SOR in its cluster form, on slabs of one, two and three
planes (and a last one of one plane, which runs ahead of its neighbour): the
residual that stops it is that of the fields it returns, so the sweep count,
the residual and the fields do not depend on how the blocks interleave."""
import numpy as np
import pytest

from .test_gpu_sor_resident import _sor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(40, 40, 16), (72, 40, 16), (36, 36, 32), (48, 48, 40)])
def test_cluster_sor_repeats_bit_by_bit(oracle, monkeypatch, shape):
    monkeypatch.setenv("FLURSYS_SOR_RESIDENT", "0")
    p0, r0 = _sor(oracle, shape, 4000, 8.0)
    monkeypatch.setenv("FLURSYS_SOR_RESIDENT", "1")
    runs = [_sor(oracle, shape, 4000, 8.0) for _ in range(6)]
    p1, r1 = runs[0]
    for p, r in runs[1:]:
        assert r.pressure_iterations == r1.pressure_iterations
        assert r.pressure_residual == r1.pressure_residual
        assert np.array_equal(p, p1)
    # against the streaming sweeps, to the rounding that a quotient may differ by
    assert r1.pressure_iterations == r0.pressure_iterations and 1 < r0.pressure_iterations < 4000
    assert np.max(np.abs(p1 - p0)) <= 1e-12 * np.max(np.abs(p0))
