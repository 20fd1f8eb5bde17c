"""Mixed precision of the resident 2D PCG: the step length alpha is applied as
the FP64 number it is. After one iteration the pressure is alpha times the
direction, so that alpha shows as the scale of the pressure against that of the
streaming form (FLURSYS_2D_RESIDENT=0); the FP32 rounding of the two directions'
cells averages out."""
import numpy as np
import pytest

from flursys_b200 import _abi
from flursys_b200.solver import _Handle

from .test_gpu_cavity2d import cfg2d

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(96, 96), (128, 90), (101, 160), (300, 200), (331, 251), (500, 400)])
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_alpha_is_not_rounded_to_32_bits(oracle, monkeypatch, shape, seed):
    p = []
    for env in ("0", "1"):
        monkeypatch.setenv("FLURSYS_2D_RESIDENT", env)
        c = cfg2d(oracle, *shape, dt=1e-4, precision=_abi.PRECISION_MIXED)
        c.residual_replacement_every = 50
        c.stop_rule = _abi.STOP_REL_L2
        c.pressure_atol, c.pressure_rtol = 0.0, 1e-12
        c.pressure_max_iters = 1
        h = _Handle(c)
        h.upload(_abi.FIELD_U, 0.1 * np.random.default_rng(seed).standard_normal((shape[0] + 1) * shape[1]))
        assert h.step(1).pressure_iterations == 1
        p.append(h.download(_abi.FIELD_PRESSURE))
    scale = float(p[1] @ p[0]) / float(p[0] @ p[0])
    # each direction's cells are off by at most 2^-24 of their value, at random:
    # the projection by 2^-24 / sqrt(cells) per form (and alpha, a quotient of
    # sums over the same cells, by as much); five times the sum of four
    assert abs(scale - 1.0) <= 5.0 * 2.0 * 2.0 ** -24 / np.sqrt(shape[0] * shape[1])
