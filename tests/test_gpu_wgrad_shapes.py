"""Gradients of the network at grid sizes that exercise the weight-gradient
kernels' edges: rows shorter than a 16-voxel step, rows of one and of several
pieces with a remainder, fewer pieces than blocks."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
from oracle import fcgnet_oracle as fo  # noqa: E402

from .paritylib import rel_l2  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(8, 8, 8), (24, 16, 8), (40, 8, 16), (72, 8, 8), (136, 8, 8), (16, 32, 24)])
def test_gradient_matches_oracle(dims):
    from flursys_b200 import _abi
    from flursys_b200.learned import FcgNet, init_params
    nx, ny, nz = dims
    params = init_params(5)
    rng = np.random.default_rng(nx)
    p = rng.standard_normal((nz, ny, nx))
    b = fo.lap_neumann(p)
    s = np.sqrt(np.mean(b * b))
    b, p = (b / s).astype(np.float32), (p / s).astype(np.float32)
    norm = float(np.sum(b.astype(np.float64) ** 2))
    net = FcgNet(params)
    g = torch.zeros(params.size, dtype=torch.float32, device="cuda")
    loss = torch.zeros(1, dtype=torch.float64, device="cuda")
    net.train_sample(torch.from_numpy(b.ravel()).cuda(), torch.from_numpy(p.ravel()).cuda(), norm, g, loss, dims,
                     loss_kind=_abi.FCG_LOSS_RESIDUAL)
    l_ref, g_ref = fo.loss_and_grad(params.astype(np.float64), b.astype(np.float64), p.astype(np.float64), norm,
                                    loss="residual")
    assert abs(loss.item() - l_ref) <= 1e-2 * abs(l_ref)
    gd = g.cpu().numpy()
    offs = np.cumsum([0] + [27 * a * c for a, c in zip(fo.CIN, fo.COUT)])
    for layer in range(7):
        sl = slice(offs[layer], offs[layer + 1])
        # BF16 rounding flips between the device's FP32 and the oracle's FP64
        # sums: the bound of the other gradient test
        assert rel_l2(gd[sl], g_ref[sl]) < 3e-2, layer
