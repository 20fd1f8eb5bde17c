"""CG and Jacobi-PCG of banded CSR matrices on the chip (csr_band.cu) against
the kernel that streams its vectors: row counts around the block size, bands
from none to the whole matrix, rows of equal and of different length, iterates
at the cap, and the failures of both."""
import numpy as np
import pytest

from flursys_b200 import _abi

from .paritylib import rel_l2
from .test_gpu_linear import gpu_solve, poisson_csr

pytestmark = pytest.mark.gpu


def _banded(n, reach, seed, density=0.5):
    """Symmetric, diagonally dominant, entries at random within the band."""
    rng = np.random.default_rng(seed)
    off = {}
    for i in range(n):
        for j in rng.integers(max(0, i - reach), i + 1, size=3):
            if j < i and rng.random() < density:
                off[(i, int(j))] = off[(int(j), i)] = -rng.random()
    rows = [[] for _ in range(n)]
    for (i, j), v in off.items():
        rows[i].append((j, v))
    ro, ci, va = [0], [], []
    for i in range(n):
        r = rows[i] + [(i, 0.05 + rng.random() * 0.01 - sum(v for _, v in rows[i]))]
        for j, v in sorted(r):
            ci.append(j)
            va.append(v)
        ro.append(len(ci))
    return np.array(ro), np.array(ci), np.array(va)


def _poisson(oracle, nx, ny, shift):
    r, c, v = poisson_csr(nx, ny, shift=shift)
    st, ro, ci, va = oracle.csr_build(nx * ny, nx * ny, r, c, v)
    assert st == 0
    return ro, ci, va


def _both(cudalib, monkeypatch, method, mat, rhs, x0, opts):
    out = []
    for env in ("1", "0"):
        monkeypatch.setenv("FLURSYS_CSR_BAND", env)
        out.append(gpu_solve(cudalib, method, *mat, rhs, x0, opts))
    return out


@pytest.mark.parametrize("method", ["cg", "pcg"])
@pytest.mark.parametrize("n,reach", [(1, 0), (2, 1), (127, 3), (128, 127), (129, 40), (300, 0), (515, 514), (5000, 70),
                                     (148 * 128 + 1, 600), (30000, 2000)])
def test_band_form_solves_as_the_streaming_kernel(cudalib, monkeypatch, method, n, reach):
    mat = _banded(n, reach, n)
    rng = np.random.default_rng(n)
    rhs, x0 = rng.standard_normal(n), rng.standard_normal(n)
    (sa, xa, ra), (sb, xb, rb) = _both(cudalib, monkeypatch, method, mat, rhs, x0, _abi.LinearSolverOptions(0.0, 1e-12, 5000))
    assert sa == sb == 0 and ra.status == rb.status == _abi.LINEAR_CONVERGED
    assert abs(ra.iterations - rb.iterations) <= 1 + rb.iterations // 50
    assert ra.initial_residual == pytest.approx(rb.initial_residual, rel=1e-12)
    # two solutions of relative residual 1e-12: 2e-12 cond(A) (1 + |x0| / |x|); the
    # rows' sums are at least 0.05 and their absolute sums at most 2 * 6 + 0.06
    assert rel_l2(xa, xb) <= 2e-12 * 12.1 / 0.05 * (1.0 + np.linalg.norm(x0) / np.linalg.norm(xb))


@pytest.mark.parametrize("method", ["cg", "pcg"])
@pytest.mark.parametrize("shape", [(16, 9), (100, 70), (33, 600), (700, 41)])
@pytest.mark.parametrize("iters", [0, 1, 2, 25])
def test_band_form_iterate_at_the_cap(oracle, cudalib, monkeypatch, method, shape, iters):
    nx, ny = shape
    mat = _poisson(oracle, nx, ny, 0.01)
    rng = np.random.default_rng(nx)
    rhs = rng.standard_normal(nx * ny)
    (sa, xa, ra), (sb, xb, rb) = _both(cudalib, monkeypatch, method, mat, rhs, np.zeros(nx * ny),
                                       _abi.LinearSolverOptions(0.0, 1e-15, iters))
    assert sa == sb == 0 and ra.status == rb.status == _abi.LINEAR_MAX_ITERATIONS
    assert ra.iterations == rb.iterations == iters
    # FP64 rounding of a few hundred operations per iteration
    assert np.linalg.norm(xa - xb) <= 1e-12 * (1 + iters) * max(np.linalg.norm(xb), 1e-300)
    assert ra.final_residual == pytest.approx(rb.final_residual, rel=1e-12 * (1 + iters))


def test_band_form_fails_as_the_streaming_kernel(cudalib, monkeypatch):
    opts = _abi.LinearSolverOptions(0.0, 1e-12, 100)
    n = 200
    ro, ci = np.arange(n + 1), np.arange(n)
    ones = np.ones(n)
    for va, rhs in ((np.full(n, 1e300), np.full(n, 1e300)),           # overflow in the sums
                    (np.full(n, 1e-40), ones),                        # d.q below the breakdown bound
                    (np.where(np.arange(n) % 2, 1.0, -1.0), ones)):   # r.Mr or d.q is 0
        for method in ("cg", "pcg"):
            (sa, _, _), (sb, _, _) = _both(cudalib, monkeypatch, method, (ro, ci, va), rhs, np.zeros(n), opts)
            assert sa == sb and (sa or method == "pcg")  # Jacobi scaling lets some of them converge
