"""The reciprocal and the quotients of gridreduce.cuh against CUDA's own
division: a small library is compiled from the header and run over random
operands of all normal exponents in their range, both signs, operands next to
powers of two, and operands that are not finite."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from flursys_b200 import build as fb

SOURCE = r"""
#include "gridreduce.cuh"
using namespace flursys;
__global__ void run(int n, const double *a, const double *b, double *o) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double y = fast_recip(b[i]);
        o[i] = y;
        o[n + i] = 1.0 / b[i];
        o[2 * n + i] = quotient(a[i], b[i], y);
        o[3 * n + i] = a[i] / b[i];
        o[4 * n + i] = rounded_quotient(a[i], b[i], 1.0 / b[i]);
    }
}
extern "C" int quotients(int n, const double *a, const double *b, double *o) {
    double *d = nullptr;
    cudaError_t e = cudaMalloc(&d, 7 * sizeof(double) * n);
    if (e == cudaSuccess) e = cudaMemcpy(d, a, sizeof(double) * n, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(d + n, b, sizeof(double) * n, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        run<<<256, 256>>>(n, d, d + n, d + 2 * n);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(o, d + 2 * n, 5 * sizeof(double) * n, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return (int)e;
}
"""


@pytest.fixture(scope="module")
def quotients(tmp_path_factory):
    d = tmp_path_factory.mktemp("quotient")
    (d / "q.cu").write_text(SOURCE)
    subprocess.run([fb._nvcc(), *fb.NVCC_FLAGS, "-shared", "-o", str(d / "q.so"), str(d / "q.cu")], check=True)
    fn = C.CDLL(os.path.join(d, "q.so")).quotients

    def run(a, b):
        a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
        o = np.empty((5, a.size))
        p = [C.c_void_p(t.ctypes.data) for t in (a, b, o)]
        assert fn(C.c_int(a.size), *p) == 0
        return o
    return run


def _ulps(x, y):
    """Distance in representable numbers (finite, of one sign)."""
    return np.abs(x.view(np.int64) - y.view(np.int64))


def _mantissas(rng, n):
    m = 1.0 + rng.random(n)
    near = rng.integers(0, 64, n) * 2.0 ** -52  # next to a power of two, from either side
    return np.where(rng.random(n) < 0.2, 1.0 + near, np.where(rng.random(n) < 0.25, 2.0 - 2.0 ** -52 - near, m))


@pytest.mark.gpu
@pytest.mark.parametrize("span", [4, 60, 480])  # exponents of both operands: the quotient and its remainder stay normal
def test_quotients_against_the_division(quotients, span):
    rng = np.random.default_rng(span)
    n = 4_000_000
    sign = lambda: rng.choice([-1.0, 1.0], n)  # noqa: E731
    a = sign() * np.ldexp(_mantissas(rng, n), rng.integers(-span, span, n))
    b = sign() * np.ldexp(_mantissas(rng, n), rng.integers(-span, span, n))
    y, one, q, div, exact = quotients(a, b)
    # the last iteration's own two roundings, each half a unit of the result or
    # of a term that is no larger, and one for the binade's change
    assert _ulps(y, one).max() <= 2
    assert _ulps(q, div).max() <= 1
    assert np.array_equal(exact, div)


@pytest.mark.gpu
def test_quotients_of_operands_that_are_not_finite(quotients):
    big = 1.7e308
    a = np.array([np.inf, -np.inf, np.nan, 1.0, big, 0.0, -0.0])
    b = np.array([3.0, 3.0, 3.0, np.nan, 0.5, 7.0, 7.0])
    _, _, q, div, exact = quotients(a, b)
    np.testing.assert_array_equal(exact, div)
    assert not np.isfinite(q[:5]).any() and np.all(q[5:] == 0.0)
    _, _, q, div, _ = quotients(np.array([1.0, 0.0]), np.array([0.0, 0.0]))
    assert not np.isfinite(q).any()
