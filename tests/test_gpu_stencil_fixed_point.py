"""JACOBI_2D and HEAT_3D by default (their adds in fixed point on the integer
pipes, f64fix): bit for bit the suite's arithmetic as numpy rounds it, at sizes
around the kernels' row counts and blocks and for values inside and outside the
fixed-point window."""
import ctypes

import numpy as np
import pytest

import rajaperf_gb300 as rp
from tests import gpu_util as gu

pytestmark = pytest.mark.gpu


def _values(kind, shape, rng):
    x = rng.uniform(0.5, 1.5, shape)
    if kind == "negative":
        return -x
    if kind == "constant":
        return np.full(shape, 0.3)
    if kind == "mixed":
        return np.where(rng.uniform(size=shape) < 0.02, -x, x)
    if kind == "sparse":
        return np.where(rng.uniform(size=shape) < 0.02, x, 0.0)
    if kind == "wide":
        return x * 2.0 ** rng.integers(-5, 6, shape)
    if kind == "ties":  # last bits set, exponents across the window
        return (1.0 + rng.integers(0, 8, shape) * 2.0 ** -52) * 2.0 ** rng.integers(-3, 4, shape)
    if kind == "huge":
        return x * 2.0 ** 1020
    if kind == "tiny":
        return x * 2.0 ** -1021
    return x


KINDS = ["uniform", "negative", "constant", "mixed", "sparse", "wide", "ties", "huge", "tiny"]


def _jacobi(a, b):
    for s, d in ((a, b), (b, a)):
        d[1:-1, 1:-1] = 0.2 * ((((s[1:-1, 1:-1] + s[1:-1, :-2]) + s[1:-1, 2:]) + s[2:, 1:-1]) +
                               s[:-2, 1:-1])


def _heat(a, b):
    m, u, w = slice(1, -1), slice(2, None), slice(None, -2)
    for s, d in ((a, b), (b, a)):
        c = s[m, m, m]
        t = [0.125 * ((s[hi] - 2.0 * c) + s[lo])
             for hi, lo in (((u, m, m), (w, m, m)), ((m, u, m), (m, w, m)), ((m, m, u), (m, m, w)))]
        d[m, m, m] = ((t[0] + t[1]) + t[2]) + c


def _check(entry, step, shape, kind, steps):
    rng = np.random.default_rng(shape[0])
    a, b = _values(kind, shape, rng), _values(kind, shape, rng)
    da, db = gu.dev(a.ravel()), gu.dev(b.ravel())
    rp.check(entry(da.data_ptr(), db.data_ptr(), shape[0], steps, None, gu.stream()))
    with np.errstate(over="ignore", invalid="ignore"):
        for _ in range(steps):
            step(a, b)
    got_a, got_b = gu.host(da).reshape(shape), gu.host(db).reshape(shape)
    assert np.array_equal(got_a.view(np.int64), a.view(np.int64)) or \
        np.array_equal(got_a, a, equal_nan=True)
    assert np.array_equal(got_b, b, equal_nan=True)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", [3, 4, 5, 129, 130, 259, 1003])
def test_jacobi_fixed_point(n, kind):
    _check(rp.b200().b200_polybench_jacobi_2d, _jacobi, (n, n), kind, 3)


@pytest.mark.parametrize("kind", [k for k in KINDS if k != "tiny"])
@pytest.mark.parametrize("n", [3, 4, 10, 35, 67, 83, 130, 171])
def test_heat_fixed_point(n, kind):
    _check(rp.b200().b200_polybench_heat_3d, _heat, (n, n, n), kind, 2)


@pytest.mark.parametrize("n", [3, 4, 10, 35, 67, 83, 130, 171])
def test_heat_fixed_point_tiny(n):
    """Near the subnormals 0.125 * x is inexact, and the suite's expression as
    nvcc contracts it (an FMA) differs from numpy's two roundings: the
    reference is the kernel with every add on the FP64 pipe."""
    rng = np.random.default_rng(n)
    a, b = (_values("tiny", (n, n, n), rng) for _ in range(2))
    got, want = ([gu.dev(a.ravel()), gu.dev(b.ravel())] for _ in range(2))
    fp64 = rp.Tune(tile_z=1)
    for t, (da, db) in ((None, got), (fp64, want)):
        rp.check(rp.b200().b200_polybench_heat_3d(
            da.data_ptr(), db.data_ptr(), n, 2, ctypes.byref(t) if t else None, gu.stream()))
    for g, w in zip(got, want):
        assert np.array_equal(gu.host(g).view(np.int64), gu.host(w).view(np.int64))
