"""3MM's products on the tensor cores against the FP64 pipe (tune->algo 1) where
rows and columns hold values of very different size: no element may be further
from the exact product than one rounding and what the digits leave out, a
quarter of the unit 2^-53 of the element; elements that the digits do not serve
are FP64 dot products."""
import ctypes

import numpy as np
import pytest

import rajaperf_gb300 as rp
from tests import gpu_util as gu

pytestmark = pytest.mark.gpu


def _first(a, b, tune=None):
    """E = a b of a 3MM call whose other products are small."""
    torch = gu.torch_cuda()
    (ni, nk), nj = a.shape, b.shape[1]
    nl = nm = 32
    ins = [gu.dev(np.ascontiguousarray(m).ravel())
           for m in (a, b, np.ones((nj, nm)), np.ones((nm, nl)))]
    e, f, g = (torch.zeros(n, dtype=torch.float64, device="cuda")
               for n in (ni * nj, nj * nl, ni * nl))
    rp.check(rp.b200().b200_polybench_3mm(*[t.data_ptr() for t in (*ins, e, f, g)],
                                          ni, nj, nk, nl, nm,
                                          ctypes.byref(tune) if tune else None, gu.stream()))
    return gu.host(e).reshape(ni, nj)


def _errors(a, b):
    want = a.astype(np.longdouble) @ b.astype(np.longdouble)
    return want, [(_first(a, b, t) - want).astype(np.float64) for t in (None, rp.Tune(algo=1))]


def _outlier(shape, axis, small, rng):
    """Positive values around `small`, and one 1.0 in every row or column."""
    x = small * rng.uniform(0.5, 1.0, shape)
    x[(slice(None), 0) if axis else (0, slice(None))] = 1.0
    return x


@pytest.mark.parametrize("k,s", [(1000, 10), (1000, 14), (4096, 14), (4096, 17)])
def test_one_large_value_meets_a_small_one(k, s):
    """Row: 1.0 and values near 2^-s; column: 2^-40 opposite the 1.0."""
    rng = np.random.default_rng(k + s)
    a = _outlier((128, k), 1, 2.0 ** -s, rng)
    b = rng.uniform(0.5, 1.0, (k, 32))
    b[0] = 2.0 ** -40
    want, (got, chain) = _errors(a, b)
    assert np.all(np.abs(got) <= 1.26 * gu.U * np.abs(want).astype(np.float64))
    assert np.sqrt(np.mean(got ** 2)) <= np.sqrt(np.mean(chain ** 2))


@pytest.mark.parametrize("k,small", [(1000, 2.0 ** -7.6), (1000, 2.0 ** -7.2), (4096, 2.0 ** -8.6)])
def test_large_values_meet_zeros(k, small):
    """Rows and columns with one 1.0 each, which meets a zero."""
    rng = np.random.default_rng(k)
    a, b = _outlier((130, k), 1, small, rng), _outlier((k, 40), 0, small, rng)
    a[:, 1], b[1] = 1.0, 0.0
    a[:, 0], b[0] = 0.0, 1.0
    want, (got, chain) = _errors(a, b)
    assert np.all(np.abs(got) <= 1.26 * gu.U * np.abs(want).astype(np.float64))
    assert np.sqrt(np.mean(got ** 2)) <= np.sqrt(np.mean(chain ** 2))


@pytest.mark.parametrize("kind", ["uniform", "positive", "normal", "laplace", "student",
                                  "lognormal", "diagonal"])
@pytest.mark.parametrize("k", [32, 100, 1000])
def test_no_less_accurate_than_the_fp64_pipe(k, kind):
    rng = np.random.default_rng(k)

    def values(shape):
        if kind == "positive":
            return rng.uniform(0.0, 1.0, shape)
        if kind == "normal":
            return rng.standard_normal(shape)
        if kind == "laplace":
            return rng.laplace(size=shape)
        if kind == "student":
            return rng.standard_t(3, shape)
        if kind == "lognormal":
            return rng.lognormal(0.0, 2.0, shape) * rng.choice([-1.0, 1.0], shape)
        x = rng.uniform(-1.0, 1.0, shape)
        if kind == "diagonal":
            i = np.arange(min(shape))
            x[i, i] = float(k)
        return x

    _, (got, chain) = _errors(values((256, k)), values((k, 64)))
    assert np.sqrt(np.mean(got ** 2)) <= np.sqrt(np.mean(chain ** 2))


@pytest.mark.parametrize("k", [33, 1000])
def test_digits_are_exact(k):
    """Integers whose products and sums fit in 53 bits, one far above the rest:
    nothing is cut, every digit product that counts is kept."""
    rng = np.random.default_rng(k)
    a = rng.integers(-300, 301, (129, k)).astype(np.float64)
    b = rng.integers(-300, 301, (k, 33)).astype(np.float64)
    a[:, 5], b[7] = 2.0 ** 21, 2.0 ** 20
    want = a.astype(np.longdouble) @ b.astype(np.longdouble)
    assert np.array_equal(_first(a, b), want.astype(np.float64))
