"""3MM's products on the tensor cores (dgemm_tc): every element within the
error bound of a chain of FP64 FMAs, k * u * sum |a||b|, at sizes around its
128 x 32 tiles and k steps of 32, for values that it cuts exactly, cuts off, or
hands to the FP64 pipe."""
import ctypes

import numpy as np
import pytest

import rajaperf_gb300 as rp
from tests import gpu_util as gu

pytestmark = pytest.mark.gpu


def _values(kind, shape, rng):
    x = rng.uniform(-1.0, 1.0, shape)
    if kind == "positive":
        return np.abs(x)
    if kind == "integers":
        return np.round(100.0 * x)
    if kind == "scaled":  # rows and columns of very different size
        return x * np.exp(30.0 * rng.standard_normal((shape[0], 1)))
    if kind == "wide":
        return x * np.exp(10.0 * rng.standard_normal(shape))
    if kind == "sparse":
        return np.where(rng.uniform(size=shape) < 0.9, 0.0, x)
    if kind == "zero rows":
        x[::3] = 0.0
        return x
    if kind == "huge":
        return x * 2.0 ** 450
    if kind == "tiny":
        return x * 2.0 ** -450
    return x


def _mm3(mats, dims, tune=None):
    ni, nj, nk, nl, nm = dims
    torch = gu.torch_cuda()
    ins = [gu.dev(np.ascontiguousarray(m).ravel()) for m in mats]
    outs = [torch.full((r * c,), 7.0, dtype=torch.float64, device="cuda")
            for r, c in ((ni, nj), (nj, nl), (ni, nl))]
    rp.check(rp.b200().b200_polybench_3mm(*[t.data_ptr() for t in ins + outs], *dims,
                                          ctypes.byref(tune) if tune else None, gu.stream()))
    return [gu.host(t).reshape(s) for t, s in zip(outs, ((ni, nj), (nj, nl), (ni, nl)))]


def _shapes(dims):
    ni, nj, nk, nl, nm = dims
    return (ni, nk), (nk, nj), (nj, nm), (nm, nl)


@pytest.mark.parametrize("kind", ["uniform", "positive", "integers", "scaled", "wide", "sparse",
                                  "zero rows", "huge", "tiny"])
@pytest.mark.parametrize("dims", [(128, 32, 32, 32, 32), (32, 33, 32, 31, 40),
                                  (127, 65, 63, 129, 64), (129, 97, 96, 130, 161),
                                  (257, 100, 1000, 40, 33), (1, 1100, 40, 1200, 35)])
def test_products_within_the_fma_chain_bound(dims, kind):
    rng = np.random.default_rng(dims[0])
    mats = [_values(kind, s, rng) for s in _shapes(dims)]
    E, F, G = _mm3(mats, dims)
    beyond = kind in ("huge", "tiny")  # G's products leave FP64's range: as the FP64 pipe has them
    if beyond:
        assert np.array_equal(G, _mm3(mats, dims, rp.Tune(algo=1))[2], equal_nan=True)
    for got, (a, b) in ((E, mats[:2]), (F, mats[2:]), (G, (E, F)))[:2 if beyond else 3]:
        al, bl = a.astype(np.longdouble), b.astype(np.longdouble)
        bound = (a.shape[1] + 1) * gu.U * (np.abs(al) @ np.abs(bl))
        assert np.all(np.abs(got - al @ bl) <= bound)
        if kind == "integers" and got is not G:
            assert np.array_equal(got, (al @ bl).astype(np.float64))


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_non_finite_values(bad):
    dims = (200, 70, 90, 50, 64)
    rng = np.random.default_rng(5)
    mats = [_values("uniform", s, rng) for s in _shapes(dims)]
    mats[0][150, 3] = bad
    mats[3][10, 20] = bad
    got, want = _mm3(mats, dims), _mm3(mats, dims, rp.Tune(algo=1))
    for g, w in zip(got, want):
        assert np.array_equal(np.isnan(g), np.isnan(w))
        assert np.array_equal(g[np.isinf(w)], w[np.isinf(w)])
        ok = np.isfinite(w)
        assert np.array_equal(ok, np.isfinite(g))
        assert np.linalg.norm(g[ok] - w[ok]) <= 1e-14 * np.linalg.norm(w[ok])


@pytest.mark.parametrize("k", [4096, 4097])
def test_largest_inner_dimension(k):
    """All digits at their largest: the sums reach the bound of exactness."""
    dims = (40, 36, k, 33, 40)
    mats = [np.full(s, 2.0 - 2.0 ** -52) for s in _shapes(dims)]
    E, F, _ = _mm3(mats, dims)
    x = np.longdouble(2.0 - 2.0 ** -52)
    assert np.all(np.abs(E - k * x * x) <= (k + 1) * gu.U * float(k * x * x))
    assert np.all(np.abs(F - 40 * x * x) <= 41 * gu.U * float(40 * x * x))


def test_more_accurate_than_the_fp64_pipe():
    dims = (300, 310, 1000, 290, 305)
    rng = np.random.default_rng(9)
    mats = [_values("uniform", s, rng) for s in _shapes(dims)]
    want = mats[0].astype(np.longdouble) @ mats[1].astype(np.longdouble)
    err = [float(np.linalg.norm((_mm3(mats, dims, t)[0] - want).astype(np.float64)))
           for t in (None, rp.Tune(algo=1))]
    assert err[0] <= err[1]


def test_products_that_share_memory():
    """F over A, which E has read by then."""
    dims = (96, 64, 96, 96, 50)
    ni, nj, nk, nl, nm = dims
    rng = np.random.default_rng(3)
    mats = [_values("uniform", s, rng) for s in _shapes(dims)]
    want = _mm3(mats, dims)
    torch = gu.torch_cuda()
    a, b, c, d = (gu.dev(m.ravel()) for m in mats)
    e, g = (torch.zeros(r * k, dtype=torch.float64, device="cuda") for r, k in ((ni, nj), (ni, nl)))
    rp.check(rp.b200().b200_polybench_3mm(*[t.data_ptr() for t in (a, b, c, d, e, a, g)], *dims,
                                          None, gu.stream()))
    assert np.array_equal(gu.host(e).reshape(ni, nj), want[0])
    assert np.array_equal(gu.host(a)[:nj * nl].reshape(nj, nl), want[1])
    assert np.array_equal(gu.host(g).reshape(ni, nl), want[2])
