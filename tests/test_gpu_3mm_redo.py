"""3MM's tensor-core products where many elements of a tile are computed again in
FP64: up to and beyond the number that one tile takes one by one, and no more
time than a quarter of the FP64 pipe's for values of ordinary distributions."""
import ctypes

import numpy as np
import pytest

import rajaperf_gb300 as rp
from tests import gpu_util as gu

pytestmark = pytest.mark.gpu


def _call(mats, dims):
    torch = gu.torch_cuda()
    ni, nj, nk, nl, nm = dims
    ins = [gu.dev(np.ascontiguousarray(m).ravel()) for m in mats]
    outs = [torch.full((n,), 7.0, dtype=torch.float64, device="cuda")
            for n in (ni * nj, nj * nl, ni * nl)]

    def call(tune=None):
        rp.check(rp.b200().b200_polybench_3mm(*[t.data_ptr() for t in ins + outs], *dims,
                                              ctypes.byref(tune) if tune else None, gu.stream()))
        return outs
    return call


@pytest.mark.parametrize("k,rows", [(40, 1), (40, 15), (40, 16), (40, 17), (40, 128),
                                    (300, 27), (300, 28), (300, 29), (300, 64), (300, 127)])
def test_rows_of_zero_products(k, rows):
    """`rows` rows of A's 128 meet only zeros of B: 32 elements each are 0."""
    rng = np.random.default_rng(k + rows)
    a, b = rng.uniform(-1.0, 1.0, (128, k)), rng.uniform(-1.0, 1.0, (k, 32))
    zero = rng.permutation(128)[:rows]
    a[zero, 1:] = 0.0
    b[0] = 0.0
    dims = (128, 32, k, 32, 32)
    e = gu.host(_call([a, b, np.ones((32, 32)), np.ones((32, 32))], dims)()[0]).reshape(128, 32)
    want = a.astype(np.longdouble) @ b.astype(np.longdouble)
    assert np.all(np.abs(e - want) <=
                  (k + 1) * gu.U * (np.abs(a).astype(np.longdouble) @ np.abs(b)))
    assert np.all(e[zero] == 0.0)


@pytest.mark.parametrize("kind", ["normal", "laplace", "student", "lognormal"])
def test_ordinary_values_stay_on_the_tensor_cores(kind):
    n = 1000
    rng = np.random.default_rng(n)
    draw = {"normal": lambda: rng.standard_normal((n, n)),
            "laplace": lambda: rng.laplace(size=(n, n)),
            "student": lambda: rng.standard_t(3, (n, n)),
            "lognormal": lambda: rng.lognormal(size=(n, n)) * rng.choice([-1.0, 1.0], (n, n))}
    call = _call([draw[kind]() for _ in range(4)], (n,) * 5)
    torch = gu.torch_cuda()

    def time(tune):
        call(tune)
        times = []
        for _ in range(3):
            start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            start.record()
            call(tune)
            end.record()
            torch.cuda.synchronize()
            times.append(start.elapsed_time(end))
        return min(times)
    assert time(None) <= 0.25 * time(rp.Tune(algo=1))
