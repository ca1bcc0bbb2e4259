"""The FP64 scan's ring kernel (integer-pipe run totals and prefixes, one
scanner warp for all tiles): sizes at the edges of its 4352-item tiles and of
its scanner's rounds, and values that take each of its ways.  Every prefix is
within (n + 64) * u * sum|x| of the extended-precision one, the bound of any
order of FP64 adds."""
import ctypes

import numpy as np
import pytest

import rajaperf_gb300 as rp
from tests import gpu_util as gu

pytestmark = pytest.mark.gpu

TILE = 4352


def _values(kind, n):
    rng = np.random.default_rng(n)
    x = rng.uniform(0.0, 1.0, n)
    if kind == "negative":
        x = -x
    elif kind == "mixed":  # signs change between and within runs
        x = np.where((np.arange(n) // 4000) % 3 == 1, x - 0.5, x)
    elif kind == "wide":
        x = np.exp(40.0 * rng.standard_normal(n))
    elif kind == "sparse":
        x = np.where(rng.uniform(size=n) < 0.98, 0.0, x)
    elif kind == "growing":
        x = np.exp(np.arange(n) * (1000.0 / n) - 500.0)
    elif kind == "tiny":  # below the integer sums' range, subnormals among them
        x = x * 2.0 ** -1030
    elif kind == "cancel":  # each run's items add up to almost nothing
        x[1::2] = -x[0::2][:x[1::2].size] * (1 + 2.0 ** -50)
    return x


def _scan(x, init):
    L = rp.b200()
    torch = gu.torch_cuda()
    n = x.size
    dx = gu.dev(x)
    dy = torch.zeros(n, dtype=torch.float64, device="cuda")
    wb = L.b200_scan_workspace_bytes(n)
    ws = torch.zeros(wb, dtype=torch.uint8, device="cuda")
    t = rp.Tune(algo=2)
    for _ in range(2):  # the second call finds the first one's descriptors
        rp.check(L.b200_algorithm_scan(dx.data_ptr(), dy.data_ptr(), n, init, ws.data_ptr(), wb,
                                       ctypes.byref(t), gu.stream()))
    assert L.b200_workspace_status(ws.data_ptr(), wb, gu.stream()) == rp.B200_OK
    return gu.host(dy)


@pytest.mark.parametrize("kind", ["uniform", "negative", "mixed", "wide", "sparse", "growing",
                                  "tiny", "cancel"])
@pytest.mark.parametrize("n", [1, 3, 34, 35, 4095, TILE - 1, TILE, TILE + 1, 2 * TILE,
                               129 * TILE + 7, 400 * TILE - 1])
def test_ring_scan_of_values(n, kind):
    x = _values(kind, n)
    xl = x.astype(np.longdouble)
    for init in (0.0, -3.0e6):
        want = init + np.concatenate([[0], np.cumsum(xl)[:-1]])
        size = abs(init) + np.concatenate([[0], np.cumsum(np.abs(xl))[:-1]])
        got = _scan(x, init)
        assert np.all(np.abs(got - want) <= (n + 64) * gu.U * size + 2.0 ** -1074 * n)


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_ring_scan_of_a_non_finite_value(bad):
    n, at = 40 * TILE, 9 * TILE + 17
    x = _values("uniform", n)
    want = np.concatenate([[0], np.cumsum(x)[:-1]])
    x[at] = bad
    got = _scan(x, 0.0)
    assert np.all(np.abs(got[:at + 1] - want[:at + 1]) <= (n + 64) * gu.U * want[:at + 1])
    assert np.array_equal(got[at + 1:], np.full(n - at - 1, bad), equal_nan=True)
