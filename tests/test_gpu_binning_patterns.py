"""HISTOGRAM and MULTI_REDUCE in shared memory where the lanes of a warp hold few
bins: runs of any length and offset, bins in turn, one frequent bin, items
outside the bins among them, aligned and unaligned arrays.  Counts are exact;
sums are within the bound of any order of FP64 adds.  And such data take no
longer than random bins do by more than a small factor: lanes that hit one bin
are summed together instead of repeating each other's adds."""
import numpy as np
import pytest

import rajaperf_gb300 as rp
from tests import gpu_util as gu

pytestmark = pytest.mark.gpu


def _layout(kind, n, nb, rng):
    i = np.arange(n)
    if kind == "random":
        return rng.integers(0, nb, n)
    if kind == "in turn":
        return i % nb
    if kind == "two":
        return i % 2 * (nb // 2)
    if kind == "frequent":
        return np.where(rng.uniform(size=n) < 0.9, nb - 1, rng.integers(0, nb, n))
    if kind == "one":
        return np.full(n, nb - 1)
    return i // int(kind) % nb  # runs


def _calls(b, x, nb, offset=0):
    L, torch = rp.b200(), gu.torch_cuda()
    n = b.size
    db, dx = (gu.dev(np.concatenate([a[:offset], a]))[offset:] for a in (b, x))
    c0, s0 = gu.dev(np.full(nb, 3, dtype=np.int64)), gu.dev(np.full(nb, 0.25))
    c, s = torch.zeros_like(c0), torch.zeros_like(s0)
    wb = max(L.b200_multi_reduce_workspace_bytes(n, nb), 256)
    ws = torch.zeros(wb, dtype=torch.uint8, device="cuda")

    def histogram():
        rp.check(L.b200_algorithm_histogram(db.data_ptr(), n, nb, c0.data_ptr(), c.data_ptr(),
                                            None, gu.stream()))
        return c

    def multi_reduce():
        rp.check(L.b200_basic_multi_reduce(db.data_ptr(), dx.data_ptr(), n, nb, s0.data_ptr(),
                                           s.data_ptr(), ws.data_ptr(), wb, None, gu.stream()))
        return s
    return histogram, multi_reduce


@pytest.mark.parametrize("kind", ["random", "in turn", "two", "frequent", "one", "2", "3", "4",
                                  "7", "20", "31", "130"])
@pytest.mark.parametrize("n,nb,offset", [((1 << 18) + 3, 97, 0), ((1 << 18) + 3, 98, 1),
                                         ((1 << 18) + 1, 749, 0), (1050001, 2999, 1)])
def test_patterns(n, nb, offset, kind):
    rng = np.random.default_rng(nb)
    b = _layout(kind, n, nb, rng)
    b[rng.integers(0, n, 50)] = -1
    b[rng.integers(0, n, 50)] = nb
    x = rng.uniform(-0.5, 1.5, n)
    inside = (b >= 0) & (b < nb)
    histogram, multi_reduce = _calls(b, x, nb, offset)
    count = np.bincount(b[inside], minlength=nb)
    assert np.array_equal(gu.host(histogram()), 3 + count)
    want = 0.25 + np.bincount(b[inside], weights=x[inside], minlength=nb)
    size = 0.25 + np.bincount(b[inside], weights=np.abs(x[inside]), minlength=nb)
    assert np.all(np.abs(gu.host(multi_reduce()) - want) <= 2 * (count + 16) * gu.U * size)


@pytest.mark.parametrize("value", [np.inf, np.nan])
def test_non_finite_values_stay_in_their_bin(value):
    n, nb = 1 << 18, 128
    rng = np.random.default_rng(2)
    for kind in ("random", "two", "frequent", "9"):
        b = _layout(kind, n, nb, rng)
        x = rng.uniform(-0.5, 1.5, n)
        x[n // 3] = value
        got = gu.host(_calls(b, x, nb)[1]())
        assert not np.isfinite(got[b[n // 3]])
        assert np.all(np.isfinite(np.delete(got, b[n // 3])))


def _time(call):
    torch = gu.torch_cuda()
    call()
    times = []
    for _ in range(5):
        start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        start.record()
        call()
        end.record()
        torch.cuda.synchronize()
        times.append(start.elapsed_time(end))
    return min(times)


@pytest.mark.parametrize("which,kind,factor", [
    (0, "two", 1.25), (0, "20", 1.25), (0, "frequent", 1.35),
    (1, "8", 1.25), (1, "20", 1.5)])
def test_few_bins_in_a_warp_cost_little(which, kind, factor):
    n, nb = 1 << 24, 16384
    rng = np.random.default_rng(3)
    x = rng.uniform(size=n)
    random, few = (_time(_calls(_layout(k, n, nb, rng), x, nb)[which]) for k in ("random", kind))
    assert few <= factor * random
