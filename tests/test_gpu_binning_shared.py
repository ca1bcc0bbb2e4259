"""HISTOGRAM and MULTI_REDUCE on either side of their kernels' bin counts and
lengths, for random bins, runs of one bin and single-bin data, items outside
the bins among them.  Counts are exact; sums are within the bound of any order
of FP64 adds."""
import numpy as np
import pytest

import rajaperf_gb300 as rp
from tests import gpu_util as gu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", ["random", "runs", "one"])
@pytest.mark.parametrize("n,nb", [(1 << 18, 96), ((1 << 18) - 1, 97), (1 << 18, 97),
                                  (300001, 1171), (300001, 1172), (1 << 19, 2048),
                                  (1 << 19, 2049), (1100003, 16384), (1100003, 16385),
                                  (7200001, 28000), (7200001, 28001), (3600007, 55000),
                                  (3600007, 55001)])
def test_bins(n, nb, layout):
    L, torch = rp.b200(), gu.torch_cuda()
    rng = np.random.default_rng(nb)
    b = {"random": rng.integers(0, nb, n), "runs": np.arange(n) * nb // n,
         "one": np.full(n, nb - 1)}[layout]
    b[rng.integers(0, n, 50)] = -1
    b[rng.integers(0, n, 50)] = nb
    x = rng.uniform(-0.5, 1.5, n)
    inside = (b >= 0) & (b < nb)
    db, dx = gu.dev(b), gu.dev(x)
    c0, s0 = gu.dev(np.full(nb, 3, dtype=np.int64)), gu.dev(np.full(nb, 0.25))
    c = torch.zeros(nb, dtype=torch.int64, device="cuda")
    s = torch.zeros(nb, dtype=torch.float64, device="cuda")
    wb = max(L.b200_multi_reduce_workspace_bytes(n, nb), 256)
    ws = torch.zeros(wb, dtype=torch.uint8, device="cuda")
    rp.check(L.b200_algorithm_histogram(db.data_ptr(), n, nb, c0.data_ptr(), c.data_ptr(), None,
                                        gu.stream()))
    rp.check(L.b200_basic_multi_reduce(db.data_ptr(), dx.data_ptr(), n, nb, s0.data_ptr(),
                                       s.data_ptr(), ws.data_ptr(), wb, None, gu.stream()))
    count = np.bincount(b[inside], minlength=nb)
    assert np.array_equal(gu.host(c), 3 + count)
    want = 0.25 + np.bincount(b[inside], weights=x[inside], minlength=nb)
    size = 0.25 + np.bincount(b[inside], weights=np.abs(x[inside]), minlength=nb)
    assert np.all(np.abs(gu.host(s) - want) <= 2 * (count + 16) * gu.U * size)
