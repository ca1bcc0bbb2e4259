"""Chains of dependent calls on one stream: each kernel is set up while its
predecessor runs, so each has to wait for the data it reads.  Every value
is exact in FP64, so results are compared bit for bit with numpy."""
import numpy as np
import pytest

import rajaperf_gb300 as rp
from tests import gpu_util as gu

pytestmark = pytest.mark.gpu

# one element, odd tails of the 16-byte path, tile edges, one CTA per SM and
# many tiles per CTA
SIZES = [1, 2, 3, 511, 512, 2049, 4099, 77824, 77825, 1000003, (1 << 22) + 1]


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("n", SIZES)
def test_stream_chain(n, offset):
    """offset 1: pointers 8 bytes past a 16-byte boundary (scalar path)."""
    torch = gu.torch_cuda()
    L = rp.b200()
    rng = np.random.default_rng(n)
    a0 = rng.integers(-8, 8, n).astype(np.float64)
    full = [torch.full((n + 2,), 77.0, dtype=torch.float64, device="cuda") for _ in range(4)]
    full[0][offset:offset + n] = torch.from_numpy(a0).cuda()
    a, b, c, d = [t.data_ptr() + 8 * offset for t in full]
    dot = torch.zeros(1, dtype=torch.float64, device="cuda")
    wb = L.b200_reduce_workspace_bytes(n, None)
    ws = torch.zeros(wb, dtype=torch.uint8, device="cuda")
    s = gu.stream()
    ra, want = a0.copy(), 0.0
    for _ in range(3):
        rp.check(L.b200_stream_copy(a, c, n, None, s))
        rp.check(L.b200_stream_mul(b, c, 0.5, n, None, s))
        rp.check(L.b200_stream_add(a, b, c, n, None, s))
        rp.check(L.b200_stream_triad(d, b, c, 0.5, n, None, s))
        rp.check(L.b200_stream_dot(d, b, n, 0.0, dot.data_ptr(), ws.data_ptr(), wb, None, s))
        rp.check(L.b200_algorithm_memcpy(d, a, n, None, s))
        rb = 0.5 * ra
        rc = ra + rb
        ra = rb + 0.5 * rc
        want += float(np.sum(ra * rb))
    rp.check(L.b200_algorithm_memset(c, 3.0, n, None, s))
    for t, ref in zip(full, (ra, rb, np.full(n, 3.0), ra)):
        got = gu.host(t)
        assert np.array_equal(got[offset:offset + n], ref)
        rest = np.delete(got, np.arange(offset, offset + n))
        assert np.all(rest == 77.0)  # nothing written outside the arrays
    assert gu.host(dot)[0] == want


@pytest.mark.parametrize("n", SIZES)
def test_in_place_chain(n):
    """100 dependent updates of the same elements, in a graph and out of one."""
    torch = gu.torch_cuda()
    L = rp.b200()
    x = torch.ones(n, dtype=torch.float64, device="cuda")
    y = torch.zeros(n, dtype=torch.float64, device="cuda")
    z = torch.zeros(n, dtype=torch.float64, device="cuda")

    def rep(s):
        rp.check(L.b200_basic_daxpy(y.data_ptr(), x.data_ptr(), 2.0, n, None, s))
        rp.check(L.b200_stream_add(z.data_ptr(), y.data_ptr(), z.data_ptr(), n, None, s))

    for _ in range(50):
        rep(gu.stream())
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for _ in range(10):
            rep(torch.cuda.current_stream().cuda_stream)
    for _ in range(5):
        graph.replay()
    torch.cuda.synchronize()
    assert np.all(gu.host(y) == 200.0)
    assert np.all(gu.host(z) == float(sum(2 * k for k in range(1, 101))))
