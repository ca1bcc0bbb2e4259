"""FDTD_2D right behind the kernels that write its fields, and calls of it behind
each other, in a stream and in a graph: each launch is set up while its
predecessor runs and has to wait for what it reads.  Bit for bit the same calls
with a synchronization after each."""
import numpy as np
import pytest

import rajaperf_gb300 as rp
from tests import gpu_util as gu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(9, 130), (67, 257), (800, 1025), (2003, 1501)])
def test_fdtd_behind_its_inputs(nx, ny):
    torch = gu.torch_cuda()
    L = rp.b200()
    n, steps = nx * ny, 4
    rng = np.random.default_rng(nx)
    src = [gu.dev(rng.uniform(0.5, 1.5, n)) for _ in range(3)]
    fict = gu.dev(rng.uniform(0.5, 1.5, steps))
    f = torch.zeros_like(fict)
    wb = L.b200_fdtd_2d_workspace_bytes(nx, ny)
    ws = torch.zeros(wb, dtype=torch.uint8, device="cuda")

    def run(fields, wait):
        s = torch.cuda.current_stream().cuda_stream
        for a, b in zip(fields + [f], src + [fict]):
            rp.check(L.b200_stream_copy(b.data_ptr(), a.data_ptr(), a.numel(), None, s))
            wait()
        for _ in range(3):
            rp.check(L.b200_polybench_fdtd_2d_ws(*[t.data_ptr() for t in fields], f.data_ptr(),
                                                 nx, ny, steps, ws.data_ptr(), wb, None, s))
            wait()

    want = [torch.zeros_like(t) for t in src]
    run(want, torch.cuda.synchronize)
    got = [torch.zeros_like(t) for t in src]
    run(got, lambda: None)
    graph_out = [torch.zeros_like(t) for t in src]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run(graph_out, lambda: None)
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    for w, g, h in zip(want, got, graph_out):
        assert np.array_equal(gu.host(g), gu.host(w))
        assert np.array_equal(gu.host(h), gu.host(w))
