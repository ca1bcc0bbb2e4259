"""Calls of chained kernels that do not fill the chip, replayed as a graph: the
overlapped launches leave each grid spread over all SMs, so half the points or
fewer take clearly less time (they took 0.89 and 0.97 of it while a grid's CTAs
were placed beside its predecessor's)."""
import pytest

import rajaperf_gb300 as rp
from tests import gpu_util as gu

pytestmark = pytest.mark.gpu


def _per_call(call, calls=20):
    torch = gu.torch_cuda()
    call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for _ in range(calls):
            call()
    graph.replay()
    times = []
    for _ in range(5):
        start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        start.record()
        graph.replay()
        end.record()
        torch.cuda.synchronize()
        times.append(start.elapsed_time(end))
    return min(times) / calls


def _fields(n, count):
    torch = gu.torch_cuda()
    return [torch.rand(n, dtype=torch.float64, device="cuda") + 0.5 for _ in range(count)]


def _hydro(m):
    f = _fields(m * m, 11)
    return _per_call(lambda: rp.check(rp.b200().b200_lcals_hydro_2d(
        *[t.data_ptr() for t in f], 0.0041, 0.0037, m, m, None, gu.stream())))


def _fdtd(m):
    f, fict = _fields(m * m, 3), _fields(8, 1)[0]
    wb = rp.b200().b200_fdtd_2d_workspace_bytes(m, m)
    ws = gu.torch_cuda().zeros(wb, dtype=gu.torch_cuda().uint8, device="cuda")
    return _per_call(lambda: rp.check(rp.b200().b200_polybench_fdtd_2d_ws(
        *[t.data_ptr() for t in f], fict.data_ptr(), m, m, 8, ws.data_ptr(), wb, None,
        gu.stream())), 5)


@pytest.mark.parametrize("time,small,large", [(_hydro, 200, 350), (_fdtd, 500, 700)])
def test_fewer_points_take_less_time(time, small, large):
    assert time(small) <= 0.8 * time(large)
