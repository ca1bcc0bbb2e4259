"""FDTD_2D's one-launch step with its tiles' rows shared by one, two or four
groups of threads (chosen by the number of tiles): bit for bit the two-launch
form, at grids that end inside a tile, a group and a row."""
import ctypes

import numpy as np
import pytest

import rajaperf_gb300 as rp
from tests import gpu_util as gu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(1, 1), (2, 129), (3, 128), (4, 300), (5, 127), (7, 260),
                                   (8, 128), (9, 257), (100, 100), (605, 256), (611, 300),
                                   (1000, 1001), (1217, 1024), (1300, 1100)])
def test_groups_match_the_two_launch_form(nx, ny):
    L, torch, steps = rp.b200(), gu.torch_cuda(), 5
    rng = np.random.default_rng(nx * ny)
    fields = [rng.uniform(0.5, 1.5, nx * ny) for _ in range(3)]
    fict = gu.dev(rng.uniform(0.5, 1.5, steps))
    wb = L.b200_fdtd_2d_workspace_bytes(nx, ny)
    got = []
    for algo in (0, 1):
        ws = torch.zeros(wb, dtype=torch.uint8, device="cuda")
        d = [gu.dev(f) for f in fields]
        t = rp.Tune(algo=algo)
        rp.check(L.b200_polybench_fdtd_2d_ws(*[x.data_ptr() for x in d], fict.data_ptr(), nx, ny,
                                             steps, ws.data_ptr(), wb, ctypes.byref(t),
                                             gu.stream()))
        got.append([gu.host(x) for x in d])
    for a, b in zip(*got):
        assert np.array_equal(a, b)
