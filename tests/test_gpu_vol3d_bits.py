"""VOL3D's default kernel (threads walk zones jp apart) gives the bits of the map
kernel (any tuned block size): the same contractions, whatever the range."""
import ctypes

import numpy as np
import pytest

import rajaperf_gb300 as rp
from tests import gpu_util as gu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("jp,rows,planes", [(1, 3, 3), (5, 7, 6), (33, 9, 8), (72, 72, 72)])
def test_vol3d_as_the_map_kernel(jp, rows, planes):
    torch = gu.torch_cuda()
    rng = np.random.default_rng(jp)
    kp = jp * rows
    n = kp * planes
    x, y, z = (gu.dev(rng.uniform(-1.0, 1.0, n)) for _ in range(3))
    out = []
    for tune in (None, rp.Tune(block_size=256)):
        v = torch.full((n,), 5.0, dtype=torch.float64, device="cuda")
        rp.check(rp.b200().b200_apps_vol3d(x.data_ptr(), y.data_ptr(), z.data_ptr(), v.data_ptr(),
                                           1.0 / 12, jp, kp, 1, n - kp - jp - 1,
                                           ctypes.byref(tune) if tune else None, gu.stream()))
        out.append(gu.host(v).view(np.int64))
    assert np.array_equal(*out)
