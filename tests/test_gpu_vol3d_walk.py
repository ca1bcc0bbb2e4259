"""VOL3D's default kernel (threads walk zones jp apart) at ranges that end
inside a walk, with short and odd rows, on either side of its size rule."""
import numpy as np
import pytest

import oracle
import rajaperf_gb300 as rp
from tests import gpu_util as gu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("jp,rows,planes,skip", [(1, 3, 3, 0), (5, 7, 6, 3), (33, 9, 8, 1),
                                                 (104, 104, 30, 7), (71, 73, 75, 11)])
def test_vol3d_ranges(jp, rows, planes, skip):
    rng = np.random.default_rng(jp)
    kp = jp * rows
    nn = kp * planes
    i = np.arange(nn)
    x = 0.3 * (i % jp + rng.uniform(-0.1, 0.1, nn))
    y = 0.2 * (i // jp % rows + rng.uniform(-0.1, 0.1, nn))
    z = 0.1 * (i // kp + rng.uniform(-0.1, 0.1, nn))
    ib, ie = skip, nn - kp - jp - 1 - skip
    want = np.full(nn, 5.0)
    dv, dx, dy, dz = gu.dev(want), gu.dev(x), gu.dev(y), gu.dev(z)
    rp.check(rp.b200().b200_apps_vol3d(dx.data_ptr(), dy.data_ptr(), dz.data_ptr(),
                                       dv.data_ptr(), 1.0 / 12, jp, kp, ib, ie, None,
                                       gu.stream()))
    oracle.call("oracle_vol3d_rep", x, y, z, want, 1.0 / 12, jp, kp, ib, ie)
    # some 60 roundings of terms no larger than the product of the extents
    size = (np.ptp(x) + 1) * (np.ptp(y) + 1) * (np.ptp(z) + 1)
    assert np.all(np.abs(gu.host(dv) - want) <= 64 * gu.U * size)
