"""HEAT_3D by default on fields that leave a walk's fixed-point window: pulses,
exponential profiles, ramps, waves and single outliers, bit for bit the suite's
arithmetic as numpy rounds it, and no slower than the split by single operations
(tune->tile_x 4, tile_z 6)."""
import ctypes

import numpy as np
import pytest

import rajaperf_gb300 as rp
from tests import gpu_util as gu
from tests.test_gpu_stencil_fixed_point import _heat

pytestmark = pytest.mark.gpu


def _field(kind, n):
    t = np.linspace(0.0, 1.0, n)
    z, y, x = np.meshgrid(t, t, t, indexing="ij")
    if kind == "pulse":
        return np.exp(-400.0 * ((x - 0.5) ** 2 + (y - 0.5) ** 2 + (z - 0.5) ** 2))
    if kind == "profile":
        return np.exp(30.0 * (x + y + z))
    if kind == "steep":
        return np.exp(-0.7 * n * y)  # one binade per row
    if kind == "cliff":
        return np.exp2(-4.0 * np.round(n * y))  # past the window in one row
    if kind == "ramp":
        return 1.0 + 1000.0 * y
    if kind == "wave":
        return np.sin(12.0 * x) * np.cos(9.0 * y) * np.sin(5.0 * z)
    a = np.random.default_rng(n).uniform(0.5, 1.5, (n, n, n))  # outliers
    a[n // 2, n // 3, ::7] = 1e9
    a[n // 3, ::5, n // 2] = -3.0
    a[::6, n // 2, n // 3] = 0.0
    return a


def _run(a, b, steps, tune=None):
    rp.check(rp.b200().b200_polybench_heat_3d(a.data_ptr(), b.data_ptr(), a.shape[0], steps,
                                              ctypes.byref(tune) if tune else None, gu.stream()))


@pytest.mark.parametrize("kind", ["pulse", "profile", "steep", "cliff", "ramp", "wave", "outliers"])
@pytest.mark.parametrize("n", [12, 35, 83, 131, 171])  # 1, 2, 4, 8 and 16 rows per walk
def test_profiles(n, kind):
    a = _field(kind, n)
    b = a.copy()
    da, db = gu.dev(a), gu.dev(b)
    _run(da, db, 2)
    with np.errstate(under="ignore"):
        for _ in range(2):
            _heat(a, b)
    assert np.array_equal(gu.host(da), a)
    assert np.array_equal(gu.host(db), b)


@pytest.mark.parametrize("kind", ["pulse", "profile", "ramp", "wave"])
def test_profiles_take_no_longer_than_single_operations(kind):
    torch = gu.torch_cuda()
    src = gu.dev(_field(kind, 258))
    a, b = src.clone(), src.clone()

    def time(tune):
        times = []
        for _ in range(4):
            a.copy_(src)
            b.copy_(src)
            start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            start.record()
            _run(a, b, 4, tune)
            end.record()
            torch.cuda.synchronize()
            times.append(start.elapsed_time(end))
        return min(times)
    assert time(None) <= time(rp.Tune(tile_x=4, tile_z=6))
