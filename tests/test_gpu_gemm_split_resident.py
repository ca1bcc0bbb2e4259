"""The split GEMM's default engine (all digit weights resident, k <= 8192):
bit for bit the paired engine's result wherever the sums are exact, at sizes
around its 128 x 48 tiles and 64-byte blocks of k, and within the bound where
the folded sums leave the integer path."""
import numpy as np
import pytest

from tests.test_gpu_gemm_split import REL_FROB, run_split

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (127, 47, 63), (128, 48, 64), (129, 49, 65),
                                   (130, 128, 128), (256, 145, 129), (70, 257, 1000)])
@pytest.mark.parametrize("alpha,beta", [(1.0, 0.0), (-0.75, 1.25)])
def test_same_bits_as_the_paired_engine(m, n, k, alpha, beta):
    rng = np.random.default_rng(m + n + k)
    A, B, C = rng.uniform(-1, 1, (m, k)), rng.uniform(-1, 1, (k, n)), rng.uniform(-1, 1, (m, n))
    A[0], B[:, -1] = 0.0, 0.0
    A *= np.exp2(rng.integers(-300, 301, m))[:, None]
    assert np.array_equal(run_split(A, B, C, alpha, beta),
                          run_split(A, B, C, alpha, beta, engine=4))


@pytest.mark.parametrize("scale", [-1000, -520, 0, 480])
def test_result_exponents(scale):
    """Results at the ends of the exponent range take the FP64 fold."""
    rng = np.random.default_rng(11)
    A, B = rng.uniform(-1, 1, (40, 90)), rng.uniform(-1, 1, (90, 50))
    A, B, C = A * 2.0 ** scale, B * 2.0 ** (scale // 2), np.zeros((40, 50))
    assert np.array_equal(run_split(A, B, C, 1.0, 0.0), run_split(A, B, C, 1.0, 0.0, engine=4))


@pytest.mark.parametrize("k", [8191, 8192, 8193])
def test_longest_chunk_of_positive_data(k):
    rng = np.random.default_rng(k)
    A, B = rng.uniform(0, 1, (30, k)), rng.uniform(0, 1, (k, 60))
    want = A.astype(np.longdouble) @ B.astype(np.longdouble)
    got = run_split(A, B, np.zeros((30, 60)), 1.0, 0.0)
    assert np.linalg.norm((got - want).astype(np.float64)) <= \
        REL_FROB * np.linalg.norm(want.astype(np.float64))
