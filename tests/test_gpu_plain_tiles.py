"""GPU tests of the plain products at the edges of their tiles (32 rows; 8,
16 or 32 columns by size; 8 or 16 inner steps a stage) and of the radius
chains on the integer pipe: entries of every kind, spreads that double the
chains' unit often and take the FP64 steps, subnormal and near-overflow
radii, non-finite entries, odd addresses.  Every bit equals the oracle's."""
import numpy as np
import pytest

from test_gpu_ozaki import mixed_intervals
from vcp_gb300 import pidcuda, vblas
from vcp_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def same(a, b):
    a, b = np.asarray(a), np.asarray(b)
    nan = np.isnan(a) & np.isnan(b)
    return np.array_equal(a.view(np.int64)[~nan], b.view(np.int64)[~nan])


SHAPES = [(1, 17, 1), (31, 18, 7), (32, 33, 8), (33, 40, 9), (70, 65, 130), (20, 300, 40),
          (257, 129, 17), (700, 650, 11), (1100, 1030, 9)]


@pytest.mark.parametrize("m,n,k", SHAPES)
def test_interval_tiles(cuda_lib, oracle, m, n, k):
    rng = np.random.default_rng(m + n + k)
    A = mixed_intervals(rng, m, k)
    A[np.abs(A) > 1e200] = 3.0
    A = np.sort(A.reshape(-1, 2), axis=1).reshape(-1)
    B = W.interval_ephi(rng, k, n, 30, 2.0 ** -20)
    assert same(pidcuda.mulmm(A, B, m, n, k), oracle.pidblas_mulmm(m, n, k, A, B))


@pytest.mark.parametrize("scale", [-1040, -980, 970, 1010])
def test_interval_ends_of_the_range(cuda_lib, oracle, scale):
    rng = np.random.default_rng(abs(scale))
    m, n, k = 40, 20, 150
    A = np.ldexp(W.interval_ephi(rng, m, k, 6, 2.0 ** -10), scale // 2)
    B = np.ldexp(W.interval_ephi(rng, k, n, 6, 2.0 ** -10), scale - scale // 2)
    assert same(pidcuda.mulmm(A, B, m, n, k), oracle.pidblas_mulmm(m, n, k, A, B))


@pytest.mark.parametrize("what", [np.inf, np.nan])
def test_interval_nonfinite(cuda_lib, oracle, what):
    rng = np.random.default_rng(3)
    m, n, k = 35, 24, 50
    A = W.interval_ephi(rng, m, k, 4, 2.0 ** -40)
    B = W.interval_ephi(rng, k, n, 4, 2.0 ** -40)
    A[2 * (3 + 20 * m) + 1] = what
    B[2 * (7 + 2 * k)] = -what
    assert same(pidcuda.mulmm(A, B, m, n, k), oracle.pidblas_mulmm(m, n, k, A, B))


@pytest.mark.parametrize("rnd", [1, -1, 0])
@pytest.mark.parametrize("m,n,k", SHAPES)
def test_point_tiles(cuda_lib, oracle, m, n, k, rnd):
    """vblas naming: A m x k, B k x n here."""
    rng = np.random.default_rng(m * n + k)
    A, B, C = W.ephi(rng, m * k, 8), W.ephi(rng, k * n, 8), np.empty(m * n)
    vblas.rmatmul(m, k, n, A, B, C, rnd)
    assert same(C, oracle.rmatmul(m, k, n, A, B, rnd))


def test_padded_and_odd_addresses(cuda_lib, oracle):
    import torch
    rng = np.random.default_rng(8)
    m, n, k, ld = 45, 35, 70, 50
    A, B = W.interval_ephi(rng, m, k, 4, 2.0 ** -40), W.interval_ephi(rng, k, n, 4, 2.0 ** -40)
    dA = torch.full((2 * ld * k + 1,), float("nan"), dtype=torch.float64, device="cuda")[1:]
    dA.view(k, ld, 2)[:, :m, :] = torch.from_numpy(A.reshape(k, m, 2)).cuda()
    dB = torch.zeros(2 * k * n + 1, dtype=torch.float64, device="cuda")[1:]
    dB.copy_(torch.from_numpy(B))
    C = torch.full((2 * ld * n + 1,), 7.0, dtype=torch.float64, device="cuda")[1:]
    pidcuda.mulmm_dev(m, n, k, dA, ld, dB, k, C, ld, pidcuda.FORM_PLAIN)
    torch.cuda.synchronize()
    got = C.cpu().numpy().reshape(n, ld, 2)
    assert same(got[:, :m, :].reshape(-1), oracle.pidblas_mulmm(m, n, k, A, B))
    assert np.all(got[:, m:, :] == 7.0)
