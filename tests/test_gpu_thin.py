"""GPU tests of the row chains of the plain form (a lane per chain, the
non-negative ones on the integer pipe): thin products at the edges of their
blocks (32 rows, 16 columns of A a stage, 1 to 16 right columns), with
entries of every kind and spreads that make the integer chains change units
often, subnormal and near-overflow sums, non-finite entries, 8-byte aligned
operands; and the row sums of the norm.  Every bit equals the oracle's."""
import numpy as np
import pytest

from test_gpu_ozaki import mixed_intervals
from vcp_gb300 import pidcuda
from vcp_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def same(a, b):
    a, b = np.asarray(a), np.asarray(b)
    nan = np.isnan(a) & np.isnan(b)
    return np.array_equal(a.view(np.int64)[~nan], b.view(np.int64)[~nan])


@pytest.mark.parametrize("n", [1, 2, 3, 7, 16])
@pytest.mark.parametrize("m,k", [(1, 1), (31, 15), (32, 16), (33, 17), (70, 97), (5, 700)])
def test_thin_edges(cuda_lib, oracle, m, n, k):
    rng = np.random.default_rng(m + n + k)
    A = mixed_intervals(rng, m, k)
    A[np.abs(A) > 1e200] = 3.0
    A = np.sort(A.reshape(-1, 2), axis=1).reshape(-1)
    B = W.interval_ephi(rng, k, n, 30, 2.0 ** -20)
    assert same(pidcuda.mulmm(A, B, m, n, k), oracle.pidblas_mulmm(m, n, k, A, B))


@pytest.mark.parametrize("scale", [-1040, -980, 970, 1010])
def test_thin_ends_of_the_range(cuda_lib, oracle, scale):
    """Sums of subnormals, and sums that pass the largest double."""
    rng = np.random.default_rng(abs(scale))
    m, n, k = 40, 3, 200
    A = W.interval_ephi(rng, m, k, 6, 2.0 ** -10)
    B = W.interval_ephi(rng, k, n, 6, 2.0 ** -10)
    A = np.ldexp(A, scale // 2)
    B = np.ldexp(B, scale - scale // 2)
    assert same(pidcuda.mulmm(A, B, m, n, k), oracle.pidblas_mulmm(m, n, k, A, B))


@pytest.mark.parametrize("what", [np.inf, np.nan])
def test_thin_nonfinite(cuda_lib, oracle, what):
    rng = np.random.default_rng(3)
    m, n, k = 35, 4, 50
    A = W.interval_ephi(rng, m, k, 4, 2.0 ** -40)
    B = W.interval_ephi(rng, k, n, 4, 2.0 ** -40)
    A[2 * (3 + 20 * m) + 1] = what
    B[2 * (7 + 2 * k)] = -what
    assert same(pidcuda.mulmm(A, B, m, n, k), oracle.pidblas_mulmm(m, n, k, A, B))


def test_thin_operands_at_odd_addresses(cuda_lib, oracle):
    import torch
    rng = np.random.default_rng(4)
    m, n, k = 45, 5, 70
    A = W.interval_ephi(rng, m, k, 4, 2.0 ** -40)
    B = W.interval_ephi(rng, k, n, 4, 2.0 ** -40)
    dev = [torch.zeros(x + 1, dtype=torch.float64, device="cuda")[1:]
           for x in (A.size, B.size, 2 * m * n)]
    dev[0].copy_(torch.from_numpy(A))
    dev[1].copy_(torch.from_numpy(B))
    pidcuda.mulmm_dev(m, n, k, dev[0], m, dev[1], k, dev[2], m, pidcuda.FORM_PLAIN)
    torch.cuda.synchronize()
    assert same(dev[2].cpu().numpy(), oracle.pidblas_mulmm(m, n, k, A, B))


@pytest.mark.parametrize("n,phi", [(1, 4), (31, 100), (65, 400), (130, 4), (300, 30)])
def test_norm_row_sums(cuda_lib, oracle, n, phi):
    rng = np.random.default_rng(n + phi)
    A = W.interval_ephi(rng, n, n, phi, 2.0 ** -30)
    R = W.ephi(rng, n * n, min(phi, 100))
    assert pidcuda.norm_I_minus_RA(R, A, n) == oracle.norm_I_minus_RA(n, R, A)
