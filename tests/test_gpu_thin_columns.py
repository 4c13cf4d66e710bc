"""GPU tests of the thin plain product's blocks of 1, 2, 4, 8 and 16 columns
(several blocks an SM, more rows than one wave of blocks takes, ragged last
columns) for every kind of left factor: entries of every kind, ends of the range,
non-finite entries, odd addresses.  Every bit equals the oracle's."""
import numpy as np
import pytest
import torch

from test_gpu_ozaki import mixed_intervals
from vcp_gb300 import pidcuda
from vcp_gb300 import workloads as W

pytestmark = pytest.mark.gpu

# a block's columns: 1, 2, 4, 8, 16
SHAPES = [(9729, 1, 40), (3000, 7, 17), (3000, 9, 17), (5000, 7, 5), (5000, 13, 5)]


def same(a, b):
    a, b = np.asarray(a), np.asarray(b)
    nan = np.isnan(a) & np.isnan(b)
    return np.array_equal(a.view(np.int64)[~nan], b.view(np.int64)[~nan])


def some_of_every_kind(rng, rows, cols):
    A = mixed_intervals(rng, rows, cols)
    A[np.abs(A) > 1e200] = 3.0
    return np.sort(A.reshape(-1, 2), axis=1).reshape(-1)


@pytest.mark.parametrize("m,n,k", SHAPES)
def test_interval_factors(cuda_lib, oracle, m, n, k):
    rng = np.random.default_rng(m + n)
    A, B = some_of_every_kind(rng, m, k), W.interval_ephi(rng, k, n, 30, 2.0 ** -20)
    assert same(pidcuda.mulmm(A, B, m, n, k), oracle.pidblas_mulmm(m, n, k, A, B))


@pytest.mark.parametrize("side", [0, 1])
@pytest.mark.parametrize("m,n,k", SHAPES)
def test_point_factor(cuda_lib, oracle, m, n, k, side):
    rng = np.random.default_rng(m + n + side)
    L = W.ephi(rng, m * k, 30) if side else some_of_every_kind(rng, m, k)
    R = W.interval_ephi(rng, k, n, 30, 2.0 ** -20) if side else W.ephi(rng, k * n, 30)
    assert same(pidcuda.mul_point(side, L, R, m, n, k),
                oracle.pidblas_mul_point(side, m, n, k, L, R))


@pytest.mark.parametrize("scale", [-1040, -980, 970, 1010])
@pytest.mark.parametrize("m,n,k", SHAPES)
def test_ends_of_the_range(cuda_lib, oracle, m, n, k, scale):
    rng = np.random.default_rng(abs(scale) + m)
    A = np.ldexp(W.interval_ephi(rng, m, k, 6, 2.0 ** -10), scale // 2)
    B = np.ldexp(W.interval_ephi(rng, k, n, 6, 2.0 ** -10), scale - scale // 2)
    assert same(pidcuda.mulmm(A, B, m, n, k), oracle.pidblas_mulmm(m, n, k, A, B))


@pytest.mark.parametrize("what", [np.inf, np.nan])
@pytest.mark.parametrize("m,n,k", SHAPES)
def test_nonfinite_entries_at_odd_addresses(cuda_lib, oracle, m, n, k, what):
    rng = np.random.default_rng(m)
    A = W.interval_ephi(rng, m, k, 4, 2.0 ** -40)
    B = W.interval_ephi(rng, k, n, 4, 2.0 ** -40)
    A[2 * (m - 1 + (k - 1) * m) + 1] = what
    B[2 * (k - 1) + 2 * k * (n - 1)] = -what
    dev = [torch.zeros(x + 1, dtype=torch.float64, device="cuda")[1:]
           for x in (A.size, B.size, 2 * m * n)]
    dev[0].copy_(torch.from_numpy(A))
    dev[1].copy_(torch.from_numpy(B))
    pidcuda.mulmm_dev(m, n, k, dev[0], m, dev[1], k, dev[2], m, pidcuda.FORM_PLAIN)
    torch.cuda.synchronize()
    assert same(dev[2].cpu().numpy(), oracle.pidblas_mulmm(m, n, k, A, B))


@pytest.mark.parametrize("n,nrhs", [(70, 16), (923, 16), (1847, 16)])
def test_solve_columns(cuda_lib, oracle, n, nrhs):
    """The products of the solve beside R [A], with the GPU's own R [A] given."""
    rng = np.random.default_rng(n)
    eye = np.eye(n)
    mid = (eye + rng.uniform(-0.25, 0.25, (n, n)) / n).ravel(order="F")
    A = np.stack([mid - 1e-10, mid + 1e-10], -1).ravel()
    R = (2 * eye.ravel() - mid).copy()
    bm, mx = rng.uniform(-1, 1, n * nrhs), rng.uniform(-1, 1, n * nrhs)
    b = np.stack([bm - 1e-9, bm + 1e-9], -1).ravel()
    x, G = pidcuda.linearsolve_verify(A, b, R, mx, n, nrhs, form=pidcuda.FORM_PLAIN)
    E = pidcuda.mul_point(1, R, A, n, n, n, form=pidcuda.FORM_PLAIN)
    st, xo, Go = oracle.ilss_verify(n, nrhs, A, b, R, mx, E=E)
    assert st == 0 and G == Go
    assert same(x, xo)
