"""GPU tests of products of intervals off the narrow path (swfp.cuh
sw_midrad_wide): around zero, a half-width of 40 %, [0, u] and [-0, u], [-0, +0],
subnormal, and ends near the largest double whose sum overflows.  Thin plain
products equal the oracle bit for bit, tensor-core ones its host model."""
import numpy as np
import pytest

from vcp_gb300 import pidcuda
from vcp_gb300 import workloads as W

pytestmark = pytest.mark.gpu

KINDS = ["around_zero", "half", "from_zero", "zero", "subnormal", "mixed"]


def entries(rng, rows, cols, kind):
    n = rows * cols
    m = W.ephi(rng, n, 4)
    if kind == "around_zero":
        r = np.abs(m) * rng.uniform(0, 4, n)
    elif kind == "half":
        r = np.abs(m) * 0.4
    elif kind == "from_zero":
        return np.stack([np.where(rng.random(n) < 0.5, 0.0, -0.0), np.abs(m)], -1).ravel()
    elif kind == "zero":
        return np.stack([np.full(n, -0.0), np.zeros(n)], -1).ravel()
    elif kind == "subnormal":
        m = np.ldexp(m, -1030)
        r = np.abs(m) * rng.uniform(0, 2, n)
    else:
        r = np.abs(m) * np.where(rng.random(n) < 0.1, 1.5, 2.0 ** -40)
    return np.stack([m - r, m + r], -1).ravel()


def same(a, b):
    a, b = np.asarray(a), np.asarray(b)
    nan = np.isnan(a) & np.isnan(b)
    return np.array_equal(a.view(np.int64)[~nan], b.view(np.int64)[~nan])


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("m,n,k", [(33, 1, 65), (70, 5, 40)])
def test_thin(cuda_lib, oracle, m, n, k, kind):
    rng = np.random.default_rng(m + KINDS.index(kind))
    A, B = entries(rng, m, k, kind), entries(rng, k, n, kind)
    assert same(pidcuda.mulmm(A, B, m, n, k), oracle.pidblas_mulmm(m, n, k, A, B))


def test_thin_overflowing_sums(cuda_lib, oracle):
    rng = np.random.default_rng(1)
    m, n, k = 40, 3, 30
    x = rng.uniform(0.5, 0.999, m * k) * np.finfo(np.float64).max
    A = np.stack([x * 0.7, x], -1).ravel()
    B = np.ldexp(W.interval_ephi(rng, k, n, 4, 2.0 ** -10), -40)
    assert same(pidcuda.mulmm(A, B, m, n, k), oracle.pidblas_mulmm(m, n, k, A, B))


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("m,n,k", [(33, 20, 65), (130, 70, 257)])
def test_tensor_cores(cuda_lib, oracle, m, n, k, kind):
    rng = np.random.default_rng(n + KINDS.index(kind))
    A, B = entries(rng, m, k, kind), entries(rng, k, n, kind)
    C = pidcuda.mulmm(A, B, m, n, k, form=pidcuda.FORM_OZAKI)
    ref, st = oracle.ozaki_igemm(m, n, k, A, B, 8, 2)
    assert st == 0
    assert same(C, ref)
