"""GPU tests of the reassembly of the tensor-core form at the edges of its
tiles (4 rows a thread, 128 rows and 8 to 64 columns a block) and on both of
its paths: exponents within +-400, where it adds to exponent fields, and the
general one beyond them; products far below their row and column maxima.
Every bit equals the host model's."""
import numpy as np
import pytest

from vcp_gb300 import pidcuda
from vcp_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def bits(x):
    return np.asarray(x, dtype=np.float64).view(np.int64)


def check(oracle, m, n, k, A, B, s):
    C = pidcuda.mulmm(A, B, m, n, k, form=pidcuda.FORM_OZAKI, slices=s)
    ref, st = oracle.ozaki_igemm(m, n, k, A, B, s, 2)
    assert st == 0
    assert np.array_equal(bits(C), bits(ref))


@pytest.mark.parametrize("s", [0x108, 8, 3])
@pytest.mark.parametrize("m,n", [(1, 1), (3, 9), (4, 8), (5, 65), (127, 7), (128, 64), (131, 130),
                                 (257, 33)])
def test_tile_edges(cuda_lib, oracle, m, n, s):
    rng = np.random.default_rng(m + 3 * n)
    A = W.interval_ephi(rng, m, 70, 4, 2.0 ** -40)
    B = W.interval_ephi(rng, 70, n, 4, 2.0 ** -40)
    check(oracle, m, n, 70, A, B, s)


@pytest.mark.parametrize("s", [0x108, 8])
@pytest.mark.parametrize("scale", [399, 402, 480])
def test_exponents_beside_the_direct_path(cuda_lib, oracle, scale, s):
    """Rows and columns scaled to either side of the direct path's limit, and
    rows of either kind in one quad."""
    rng = np.random.default_rng(scale)
    m, n, k = 21, 19, 65
    A = W.interval_ephi(rng, m, k, 4, 2.0 ** -40)
    B = W.interval_ephi(rng, k, n, 4, 2.0 ** -40)
    A.reshape(k, m, 2)[:, ::3, :] *= 2.0 ** scale
    A.reshape(k, m, 2)[:, 1::3, :] *= 2.0 ** -scale
    B.reshape(n, k, 2)[::4, :, :] *= 2.0 ** scale
    B.reshape(n, k, 2)[1::4, :, :] *= 2.0 ** -scale
    check(oracle, m, n, k, A, B, s)


@pytest.mark.parametrize("s", [0x108, 8])
def test_products_far_below_their_maxima(cuda_lib, oracle, s):
    """Entries whose exact value is zero or far below 2^64 of its units (one
    small term under a large row maximum), zero radii, and a zero row."""
    rng = np.random.default_rng(5)
    m, n, k = 18, 12, 64
    A = np.zeros((k, m, 2))
    B = np.zeros((n, k, 2))
    A[0] = 1.0                                     # meets zeros of B
    for i in range(m - 1):
        A[1 + i % 8, i, :] = np.sign(rng.random() - 0.5) * 2.0 ** -(4 * i)
    A[:, m - 1] = 0.0
    B[:, 1:9, :] = rng.choice([-1.0, 1.0], (n, 8, 1)) * 2.0 ** -rng.integers(0, 50, (n, 8, 1))
    B[:, 20, :] = 1.0                              # meets zeros of A
    A[3, :, 1] += 2.0 ** -30                       # some radii
    check(oracle, m, n, k, A.reshape(-1), B.reshape(-1), s)


def test_unaligned_result(cuda_lib):
    """C at an 8-byte boundary (pairs then go out as two words)."""
    import torch
    rng = np.random.default_rng(6)
    m, n, k = 70, 41, 130
    A = torch.from_numpy(W.interval_ephi(rng, m, k, 4, 2.0 ** -40)).cuda()
    B = torch.from_numpy(W.interval_ephi(rng, k, n, 4, 2.0 ** -40)).cuda()
    ldc = m + 3
    out = []
    for off in (0, 1):
        buf = torch.full((2 * ldc * n + 1,), 7.0, dtype=torch.float64, device="cuda")
        pidcuda.mulmm_dev(m, n, k, A, m, B, k, buf[off:], ldc, pidcuda.FORM_OZAKI)
        torch.cuda.synchronize()
        out.append(buf[off:off + 2 * ldc * n].cpu().numpy())
    assert np.array_equal(bits(out[0]), bits(out[1]))
    assert np.all(out[1].reshape(n, ldc, 2)[:, m:, :] == 7.0)
