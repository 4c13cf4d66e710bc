"""GPU tests of the slice GEMM on CTA pairs (256-row tiles over two CTAs,
products of several 1024-deep chunks with an item for every SM) and on either
side of the line to the single-CTA kernel: odd last row blocks, ragged rows and
columns, chunk edges.  Every bit equals the host model's, or that of the same
rows taken 128 at a time (one row block: no pairs)."""
import numpy as np
import pytest

from vcp_gb300 import pidcuda
from vcp_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def bits(x):
    return np.asarray(x, dtype=np.float64).view(np.int64)


@pytest.mark.parametrize("s", [0x108, 8, 3])
@pytest.mark.parametrize("m,n,k", [(256, 1030, 1025), (257, 520, 1089), (897, 300, 1100),
                                   (1000, 256, 2048), (640, 600, 1024), (129, 1, 1500)])
def test_pair_tiles(cuda_lib, oracle, m, n, k, s):
    rng = np.random.default_rng(m + 3 * n + 7 * k)
    A = W.interval_ephi(rng, m, k, 4, 2.0 ** -40)
    B = W.interval_ephi(rng, k, n, 4, 2.0 ** -40)
    C = pidcuda.mulmm(A, B, m, n, k, form=pidcuda.FORM_OZAKI, slices=s)
    ref, st = oracle.ozaki_igemm(m, n, k, A, B, s, 2)
    assert st == 0
    assert np.array_equal(bits(C), bits(ref))


@pytest.mark.parametrize("m,n,k", [(1000, 900, 2100), (1155, 513, 4097), (2049, 100, 3072)])
def test_pairs_equal_single_row_blocks(cuda_lib, m, n, k):
    """Rows of a product depend on no other row."""
    rng = np.random.default_rng(m)
    A = W.interval_ephi(rng, m, k, 4, 2.0 ** -40).reshape(k, m, 2)
    B = W.interval_ephi(rng, k, n, 4, 2.0 ** -40)
    C = pidcuda.mulmm(A.reshape(-1), B, m, n, k, form=pidcuda.FORM_OZAKI)
    C = np.asarray(C).reshape(n, m, 2)
    for i in range(0, m, 128):
        r = min(128, m - i)
        Ai = np.ascontiguousarray(A[:, i:i + r]).reshape(-1)
        Ci = pidcuda.mulmm(Ai, B, r, n, k, form=pidcuda.FORM_OZAKI)
        assert np.array_equal(bits(C[:, i:i + r]), bits(np.asarray(Ci).reshape(n, r, 2)))
