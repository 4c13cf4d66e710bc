"""GPU test of the residue products over several 1024-deep chunks of the inner
dimension, at the chunk's edges and past 64 chunks, with ragged rows and
columns: every bit equals the host model's."""
import numpy as np
import pytest

from vcp_gb300 import pidcuda
from vcp_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def bits(x):
    return np.asarray(x, dtype=np.float64).view(np.int64)


@pytest.mark.parametrize("s", [0x108, 8])
@pytest.mark.parametrize("m,n,k", [(129, 257, 1025), (1, 1, 2048), (130, 65, 2049), (33, 31, 5000),
                                   (5, 3, 66000)])
def test_chunks(cuda_lib, oracle, m, n, k, s):
    rng = np.random.default_rng(m + 3 * n + 7 * k)
    A = W.interval_ephi(rng, m, k, 4, 2.0 ** -40)
    B = W.interval_ephi(rng, k, n, 4, 2.0 ** -40)
    C = pidcuda.mulmm(A, B, m, n, k, form=pidcuda.FORM_OZAKI, slices=s)
    ref, st = oracle.ozaki_igemm(m, n, k, A, B, s, 2)
    assert st == 0
    assert np.array_equal(bits(C), bits(ref))


@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_chunk_sums_at_their_limits(cuda_lib, oracle, sign):
    """Equal entries in every place: all chunks of a modulus carry the same
    value, the largest that these digits give."""
    m, n, k = 6, 5, 4096
    A = np.full((k, m, 2), np.nextafter(2.0, 0.0))
    B = np.full((n, k, 2), sign * np.nextafter(2.0, 0.0))
    C = pidcuda.mulmm(A.reshape(-1), B.reshape(-1), m, n, k, form=pidcuda.FORM_OZAKI, slices=0x108)
    ref, st = oracle.ozaki_igemm(m, n, k, A.reshape(-1), B.reshape(-1), 0x108, 2)
    assert st == 0
    assert np.array_equal(bits(C), bits(ref))
