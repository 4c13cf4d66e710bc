"""GPU test of the two forms of the thin product's radius chains, FP64 where
the blocks (32 rows x 1 to 16 columns) do not outnumber the SMs and integer
beyond, on either side of the line and at several columns a block, over entries
of every kind.  Every bit equals the oracle's."""
import numpy as np
import pytest

from test_gpu_ozaki import mixed_intervals
from vcp_gb300 import pidcuda
from vcp_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(4864, 1, 35), (4865, 1, 35), (2432, 2, 33), (2433, 2, 33),
                                   (700, 16, 50), (1500, 7, 20), (9729, 16, 17)])
def test_either_route(cuda_lib, oracle, m, n, k):
    rng = np.random.default_rng(m + n)
    A = mixed_intervals(rng, m, k)
    A[np.abs(A) > 1e200] = 3.0
    A = np.sort(A.reshape(-1, 2), axis=1).reshape(-1)
    B = W.interval_ephi(rng, k, n, 30, 2.0 ** -20)
    got = np.asarray(pidcuda.mulmm(A, B, m, n, k))
    ref = np.asarray(oracle.pidblas_mulmm(m, n, k, A, B))
    nan = np.isnan(got) & np.isnan(ref)
    assert np.array_equal(got.view(np.int64)[~nan], ref.view(np.int64)[~nan])
