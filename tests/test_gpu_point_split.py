"""GPU test of the split of two point factors (one double an entry): zeros,
subnormals, the smallest normals, huge values and lines whose exponents lie
beyond the direct path, at the edges of its tiles and for four and six limbs;
infinities and NaN.  Every bit of the directed product equals the interval
product of the same factors as [x, x]."""
import numpy as np
import pytest
import torch

from vcp_gb300 import pidcuda, vblas

pytestmark = pytest.mark.gpu

VALUES = np.array([0.0, -0.0, 5e-324, -2.0 ** -1030, 2.0 ** -960, 2.0 ** -959, 1.0,
                   np.nextafter(1.0, 0), -np.nextafter(2.0, 0), 3e-200, -7e150])


def both(m, n, k, A, B, slices):
    """A: [k][m], B: [n][k] (column-major matrices)."""
    dA, dB = torch.from_numpy(A.copy()).cuda(), torch.from_numpy(B.copy()).cuda()
    CU = torch.zeros(m * n, dtype=torch.float64, device="cuda")
    CD = torch.zeros_like(CU)
    vblas.udmatmul_ozaki_dev(m, k, n, dA.reshape(-1), m, dB.reshape(-1), k, CU, CD, m, slices)
    iv = lambda X: X.reshape(-1).repeat_interleave(2).contiguous()
    C = torch.zeros(2 * m * n, dtype=torch.float64, device="cuda")
    pidcuda.mulmm_dev(m, n, k, iv(dA), m, iv(dB), k, C, m, pidcuda.FORM_OZAKI, slices)
    torch.cuda.synchronize()
    return CU, CD, C.reshape(-1, 2)


@pytest.mark.parametrize("slices", [8, 9])
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (33, 9, 63), (128, 256, 64), (129, 257, 130),
                                   (7, 40, 300)])
def test_equal_to_the_interval_product(cuda_lib, m, n, k, slices):
    rng = np.random.default_rng(m + n)
    A, B = rng.standard_normal((k, m)), rng.standard_normal((n, k))
    A[:, ::3] = rng.choice(VALUES, A[:, ::3].shape)
    B[1::3] = rng.choice(VALUES, B[1::3].shape)
    A[:, m // 2] *= 2.0 ** -1000                # a row and a column beyond the direct path
    B[n // 2] = rng.choice(VALUES[:6], k)
    CU, CD, C = both(m, n, k, A, B, slices)
    assert torch.equal(CD.view(torch.int64), C[:, 0].contiguous().view(torch.int64))
    assert torch.equal(CU.view(torch.int64), C[:, 1].contiguous().view(torch.int64))


@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_not_finite(cuda_lib, bad):
    rng = np.random.default_rng(5)
    m, n, k = 40, 12, 70
    A, B = rng.standard_normal((k, m)), rng.standard_normal((n, k))
    B[3, 60] = bad
    CU, CD, C = both(m, n, k, A, B, 8)
    assert bool(torch.isnan(CU).all()) and bool(torch.isnan(CD).all()) and bool(torch.isnan(C).all())
    cuda_lib.vcpcu_status(torch.cuda.current_stream().cuda_stream)  # read and cleared
