"""GPU test of the maxima of point factors (high words only, entries one by
one where a thread's largest is not a normal double of biased exponent 64 or
more): zeros, subnormals, the smallest normals, the largest doubles, powers of
two and their neighbours, alone and mixed in a line; infinities and NaN.  Every
bit equals the product of the same factors given as intervals."""
import numpy as np
import pytest
import torch

from vcp_gb300 import _lib, pidcuda

POINT_RIGHT, POINT_LEFT = 0, 1  # the side that is a plain matrix (the other an interval)

pytestmark = pytest.mark.gpu

VALUES = [0.0, -0.0, 5e-324, -2.0 ** -1030, 2.0 ** -1022, 2.0 ** -960, np.nextafter(2.0 ** -959, 0),
          2.0 ** -959, 1.0, np.nextafter(1.0, 0), -np.nextafter(2.0, 0), 2.0 ** 400, 1e-300]


def product(side, m, n, k, L, R):
    dL, dR = torch.from_numpy(L.reshape(-1)).cuda(), torch.from_numpy(R.reshape(-1)).cuda()
    C = torch.zeros(2 * m * n, dtype=torch.float64, device="cuda")
    if side is None:
        pidcuda.mulmm_dev(m, n, k, dL, m, dR, k, C, m, pidcuda.FORM_OZAKI)
    else:
        _lib.call("vcpcu_igemm_point_dev", side, m, n, k, dL.data_ptr(), m, dR.data_ptr(), k,
                  C.data_ptr(), m, pidcuda.FORM_OZAKI, 0, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return C.view(torch.int64)


def lines(rng, count, k, kind):
    X = np.zeros((count, k))
    for i in range(count):
        if kind == "one":
            X[i] = VALUES[i % len(VALUES)]
        else:
            X[i] = rng.choice(VALUES, k)
            if i % 3 == 0:
                X[i, rng.integers(k)] = np.finfo(float).max / 2 ** 60
    return X


@pytest.mark.parametrize("kind", ["one", "mixed"])
@pytest.mark.parametrize("m,n,k", [(33, 5, 70), (13, 40, 300), (1, 1, 1)])
def test_point_side(cuda_lib, m, n, k, kind):
    rng = np.random.default_rng(m)
    A = lines(rng, m, k, kind).T.copy()             # column-major: [k][m]
    B = rng.standard_normal((n, k))
    iv = lambda X: np.repeat(X[..., None], 2, axis=2)
    Bi = iv(B)
    Bi[..., 1] += 2.0 ** -30
    want = product(None, m, n, k, iv(A), Bi)
    assert torch.equal(product(POINT_LEFT, m, n, k, A, Bi), want)
    A2, B2 = rng.standard_normal((k, m)), lines(rng, n, k, kind)
    Ai = iv(A2)
    Ai[..., 1] += 2.0 ** -30
    want = product(None, m, n, k, Ai, iv(B2))
    assert torch.equal(product(POINT_RIGHT, m, n, k, Ai, B2), want)


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_not_finite(cuda_lib, bad):
    rng = np.random.default_rng(3)
    m, n, k = 40, 9, 80
    A, B = rng.standard_normal((k, m)), np.repeat(rng.standard_normal((n, k))[..., None], 2, axis=2)
    A[17, 31] = bad
    C = product(POINT_LEFT, m, n, k, A, B)
    assert bool(torch.isnan(C.view(torch.float64)).all())
    cuda_lib.vcpcu_status(torch.cuda.current_stream().cuda_stream)  # read and cleared
