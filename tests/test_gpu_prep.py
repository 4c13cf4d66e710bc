"""GPU tests of the operand preparation of the tensor-core form at the edges
of its blocks (rows by 8 and 32, columns by 8, 16 and 32, k by 8, 64 and
256), with padded leading dimensions, on every mixture of entries (narrow,
zero, wide, straddling), and with a factor given as plain doubles, also at an
odd 8-byte address.  Every bit equals the host model's."""
import numpy as np
import pytest

from test_gpu_ozaki import mixed_intervals
from vcp_gb300 import pidcuda, vblas
from vcp_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def bits(x):
    return np.asarray(x, dtype=np.float64).view(np.int64)


def degenerate(P):
    out = np.empty(2 * P.size)
    out[0::2] = P
    out[1::2] = P
    return out


def padded(flat, rows, cols, ld, width, offset=0):
    """A device copy with leading dimension ld (entries of `width` doubles),
    the padding NaN, starting `offset` doubles into its buffer."""
    import torch
    buf = np.full(ld * cols * width + offset, np.nan)
    v = buf[offset:].reshape(cols, ld, width)
    v[:, :rows, :] = flat.reshape(cols, rows, width)
    return torch.from_numpy(buf).cuda()[offset:]


SHAPES = [(1, 1, 1), (7, 9, 63), (8, 8, 64), (9, 33, 65), (33, 15, 129), (40, 17, 192),
          (31, 70, 257), (3, 5, 2300)]


@pytest.mark.parametrize("s", [8, 9, 0x108])
@pytest.mark.parametrize("m,n,k", SHAPES)
def test_block_edges_and_padding(cuda_lib, oracle, m, n, k, s):
    import torch
    rng = np.random.default_rng(m + n + k)
    A = mixed_intervals(rng, m, k) if k > 100 else W.interval_ephi(rng, m, k, 4, 2.0 ** -3)
    B = W.interval_ephi(rng, k, n, 4, 2.0 ** -40)
    A[np.abs(A) > 1e200] = 1.0   # keep the products finite
    A = np.sort(A.reshape(-1, 2), axis=1).reshape(-1)
    C = torch.full((2 * (m + 5) * n,), 7.0, dtype=torch.float64, device="cuda")
    pidcuda.mulmm_dev(m, n, k, padded(A, m, k, m + 3, 2), m + 3, padded(B, k, n, k + 1, 2), k + 1,
                      C, m + 5, pidcuda.FORM_OZAKI, s)
    torch.cuda.synchronize()
    ref, st = oracle.ozaki_igemm(m, n, k, A, B, s, 2)
    got = C.cpu().numpy().reshape(n, m + 5, 2)
    assert st == 0
    assert np.array_equal(bits(got[:, :m, :]), bits(ref.reshape(n, m, 2)))
    assert np.all(got[:, m:, :] == 7.0)


@pytest.mark.parametrize("side", [0, 1])
@pytest.mark.parametrize("m,n,k", SHAPES)
def test_point_factor_as_it_is(cuda_lib, oracle, m, n, k, side):
    """[L] R and L [R] with the point factor at an odd address."""
    import torch
    from vcp_gb300 import _lib
    rng = np.random.default_rng(m + n + k + side)
    L = W.interval_ephi(rng, m, k, 4, 2.0 ** -40) if side == 0 else W.ephi(rng, m * k, 6)
    R = W.ephi(rng, k * n, 6) if side == 0 else W.interval_ephi(rng, k, n, 4, 2.0 ** -40)
    dL = padded(L, m, k, m + 1, 2 - side, side)
    dR = padded(R, k, n, k + 2, 1 + side, 1 - side)
    C = torch.empty(2 * m * n, dtype=torch.float64, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    _lib.call("vcpcu_igemm_point_dev", side, m, n, k, dL.data_ptr(), m + 1, dR.data_ptr(), k + 2,
              C.data_ptr(), m, pidcuda.FORM_OZAKI, 0, st)
    torch.cuda.synchronize()
    Li, Ri = (L, degenerate(R)) if side == 0 else (degenerate(L), R)
    ref, ok = oracle.ozaki_igemm(m, n, k, Li, Ri, 8, 2)
    assert ok == 0
    assert np.array_equal(bits(C.cpu().numpy()), bits(ref))


@pytest.mark.parametrize("m,n,k", SHAPES)
def test_point_factors_and_plain_results(cuda_lib, oracle, m, n, k):
    """Both ends as plain matrices with a padded leading dimension, all four
    at odd addresses."""
    import torch
    rng = np.random.default_rng(m * n + k)
    A, B = W.ephi(rng, m * k, 8), W.ephi(rng, k * n, 8)
    out = torch.full((2, (m + 3) * n + 1), 7.0, dtype=torch.float64, device="cuda")
    CU, CD = out[0, 1:], out[1, 1:]
    vblas.udmatmul_ozaki_dev(m, k, n, padded(A, m, k, m + 1, 1, 1), m + 1,
                             padded(B, k, n, k + 2, 1, 1), k + 2, CU, CD, m + 3)
    torch.cuda.synchronize()
    ref, ok = oracle.ozaki_igemm(m, n, k, degenerate(A), degenerate(B), crt=True)
    assert ok == 0
    for t, which in ((CU, 1), (CD, 0)):
        got = t.cpu().numpy().reshape(n, m + 3)
        assert np.array_equal(bits(got[:, :m].reshape(-1)), bits(ref[which::2]))
        assert np.all(got[:, m:] == 7.0)
