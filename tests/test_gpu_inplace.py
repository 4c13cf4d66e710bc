"""GPU tests of interval products whose result lies over a factor: C == A, C a
few entries into A, C == B, in the thin and tiled plain kernels and on the tensor
cores.  Every bit equals the product into a buffer of its own."""
import numpy as np
import pytest
import torch

from vcp_gb300 import _lib, pidcuda
from vcp_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def dev(x, room=0):
    t = torch.zeros(x.size + room, dtype=torch.float64, device="cuda")
    t[:x.size] = torch.from_numpy(x).cuda()
    return t


@pytest.mark.parametrize("form,n", [(pidcuda.FORM_PLAIN, 1), (pidcuda.FORM_PLAIN, 5),
                                    (pidcuda.FORM_PLAIN, 16), (pidcuda.FORM_PLAIN, 24),
                                    (pidcuda.FORM_OZAKI, 16), (pidcuda.FORM_OZAKI, 40)])
@pytest.mark.parametrize("m", [1, 33, 700, 9729])
@pytest.mark.parametrize("shift", [0, 3])
def test_result_over_the_left_factor(cuda_lib, form, n, m, shift):
    rng = np.random.default_rng(m + n + shift)
    A = dev(W.interval_ephi(rng, m, n, 4, 2.0 ** -30), 2 * shift)
    B = dev(W.interval_ephi(rng, n, n, 4, 2.0 ** -30))
    C = torch.zeros(2 * m * n, dtype=torch.float64, device="cuda")
    pidcuda.mulmm_dev(m, n, n, A, m, B, n, C, m, form)
    over = A[2 * shift:2 * shift + 2 * m * n]
    pidcuda.mulmm_dev(m, n, n, A, m, B, n, over, m, form)
    torch.cuda.synchronize()
    assert torch.equal(over.view(torch.int64), C.view(torch.int64))


@pytest.mark.parametrize("form,n", [(pidcuda.FORM_PLAIN, 1), (pidcuda.FORM_PLAIN, 16),
                                    (pidcuda.FORM_PLAIN, 24), (pidcuda.FORM_OZAKI, 40)])
@pytest.mark.parametrize("m", [33, 500])
def test_result_over_the_right_factor(cuda_lib, form, n, m):
    rng = np.random.default_rng(m + n)
    A = dev(W.interval_ephi(rng, m, m, 4, 2.0 ** -30))
    B = dev(W.interval_ephi(rng, m, n, 4, 2.0 ** -30))
    C = torch.zeros(2 * m * n, dtype=torch.float64, device="cuda")
    pidcuda.mulmm_dev(m, n, m, A, m, B, m, C, m, form)
    pidcuda.mulmm_dev(m, n, m, A, m, B, m, B, m, form)
    torch.cuda.synchronize()
    assert torch.equal(B.view(torch.int64), C.view(torch.int64))


@pytest.mark.parametrize("side,form,n", [(0, pidcuda.FORM_PLAIN, 7), (1, pidcuda.FORM_PLAIN, 7),
                                         (0, pidcuda.FORM_OZAKI, 30), (1, pidcuda.FORM_OZAKI, 30)])
def test_point_product_over_the_left_factor(cuda_lib, side, form, n):
    rng = np.random.default_rng(side + n)
    m = 6000
    L = dev(W.ephi(rng, m * n, 4) if side else W.interval_ephi(rng, m, n, 4, 2.0 ** -30), m * n)
    R = dev(W.interval_ephi(rng, n, n, 4, 2.0 ** -30) if side else W.ephi(rng, n * n, 4))
    C = torch.zeros(2 * m * n, dtype=torch.float64, device="cuda")
    s = torch.cuda.current_stream().cuda_stream

    def call(out):
        _lib.call("vcpcu_igemm_point_dev", side, m, n, n, L.data_ptr(), m, R.data_ptr(), n,
                  out.data_ptr(), m, form, 0, s)

    call(C)
    over = L[:2 * m * n]
    call(over)
    torch.cuda.synchronize()
    assert torch.equal(over.view(torch.int64), C.view(torch.int64))
