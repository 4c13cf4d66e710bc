"""GPU tests of the chained kernels of one product (each may start while the
one before it still runs): products one after another on a stream over the same
buffers, on two streams at a time, and captured into a graph and replayed over
new inputs.  Every bit equals the product by itself."""
import numpy as np
import pytest
import torch

from vcp_gb300 import _lib, pidcuda
from vcp_gb300 import workloads as W

pytestmark = pytest.mark.gpu

SIZES = [(61, 48, 97), (300, 270, 130), (640, 600, 1100), (1, 1, 1)]


def operands(rng, m, n, k):
    return (torch.from_numpy(W.interval_ephi(rng, m, k, 4, 2.0 ** -40)).cuda(),
            torch.from_numpy(W.interval_ephi(rng, k, n, 4, 2.0 ** -40)).cuda())


def alone(m, n, k, A, B):
    C = torch.zeros(2 * m * n, dtype=torch.float64, device="cuda")
    pidcuda.mulmm_dev(m, n, k, A, m, B, k, C, m, pidcuda.FORM_OZAKI)
    torch.cuda.synchronize()
    return C.view(torch.int64)


def test_chains_behind_one_another(cuda_lib):
    """A product whose factor is the result before it, thirty in a row."""
    rng = np.random.default_rng(1)
    n = 130
    A, X = operands(rng, n, n, n)
    A *= 2.0 ** -4
    steps = []
    Y = X.clone()
    for _ in range(30):
        C = torch.zeros_like(Y)
        pidcuda.mulmm_dev(n, n, n, A, n, Y, n, C, n, pidcuda.FORM_OZAKI)
        steps.append(C)
        Y = C
    torch.cuda.synchronize()
    Y = X
    for C in steps:
        assert torch.equal(C.view(torch.int64), alone(n, n, n, A, Y))
        Y = C


def test_two_streams(cuda_lib):
    rng = np.random.default_rng(2)
    work = [(s, operands(rng, *s)) for s in SIZES]
    want = [alone(*s, *ab) for s, ab in work]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    out = []
    for r in range(8):
        for (s, ab) in work:
            m, n, k = s
            st = streams[(r + len(out)) % 2]
            C = torch.zeros(2 * m * n, dtype=torch.float64, device="cuda")
            st.wait_stream(torch.cuda.current_stream())
            pidcuda.mulmm_dev(m, n, k, ab[0], m, ab[1], k, C, m, pidcuda.FORM_OZAKI, stream=st)
            out.append(C)
    torch.cuda.synchronize()
    for i, C in enumerate(out):
        assert torch.equal(C.view(torch.int64), want[i % len(work)])


@pytest.mark.parametrize("noalloc", [True, False])
@pytest.mark.parametrize("m,n,k", SIZES)
def test_captured(cuda_lib, m, n, k, noalloc):
    if noalloc and m > 400:
        pytest.skip("beyond the static scratch")
    rng = np.random.default_rng(3)
    A, B = operands(rng, m, n, k)
    C = torch.zeros(2 * m * n, dtype=torch.float64, device="cuda")

    def call():
        if noalloc:
            _lib.call("vcpcu_igemm_noalloc_dev", m, n, k, A.data_ptr(), m, B.data_ptr(), k,
                      C.data_ptr(), m, 0, torch.cuda.current_stream().cuda_stream)
        else:
            pidcuda.mulmm_dev(m, n, k, A, m, B, k, C, m, pidcuda.FORM_OZAKI)

    call()  # (attributes and the static scratch are set up outside the capture)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        call()
    for seed in (4, 5):
        A2, B2 = operands(np.random.default_rng(seed), m, n, k)
        A.copy_(A2)
        B.copy_(B2)
        C.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(C.view(torch.int64), alone(m, n, k, A2, B2))
