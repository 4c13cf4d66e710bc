"""GPU tests of the slice GEMM on CTA pairs in the products that
test_gpu_pairs.py leaves out -- dd (up to 32 moduli), a point factor on either
side (one radius product), two point factors (none), the slice form's radius
products -- with an odd number of row blocks and k past a chunk, and of chained
launches of the pair kernel: captured into a graph, and on two streams.  Rows of
a product depend on no other row: every bit equals that of the same rows taken
128 at a time (one row block: no pairs)."""
import numpy as np
import pytest
import torch

from vcp_gb300 import pddcuda, pidcuda, vblas
from vcp_gb300 import workloads as W

pytestmark = pytest.mark.gpu

SHAPES = [(257, 1000, 1100), (385, 700, 1089), (897, 300, 2049)]


def bits(x):
    return np.asarray(x, dtype=np.float64).view(np.int64)


def row_blocks(A, m, k, words):
    """(first row, rows, flat column-major block) of A, 128 rows at a time."""
    M = A.reshape(k, m, words)
    for i in range(0, m, 128):
        yield i, min(128, m - i), np.ascontiguousarray(M[:, i:i + 128]).reshape(-1)


@pytest.mark.parametrize("m,n,k", SHAPES)
def test_dd(cuda_lib, m, n, k):
    rng = np.random.default_rng(m)

    def dd(count):
        hi = W.ephi(rng, count, 8)
        return np.stack([hi, hi * 2.0 ** -54 * rng.uniform(-1, 1, count)], -1).ravel()

    A, B = dd(m * k), dd(k * n)
    C, E = pddcuda.mulmm(A, B, m, n, k)
    C, E = C.reshape(n, m, 2), E.reshape(n, m)
    for i, r, Ai in row_blocks(A, m, k, 2):
        Ci, Ei = pddcuda.mulmm(Ai, B, r, n, k)
        assert np.array_equal(bits(C[:, i:i + r]), bits(Ci.reshape(n, r, 2)))
        assert np.array_equal(bits(E[:, i:i + r]), bits(Ei.reshape(n, r)))


@pytest.mark.parametrize("side", [0, 1])
@pytest.mark.parametrize("m,n,k", SHAPES)
def test_point_factor(cuda_lib, m, n, k, side):
    rng = np.random.default_rng(m + side)
    L = W.ephi(rng, m * k, 4) if side else W.interval_ephi(rng, m, k, 4, 2.0 ** -40)
    R = W.interval_ephi(rng, k, n, 4, 2.0 ** -40) if side else W.ephi(rng, k * n, 4)
    C = pidcuda.mul_point(side, L, R, m, n, k, form=pidcuda.FORM_OZAKI).reshape(n, m, 2)
    for i, r, Li in row_blocks(L, m, k, 1 if side else 2):
        Ci = pidcuda.mul_point(side, Li, R, r, n, k, form=pidcuda.FORM_OZAKI)
        assert np.array_equal(bits(C[:, i:i + r]), bits(Ci.reshape(n, r, 2)))


@pytest.mark.parametrize("m,n,k", SHAPES)
def test_two_point_factors(cuda_lib, m, n, k):
    """vblas naming: A m x k, B k x n here."""
    rng = np.random.default_rng(m)
    A, B = W.ephi(rng, m * k, 8), W.ephi(rng, k * n, 8)

    def both(Ai, r):
        U, D = np.empty(r * n), np.empty(r * n)
        vblas.udmatmul_ozaki(r, k, n, Ai, B, U, D)
        return U.reshape(n, r), D.reshape(n, r)

    U, D = both(A, m)
    for i, r, Ai in row_blocks(A, m, k, 1):
        Ui, Di = both(Ai, r)
        assert np.array_equal(bits(U[:, i:i + r]), bits(Ui))
        assert np.array_equal(bits(D[:, i:i + r]), bits(Di))


def test_slice_form(cuda_lib):
    m, n, k = 2177, 2400, 1089
    rng = np.random.default_rng(m)
    A, B = W.interval_ephi(rng, m, k, 4, 2.0 ** -40), W.interval_ephi(rng, k, n, 4, 2.0 ** -40)
    C = pidcuda.mulmm(A, B, m, n, k, form=pidcuda.FORM_OZAKI_SLICES, slices=3).reshape(n, m, 2)
    for i, r, Ai in row_blocks(A, m, k, 2):
        if i in (0, 1024, 2048, 2176):
            Ci = pidcuda.mulmm(Ai, B, r, n, k, form=pidcuda.FORM_OZAKI_SLICES, slices=3)
            assert np.array_equal(bits(C[:, i:i + r]), bits(Ci.reshape(n, r, 2)))


def operands(seed, m, n, k):
    rng = np.random.default_rng(seed)
    return (torch.from_numpy(W.interval_ephi(rng, m, k, 4, 2.0 ** -40)).cuda(),
            torch.from_numpy(W.interval_ephi(rng, k, n, 4, 2.0 ** -40)).cuda())


def in_row_blocks(m, n, k, A, B):
    C = torch.zeros(n, m, 2, dtype=torch.float64, device="cuda")
    for i in range(0, m, 128):
        r = min(128, m - i)
        Ci = torch.zeros(2 * r * n, dtype=torch.float64, device="cuda")
        pidcuda.mulmm_dev(r, n, k, A[2 * i:], m, B, k, Ci, r, pidcuda.FORM_OZAKI)
        C[:, i:i + r] = Ci.view(n, r, 2)
    torch.cuda.synchronize()
    return C.reshape(-1).view(torch.int64)


@pytest.mark.parametrize("m,n,k", [(897, 300, 1100), (1000, 900, 2100)])
def test_chained_pairs_captured(cuda_lib, m, n, k):
    A, B = operands(1, m, n, k)
    C = torch.zeros(2 * m * n, dtype=torch.float64, device="cuda")

    def call():
        pidcuda.mulmm_dev(m, n, k, A, m, B, k, C, m, pidcuda.FORM_OZAKI)

    call()  # (attributes are set up outside the capture)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        call()
    for seed in (2, 3):
        A2, B2 = operands(seed, m, n, k)
        A.copy_(A2)
        B.copy_(B2)
        C.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(C.view(torch.int64), in_row_blocks(m, n, k, A2, B2))


def test_chained_pairs_on_two_streams(cuda_lib):
    work = [(s, operands(sum(s), *s)) for s in ((897, 300, 1100), (1000, 900, 2100),
                                                (257, 1000, 1100))]
    want = [in_row_blocks(*s, *ab) for s, ab in work]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    out = []
    for r in range(6):
        for (m, n, k), (A, B) in work:
            st = streams[(r + len(out)) % 2]
            C = torch.zeros(2 * m * n, dtype=torch.float64, device="cuda")
            st.wait_stream(torch.cuda.current_stream())
            pidcuda.mulmm_dev(m, n, k, A, m, B, k, C, m, pidcuda.FORM_OZAKI, stream=st)
            out.append(C)
    torch.cuda.synchronize()
    for i, C in enumerate(out):
        assert torch.equal(C.view(torch.int64), want[i % len(work)])
