"""GPU tests of the reassembly on either side of its direct path: sums of a row's
and a column's exponent beside the limits (every value a normal double), rows and
columns of both kinds in one quad and one block, zero rows and columns, zero
midpoints with radii, point factors, every slice count that changes the limits.
Every bit equals the host model's."""
import numpy as np
import pytest

from vcp_gb300 import pidcuda, vblas
from vcp_gb300 import workloads as W

pytestmark = pytest.mark.gpu

# exponents that rows and columns are scaled by: sums beside 990, 2 w - 1020 for w
# = 14 .. 62, -970 for the radii (40 binades below), and single ones beside +-1000
SETS = {
    "high": ([0, 495, 501, 508, 980], [0, 470, 478, 484, 490]),
    "low": ([0, -440, -452, -460, -470, -500], [0, -440, -448, -456, -464, -500]),
    "radii": ([0, -450, -462, -468], [0, -455, -461, -470, 500]),
    "columns": ([0, 3], [985, 994, 998, -960, -975, -1004, -1012]),
    "spread": ([-980, -700, -300, 0, 300, 700, 980], [-980, -500, 0, 20, 500, 970]),
}


def same(a, b):
    a, b = np.asarray(a), np.asarray(b)
    nan = np.isnan(a) & np.isnan(b)
    return np.array_equal(a.view(np.int64)[~nan], b.view(np.int64)[~nan])


def scaled(rng, m, n, k, rows, cols, rad=2.0 ** -40):
    A = W.interval_ephi(rng, m, k, 2, rad).reshape(k, m, 2)
    B = W.interval_ephi(rng, k, n, 2, rad).reshape(n, k, 2)
    A = np.ldexp(A, rng.choice(rows, m)[None, :, None])
    B = np.ldexp(B, rng.choice(cols, n)[:, None, None])
    return A, B


@pytest.mark.parametrize("s", [2, 0x108, 8, 9])
@pytest.mark.parametrize("name", list(SETS))
def test_exponent_sums_beside_the_limits(cuda_lib, oracle, name, s):
    rng = np.random.default_rng(sorted(SETS).index(name) + s)
    m, n, k = 37, 70, 65
    A, B = (x.reshape(-1) for x in scaled(rng, m, n, k, *SETS[name]))
    C = pidcuda.mulmm(A, B, m, n, k, form=pidcuda.FORM_OZAKI, slices=s)
    ref, st = oracle.ozaki_igemm(m, n, k, A, B, s, 2)
    assert st == 0
    assert same(C, ref)


@pytest.mark.parametrize("s", [0x108, 8])
@pytest.mark.parametrize("scales", [([0], [0]), SETS["spread"]])
def test_zero_rows_and_columns(cuda_lib, oracle, s, scales):
    """Zero rows and columns, and rows and columns of zero midpoints with radii."""
    rng = np.random.default_rng(s)
    m, n, k = 45, 133, 66
    A, B = scaled(rng, m, n, k, *scales)
    A[:, ::3] = 0.0
    A[:, 1::6] = np.array([-2.0 ** -20, 2.0 ** -20])
    B[::5] = 0.0
    B[1::7] = np.array([-2.0 ** -10, 2.0 ** -10])
    A, B = A.reshape(-1), B.reshape(-1)
    C = pidcuda.mulmm(A, B, m, n, k, form=pidcuda.FORM_OZAKI, slices=s)
    ref, st = oracle.ozaki_igemm(m, n, k, A, B, s, 2)
    assert st == 0
    assert same(C, ref)


@pytest.mark.parametrize("name", list(SETS))
def test_point_factors(cuda_lib, oracle, name):
    """[x, x] on either side and on both; two points also as plain matrices."""
    rng = np.random.default_rng(len(name))
    m, n, k = 34, 41, 65
    A, B = scaled(rng, m, n, k, *SETS[name])
    Ap, Bp = A[:, :, 0].copy(), B[:, :, 0].copy()
    Ap[:, ::4] = 0.0
    Bp[::6] = 0.0
    Ai, Bi = np.repeat(Ap.reshape(-1), 2), np.repeat(Bp.reshape(-1), 2)
    A, B, Ap, Bp = A.reshape(-1), B.reshape(-1), Ap.reshape(-1), Bp.reshape(-1)
    F = pidcuda.FORM_OZAKI
    for got, (x, y) in ((pidcuda.mul_point(1, Ap, B, m, n, k, form=F), (Ai, B)),
                        (pidcuda.mul_point(0, A, Bp, m, n, k, form=F), (A, Bi))):
        ref, st = oracle.ozaki_igemm(m, n, k, x, y, 8, 2)
        assert st == 0
        assert same(got, ref)
    U, D = np.empty(m * n), np.empty(m * n)
    vblas.udmatmul_ozaki(m, k, n, Ap, Bp, U, D)
    ref, st = oracle.ozaki_igemm(m, n, k, Ai, Bi, 8, 2)
    assert st == 0
    assert same(D, ref[0::2].copy()) and same(U, ref[1::2].copy())


def test_batch(cuda_lib, oracle):
    """The grouped reassembly over problems of both kinds."""
    import torch

    from vcp_gb300 import batch
    rng = np.random.default_rng(3)
    probs, want = [], []
    for t, name in enumerate(list(SETS) + ["plain"]):
        m, n, k = 20 + 9 * t, 33 + 5 * t, 40 + 30 * t
        A, B = scaled(rng, m, n, k, *SETS.get(name, ([0], [0])))
        A[:, ::7] = 0.0
        A, B = A.reshape(-1), B.reshape(-1)
        C = torch.zeros(2 * m * n, dtype=torch.float64, device="cuda")
        probs.append((m, n, k, torch.from_numpy(A).cuda(), m, torch.from_numpy(B).cuda(), k, C, m))
        ref, st = oracle.ozaki_igemm(m, n, k, A, B, 8, 2)
        assert st == 0
        want.append(ref)
    batch.run(probs, pidcuda.FORM_OZAKI)
    torch.cuda.synchronize()
    for p, ref in zip(probs, want):
        assert same(p[7].cpu().numpy(), ref)
