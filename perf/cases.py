"""Performance cases of the verified matrix products: what a user of this
package runs, through its public entry points, from the smallest products of a
Newton step to the n = 8192 interval product.

``listed()`` gives the standing cases, ``draw(rng)`` more of the same ranges;
``prepare(case, seed)`` makes what a caller has in hand before the call,
``run(state)`` is one pass, ``work(case)`` the bytes and operations that the
pass cannot do without, ``exact(case, seed)`` the same results in 64-bit
arithmetic without this package.

Matrices are column-major; intervals are {inf, sup} pairs and dd values
{a1, a2} pairs, flat, as the C ABI takes them.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from vcp_gb300 import batch, pddcuda, pidcuda, vblas

FORMS = {"plain": pidcuda.FORM_PLAIN, "tensor": pidcuda.FORM_OZAKI}
FAST = 8 | pidcuda.SLICES_FAST_RADIUS


def listed() -> list[dict]:
    return [
        # One of the many small products of a Newton or verification step: the
        # time is the call and its launches.
        {"name": "interval_small", "op": "interval", "form": "tensor", "slices": 0,
         "m": 61, "n": 48, "k": 97, "phi": 0, "rad": 40},
        # The n = 512 product of intervals, the first workload of the benchmark,
        # in the policies' default form and precision.
        {"name": "interval_512", "op": "interval", "form": "tensor", "slices": 0,
         "m": 512, "n": 512, "k": 512, "phi": 4, "rad": 40},
        # Phi diag(w u) Phi^T of Emden's equation, Legendre order 70: a long
        # inner dimension under an odd, mid-sized result.
        {"name": "interval_basis_1225", "op": "interval", "form": "tensor", "slices": 0,
         "m": 1225, "n": 1225, "k": 12544, "phi": 2, "rad": 44},
        # The large product, at the precision that the autotuner picks for it.
        {"name": "interval_8192", "op": "interval", "form": "tensor", "slices": FAST,
         "m": 8192, "n": 8192, "k": 8192, "phi": 4, "rad": 40},
        # The bit-for-bit pidblas form, where a caller needs its very bits.
        {"name": "interval_plain_512", "op": "interval", "form": "plain", "slices": 0,
         "m": 512, "n": 512, "k": 512, "phi": 4, "rad": 40},
        # vblas udmatmul: both roundings of a point product, the FMA-chain bits.
        {"name": "updown_1024", "op": "updown", "m": 1024, "n": 1024, "k": 1024, "phi": 8},
        # The same enclosure on the tensor cores, tall and thin.
        {"name": "updown_tensor_tall", "op": "updown_tensor", "slices": 8,
         "m": 16384, "n": 16384, "k": 256, "phi": 8},
        # The product under pddblas's refinements, with its error bound.
        {"name": "dd_2048", "op": "dd", "m": 2048, "n": 2048, "k": 2048, "phi": 0},
        # A batch of uneven products replayed from its graph.
        {"name": "batch_256", "op": "batch", "form": "tensor", "count": 256, "lo": 32, "hi": 1024,
         "shapes": 4096},
        # The verification of a linear solve, one right-hand side.
        {"name": "solve_4096", "op": "solve", "n": 4096, "nrhs": 1},
        # The verification of the generalized eigenvalues of the Emden run.
        {"name": "eig_1225", "op": "eig", "n": 1225},
        # The drop-in behind vcp::matrix: ordinary host memory in and out.
        {"name": "host_1000", "op": "host", "form": "tensor", "slices": 0,
         "m": 1100, "n": 900, "k": 1000, "phi": 4, "rad": 40},
    ]


def _size(rng, lo: int, hi: int) -> int:
    """A size spread over the logarithm of [lo, hi]; one in four a multiple of 64."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if v >= 64 and rng.random() < 0.25:
        v = v // 64 * 64
    return max(lo, min(hi, v))


def draw(rng) -> dict:
    op = rng.choice(["interval", "interval", "interval", "plain", "updown", "updown_tensor", "dd",
                     "batch", "solve", "eig", "host"])
    if op == "interval":
        while True:
            m, n, k = _size(rng, 16, 8192), _size(rng, 16, 8192), _size(rng, 16, 16384)
            if m * n * k <= 2 ** 38 and max(m, n) * k <= 2 ** 27:
                break
        return {"op": "interval", "form": "tensor", "slices": rng.choice([0, 0, FAST, 7, 9]),
                "m": m, "n": n, "k": k, "phi": rng.randint(0, 8), "rad": rng.randint(24, 48)}
    if op == "plain":
        return {"op": "interval", "form": "plain", "slices": 0, "m": _size(rng, 16, 1024),
                "n": _size(rng, 16, 1024), "k": _size(rng, 16, 1024), "phi": rng.randint(0, 8),
                "rad": rng.randint(24, 48)}
    if op == "updown":
        return {"op": "updown", "m": _size(rng, 16, 1500), "n": _size(rng, 16, 1500),
                "k": _size(rng, 16, 1500), "phi": rng.randint(0, 16)}
    if op == "updown_tensor":
        while True:
            m, n, k = _size(rng, 64, 16384), _size(rng, 64, 16384), _size(rng, 64, 4096)
            if m * n * k <= 2 ** 36 and n * k <= 2 ** 25:
                break
        return {"op": "updown_tensor", "slices": rng.randint(6, 9), "m": m, "n": n, "k": k,
                "phi": rng.randint(0, 16)}
    if op == "dd":
        return {"op": "dd", "m": _size(rng, 16, 3000), "n": _size(rng, 16, 3000),
                "k": _size(rng, 16, 3000), "phi": rng.randint(0, 16)}
    if op == "batch":
        return {"op": "batch", "form": "tensor", "count": _size(rng, 12, 512), "lo": 32,
                "hi": rng.randint(128, 1024), "shapes": rng.randrange(1 << 20)}
    if op == "solve":
        return {"op": "solve", "n": _size(rng, 64, 4096), "nrhs": rng.randint(1, 3)}
    if op == "eig":
        return {"op": "eig", "n": _size(rng, 32, 1500)}
    return {"op": "host", "form": "tensor", "slices": 0, "m": _size(rng, 32, 1500),
            "n": _size(rng, 32, 1500), "k": _size(rng, 32, 1500), "phi": rng.randint(0, 8),
            "rad": rng.randint(24, 48)}


# ---- inputs ------------------------------------------------------------------------

def _gen(seed: int) -> torch.Generator:
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _empty(count: int) -> torch.Tensor:
    return torch.empty(count, dtype=torch.float64, device="cuda")


def _rand(count: int, g) -> torch.Tensor:
    return torch.rand(count, generator=g, dtype=torch.float64, device="cuda")


def _ephi(count: int, phi: int, g) -> torch.Tensor:
    """Mantissa U[1, 2), random sign, exponent U{-phi .. phi}."""
    v = 1.0 + _rand(count, g)
    v *= torch.randint(0, 2, (count,), generator=g, device="cuda") * 2 - 1
    if phi > 0:
        v = torch.ldexp(v, torch.randint(-phi, phi + 1, (count,), generator=g, device="cuda",
                                         dtype=torch.int32))
    return v


def _pairs(a: torch.Tensor, b: torch.Tensor) -> torch.Tensor:
    return torch.stack((a, b), dim=-1).reshape(-1)


def _kv(mid: torch.Tensor, rad: float) -> torch.Tensor:
    r = mid.abs() * rad
    return _pairs(mid - r, mid + r)


def _dims(case: dict) -> list[tuple[int, int, int]]:
    """The shapes of a batch: log-uniform in [lo, hi], the case's own."""
    rng = np.random.default_rng(case["shapes"])
    d = np.exp(rng.uniform(np.log(case["lo"]), np.log(case["hi"]), (case["count"], 3)))
    return [tuple(int(x) for x in row) for row in d.round()]


def _inputs(case: dict, seed: int) -> dict:
    g, op = _gen(seed), case["op"]
    if op in ("interval", "host"):
        m, n, k, rad = case["m"], case["n"], case["k"], 2.0 ** -case["rad"]
        return {"A": _kv(_ephi(m * k, case["phi"], g), rad),
                "B": _kv(_ephi(k * n, case["phi"], g), rad)}
    if op in ("updown", "updown_tensor"):
        m, n, k = case["m"], case["n"], case["k"]
        return {"A": _ephi(m * n, case["phi"], g), "B": _ephi(n * k, case["phi"], g)}
    if op == "dd":
        out = {}
        for name, count in (("A", case["m"] * case["k"]), ("B", case["k"] * case["n"])):
            hi = _ephi(count, case["phi"], g)
            out[name] = _pairs(hi, hi * 2.0 ** -53 * (_rand(count, g) * 2.0 - 1.0))
        return out
    if op == "batch":
        dims = _dims(case)
        return {"A": _kv(_rand(sum(m * k for m, n, k in dims), g) * 2.0 - 1.0, 1e-12),
                "B": _kv(_rand(sum(k * n for m, n, k in dims), g) * 2.0 - 1.0, 1e-12)}
    n = case["n"]
    eye = torch.eye(n, dtype=torch.float64, device="cuda")
    if op == "solve":
        mid = (_rand(n * n, g).reshape(n, n) * 2 - 1) / n ** 0.5 + eye
        b = _rand(n * case["nrhs"], g).reshape(n, -1) * 2 - 1
        R = torch.linalg.inv(mid)
        return {"Am": mid, "bm": b, "R": R, "mx": R @ b}
    Am = torch.randn(n, n, generator=g, dtype=torch.float64, device="cuda") / n ** 0.5
    Am = (Am + Am.t()) / 2
    G = eye + 0.1 * torch.randn(n, n, generator=g, dtype=torch.float64, device="cuda") / n ** 0.5
    Bm = G @ G.t()
    Bm = (Bm + Bm.t()) / 2
    Li = torch.linalg.inv(torch.linalg.cholesky(Bm))
    w, V = torch.linalg.eigh(Li @ Am @ Li.t())
    X = Li.t() @ V
    return {"Am": Am, "Bm": Bm, "X": X, "lam": w, "Y": torch.linalg.inv(Bm @ X)}


def _cols(M: torch.Tensor) -> torch.Tensor:
    """A 2-D tensor as a flat column-major buffer."""
    return M.t().contiguous().reshape(-1)


RAD = 2.0 ** -40  # of the systems of "solve" and "eig"


def prepare(case: dict, seed: int) -> dict:
    op, x = case["op"], _inputs(case, seed)
    s = dict(case)
    if op == "interval":
        s.update(x, C=_empty(2 * case["m"] * case["n"]))
    elif op == "host":
        s.update({name: v.cpu().numpy() for name, v in x.items()},
                 C=np.empty(2 * case["m"] * case["n"]))
    elif op in ("updown", "updown_tensor"):
        s.update(x, CU=_empty(case["m"] * case["k"]), CD=_empty(case["m"] * case["k"]))
    elif op == "dd":
        mn = case["m"] * case["n"]
        s.update(x, C=_empty(2 * mn), E=_empty(mn))
    elif op == "batch":
        dims = _dims(case)
        s.update(x, C=_empty(2 * sum(m * n for m, n, k in dims)))
        probs, a, b, c = [], 0, 0, 0
        for m, n, k in dims:
            probs.append((m, n, k, s["A"][a:], m, s["B"][b:], k, s["C"][c:], m))
            a, b, c = a + 2 * m * k, b + 2 * k * n, c + 2 * m * n
        s["graph"] = batch.BatchGraph(probs, FORMS[case["form"]])
    elif op == "solve":
        n, r = case["n"], case["nrhs"]
        s.update(A=_kv(_cols(x["Am"]), RAD), b=_kv(_cols(x["bm"]), RAD), R=_cols(x["R"]),
                 mx=_cols(x["mx"]), x=_empty(2 * n * r), G=_empty(1))
    else:
        n = case["n"]
        s.update(A=_kv(_cols(x["Am"]), RAD), B=_kv(_cols(x["Bm"]), RAD), X=_cols(x["X"]),
                 Y=_cols(x["Y"]), lam=x["lam"].clone(), C=_empty(2 * n * n), BX=_empty(2 * n * n),
                 M=_empty(n * n), out=_empty(2 * n), bound=_empty(1))
    return s


# ---- one pass ----------------------------------------------------------------------

def run(s: dict):
    op = s["op"]
    if op == "interval":
        m, n, k = s["m"], s["n"], s["k"]
        pidcuda.mulmm_dev(m, n, k, s["A"], m, s["B"], k, s["C"], m, FORMS[s["form"]], s["slices"])
        return s["C"]
    if op == "host":
        m, n, k = s["m"], s["n"], s["k"]
        return pidcuda.mulmm(s["A"], s["B"], m, n, k, FORMS[s["form"]], s["slices"], s["C"])
    if op == "updown":
        m, n, k = s["m"], s["n"], s["k"]
        vblas.udmatmul_dev(m, n, k, s["A"], m, s["B"], n, s["CU"], s["CD"], m)
        return s["CU"], s["CD"]
    if op == "updown_tensor":
        m, n, k = s["m"], s["n"], s["k"]
        vblas.udmatmul_ozaki_dev(m, n, k, s["A"], m, s["B"], n, s["CU"], s["CD"], m, s["slices"])
        return s["CU"], s["CD"]
    if op == "dd":
        m, n, k = s["m"], s["n"], s["k"]
        pddcuda.mulmm_dev(m, n, k, s["A"], m, s["B"], k, s["C"], m, s["E"], m)
        C = s["C"].view(-1, 2)
        return C[:, 0], C[:, 1], s["E"]
    if op == "batch":
        s["graph"].launch()
        return s["C"]
    if op == "solve":
        n, r = s["n"], s["nrhs"]
        pidcuda.linearsolve_verify_dev(n, r, s["A"], n, s["b"], n, s["R"], n, s["mx"], n, s["x"],
                                       n, s["G"], pidcuda.FORM_OZAKI)
        return s["x"], s["G"]
    n = s["n"]
    pidcuda.eigsymge_stage1_dev(n, s["A"], n, s["B"], n, s["X"], n, s["C"], s["BX"], s["M"],
                                pidcuda.FORM_OZAKI)
    pidcuda.eigsymge_stage2_dev(n, s["lam"], s["Y"], n, s["C"], s["BX"], s["out"], s["bound"],
                                pidcuda.FORM_OZAKI)
    return s["out"], s["bound"], s["BX"], s["M"]


def work(case: dict) -> dict:
    """Inputs read once, outputs written once; one real product for every
    product of the definition (midpoints and the two radius products of an
    interval product; both roundings; the three word products of dd)."""
    op = case["op"]
    if op in ("interval", "host"):
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 16 * (m * k + k * n + m * n),
                "flops": (8 if case["form"] == "plain" else 6) * m * n * k}
    if op in ("updown", "updown_tensor"):
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 8 * (m * n + n * k + 2 * m * k),
                "flops": (4 if op == "updown" else 2) * m * n * k}
    if op == "dd":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 16 * (m * k + k * n) + 24 * m * n, "flops": 6 * m * n * k}
    if op == "batch":
        dims = _dims(case)
        return {"bytes": 16 * sum(m * k + k * n + m * n for m, n, k in dims),
                "flops": 6 * sum(m * n * k for m, n, k in dims)}
    n = case["n"]
    if op == "solve":  # R [A], and three products with the right-hand sides
        r = case["nrhs"]
        return {"bytes": 24 * n * n + 40 * n * r, "flops": 4 * n ** 3 + 16 * n * n * r}
    # [A] X, [B] X, Y (AX - BX diag(lambda)), Y (BX)
    return {"bytes": (48 + 24) * n * n + 24 * n, "flops": 16 * n ** 3}


# ---- 64-bit values -----------------------------------------------------------------

def _mat(flat: torch.Tensor, rows: int, cols: int) -> torch.Tensor:
    return flat.reshape(cols, rows).t()


def _iv(flat: torch.Tensor, rows: int, cols: int):
    v = flat.reshape(cols, rows, 2)
    lo, up = v[:, :, 0].t(), v[:, :, 1].t()
    return (lo + up) / 2, (up - lo) / 2


def _ivmul(A, B, m: int, n: int, k: int) -> torch.Tensor:
    mA, rA = _iv(A, m, k)
    mB, rB = _iv(B, k, n)
    C = mA @ mB
    T = (mA.abs() + rA) @ rB
    T += rA @ mB.abs()
    return _pairs(_cols(C - T), _cols(C + T))


def _rowsum(M: torch.Tensor) -> torch.Tensor:
    return M.sum(dim=1)


def exact(case: dict, seed: int):
    op, x = case["op"], _inputs(case, seed)
    if op in ("interval", "host"):
        C = _ivmul(x["A"], x["B"], case["m"], case["n"], case["k"])
        return C.cpu().numpy() if op == "host" else C
    if op in ("updown", "updown_tensor"):
        C = _cols(_mat(x["A"], case["m"], case["n"]) @ _mat(x["B"], case["n"], case["k"]))
        return C, C.clone()
    if op == "dd":  # the leading words; the trailing ones are below 64-bit arithmetic
        m, n, k = case["m"], case["n"], case["k"]
        return _cols(_mat(x["A"].view(-1, 2)[:, 0], m, k) @ _mat(x["B"].view(-1, 2)[:, 0], k, n)), \
            None, None
    if op == "batch":
        out, a, b = [], 0, 0
        for m, n, k in _dims(case):
            out.append(_ivmul(x["A"][a:a + 2 * m * k], x["B"][b:b + 2 * k * n], m, n, k))
            a, b = a + 2 * m * k, b + 2 * k * n
        return torch.cat(out)
    if op == "solve":
        A, b, R, mx = x["Am"], x["bm"], x["R"], x["mx"]
        E = R @ A
        E.diagonal().sub_(1.0)
        E = E.abs() + (R.abs() @ A.abs()) * RAD
        G = _rowsum(E).max()
        P, Pr = A @ mx - b, RAD * (A.abs() @ mx.abs() + b.abs())
        r = (R @ P).abs() + R.abs() @ Pr
        t = (_rowsum(r) if case["nrhs"] > 1 else r).max()
        u = r + _rowsum(E)[:, None] * (t / (1.0 - G))
        return _pairs(_cols(mx - u), _cols(mx + u)), G.reshape(1)
    A, B, X, lam, Y = x["Am"], x["Bm"], x["X"], x["lam"], x["Y"]
    BX, BXr = B @ X, RAD * (B.abs() @ X.abs())
    C, Cr = A @ X - BX * lam, RAD * (A.abs() @ X.abs()) + BXr * lam.abs()
    R = (Y @ C).abs() + Y.abs() @ Cr
    S = Y @ BX
    S.diagonal().sub_(1.0)
    S = S.abs() + Y.abs() @ BXr
    bound = _rowsum(S).max()
    u = _rowsum(R) + _rowsum(S) * (_rowsum(R).max() / (1.0 - bound))
    return _pairs(lam - u, lam + u), bound.reshape(1), _pairs(_cols(BX - BXr), _cols(BX + BXr)), \
        _cols(BX)
