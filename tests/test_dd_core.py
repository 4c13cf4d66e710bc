"""CPU test of the dd product's per-entry arithmetic (vcp_gb300/csrc/ozaki_dd.cuh,
host-callable) against Python integers: the w-bit integers of doubles, the
remaindering for every modulus count the plans use -- X up to the plan's limit
M / 2 on either side, small and zero X -- and the two words of the result."""
import random
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "vcp_gb300" / "csrc"
MODULI = [256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211, 199, 197, 193,
          191, 181, 179, 173, 167, 163, 157, 151, 149, 139, 137, 131, 127, 113, 109, 107]

HARNESS = r"""
#include "ozaki_dd.cuh"
#include <cstdio>
using namespace vcpcu;
int main() {
  char kind;
  while (std::scanf(" %c", &kind) == 1) {
    if (kind == 'i') {  // the integer of a double
      unsigned long long b;
      int E, w;
      std::scanf("%llx %d %d", &b, &E, &w);
      double x;
      memcpy(&x, &b, 8);
      __int128 a = 0;
      dd_add_int(x, E, w, a);
      std::printf("%016llx%016llx\n", (unsigned long long)((unsigned __int128)a >> 64),
                  (unsigned long long)(unsigned __int128)a);
    } else {            // residues -> value and words
      int L;
      std::scanf("%d", &L);
      DdBasis B;
      dd_basis(L, &B);
      uint32_t V[DD_GROUPS] = {}, r[DDL];
      for (int l = 0; l < L; ++l) {
        unsigned c;
        std::scanf("%u", &c);
        V[l / 3] += c * B.a[l / 3][l % 3];
      }
      dd_reduce(V, B, r);
      const bool neg = dd_abs(r, B);
      std::printf("%d %d ", B.z, neg ? 1 : 0);
      for (int t = DDL - 1; t >= 0; --t) std::printf("%08x", r[t]);
      DdWords w;
      const bool ok = dd_words(r, &w);
      std::printf(" %d %llu %d %llu %d %d %d %d\n", ok ? 1 : 0, (unsigned long long)w.Mh, w.eh,
                  (unsigned long long)w.Ml, w.el, w.bl, w.lbl, w.lneg ? 1 : 0);
    }
  }
}
"""


def rn53(v: int):
    """(M, e) of v > 0 rounded to 53 bits, ties to even."""
    e = v.bit_length() - 53
    if e <= 0:
        return v << -e, e
    M, rem, half = v >> e, v & ((1 << e) - 1), 1 << (e - 1)
    return M + (rem > half or (rem == half and M & 1)), e


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("dd")
    (d / "dd.cpp").write_text(HARNESS)
    subprocess.run([gxx, "-O1", "-std=c++17", "-I", str(CSRC), str(d / "dd.cpp"), "-o",
                    str(d / "dd")], check=True)
    return lambda text: subprocess.run([str(d / "dd")], input=text, capture_output=True,
                                       text=True, check=True).stdout.split("\n")


def test_values_and_words(harness):
    rng = random.Random(4)
    cases, lines = [], []
    for L in [8, 14, 15, 16, 20, 26, 27, 28, 29, 30, 31, 32]:
        M = 1
        for m in MODULI[:L]:
            M *= m
        lim = (M - 1) // 2
        for it in range(300):
            k = it % 6
            if k == 0:
                X = rng.randrange(lim)
            elif k == 1:
                X = lim - rng.randrange(1000)
            elif k == 2:
                X = rng.randrange(1000)
            elif k == 3:
                X = rng.randrange(lim) >> rng.randrange(M.bit_length())
            elif k == 4:   # few bits: exact leading words, remainders far down
                X = (1 << rng.randrange(M.bit_length() - 2)) + (1 << rng.randrange(20))
            else:          # ties
                s = rng.randrange(max(1, M.bit_length() - 60))
                X = min(lim, (2 * rng.randrange(1 << 53) + 1) << s)
            X = min(X, lim) * rng.choice([-1, 1])
            cases.append((L, M, X))
            lines.append(f"r {L} " + " ".join(str(X % m) for m in MODULI[:L]))
    far = 0
    for (L, M, X), out in zip(cases, harness("\n".join(lines) + "\n")):
        f = out.split()
        z, neg, mag = int(f[0]), int(f[1]), int(f[2], 16)
        assert mag == abs(X) << z and neg == (X < 0), (L, X)
        ok, Mh, eh, Ml, el, bl, lbl, lneg = (int(x) for x in f[3:])
        if not ok:
            far += 1
            continue
        assert bl == mag.bit_length()
        if mag == 0:
            assert Mh == 0 and Ml == 0
            continue
        M1, e1 = rn53(mag)
        hi = M1 << e1 if e1 >= 0 else M1 >> -e1
        assert Mh * 2 ** (eh + 300) == hi << 300
        y = mag - hi
        if y == 0:
            assert Ml == 0
            continue
        assert lneg == (y < 0) and lbl == abs(y).bit_length()
        M2, e2 = rn53(abs(y))
        assert (Ml, el) == (M2, e2) or Ml * 2 ** (el + 300) == M2 * 2 ** (e2 + 300)
    assert far < len(cases) // 4


def test_integers_of_doubles(harness):
    import struct
    rng = random.Random(5)
    cases, lines = [], []
    for it in range(4000):
        e = rng.choice([0, 1, 5, 900, 1023, 1100, 2000, 2046]) if it % 3 else rng.randrange(2047)
        m = rng.getrandbits(52) if it % 5 else rng.choice([0, (1 << 52) - 1, 1 << 51])
        if it % 7 == 0:
            m &= ~((1 << rng.randrange(52)) - 1)
        b = (rng.getrandbits(1) << 63) | (e << 52) | m
        E = max(e, 1) - 1022 + 1 + rng.randrange(0, 130)   # |x| < 2^(E-1)
        w = rng.choice([56, 80, 104, 112])
        cases.append((struct.unpack("<d", struct.pack("<Q", b))[0], E, w))
        lines.append(f"i {b:x} {E} {w}")
    from fractions import Fraction
    for (x, E, w), out in zip(cases, harness("\n".join(lines) + "\n")):
        v = int(out, 16)
        v -= 1 << 128 if v >> 127 else 0
        assert v == round(Fraction(x) * Fraction(2) ** (w - E)), (x, E, w)
