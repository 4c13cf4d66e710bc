"""CPU test of the entry arithmetic that the preparation kernels of the
tensor-core form run (vcp_gb300/csrc/ozaki_prep.cuh, host-callable): on
narrow entries -- widths from zero to a whole binade, both signs, odd and
even, next to the ends of a binade -- midpoint, radius and P = RU(|m| + r)
carry the bits of the directed double operations, their exponents are those
of the general rule, and the 16-bit upward digits equal the general ones."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "vcp_gb300" / "csrc"

HARNESS = r"""
#include "ozaki_prep.cuh"
#include <cfenv>
#include <cmath>
#include <cstdio>
#include <random>
using namespace vcpcu;
static double dbl(uint64_t b) { double d; memcpy(&d, &b, 8); return d; }
static uint64_t bits(double d) { uint64_t b; memcpy(&b, &d, 8); return b; }
int main() {
  std::mt19937_64 g(3);
  long n = 0, bad = 0, wide = 0;
  const uint64_t H = 1ULL << 52;
  for (long it = 0; it < 2000000; ++it) {
    const uint64_t e = it % 7 == 0 ? 64 + g() % 1983 : 900 + g() % 200;
    uint64_t f = g() & (H - 1);
    if (it % 11 == 0) f = g() % 64;
    if (it % 13 == 0) f = H - 1 - g() % 64;
    const uint64_t room = H - 1 - f;
    uint64_t w = g() >> (12 + g() % 52);
    if (it % 5 == 0) w = g() % 5;
    if (it % 17 == 0) w = 2 * ((1ULL << (g() % 51)) | (1ULL << (g() % 51)));  // few bits in D
    if (it % 19 == 0) f &= ~(H - 1) | (g() << 40);
    if (w > H - 1 - f) w = room & (H - 1 - f);
    const bool sg = it & 1;
    const uint64_t a = (e << 52) | f, b = a + w;
    const double lo = sg ? -dbl(b) : dbl(a), up = sg ? -dbl(a) : dbl(b);
    const Words L = words_of(bits(lo)), U = words_of(bits(up));
    if (!iv_narrow(L, U)) { ++bad; continue; }
    Words m, P;
    uint64_t D;
    iv_midrad(L, U, &m, &D, &P);
    volatile double vlo = lo, vup = up, s = vlo + vup, vm, d1, d2, vp;
    vm = std::isfinite(s) ? s * 0.5 : vlo * 0.5 + vup * 0.5;
    fesetround(FE_UPWARD);
    d1 = vm - vlo;
    d2 = vup - vm;
    volatile double r = d1 > d2 ? d1 : d2, am = std::fabs(vm);
    vp = am + r;
    fesetround(FE_TONEAREST);
    ++n;
    if (w64(m) != bits(vm)) ++bad;
    if (std::ldexp((double)D, (int)e - 1075) != r) ++bad;
    const bool pinf = !std::isfinite((double)vp);
    if (!pinf && w64(P) != bits(vp)) ++bad;
    uint32_t em, er;
    iv_exponents(L, U, &em, &er);
    if (exp_dec(em) != oz_exponent(std::fabs(vm))) ++bad;
    if (exp_dec(er) != oz_exponent(r)) ++bad;
    if (!iv_all_ones(L, U) && oz_exponent(vp) != exp_dec(em)) ++bad;
    // digits against any exponent from the entry's own upwards
    const int up_by = (int)(g() % 3 == 0 ? g() % 80 : g() % 20);
    const int Ep = oz_exponent(vp) + up_by, Er = oz_exponent(r) + up_by;
    if (Ep >= -900 && Ep <= 1000 &&
        up16_bits(P.hi, P.lo, Ep + 1028) != (int)oz_scaled_int64(vp, Ep, 16, 1)) ++bad;
    if (D && Er >= -900 && Er <= 1000) {
      ++wide;
      if (up16_ulps(D, Er + 1090 - (int)e) != (int)oz_scaled_int64(r, Er, 16, 1)) ++bad;
    }
    if (up16_ulps(0, 5) != 0 || up16_bits(0, 0, 1028) != 0) ++bad;
  }
  // the same zero at both ends; entries that go the general way
  for (double a : {0.0, -0.0}) {
    const Words L = words_of(bits(a));
    Words m, P;
    uint64_t D;
    iv_midrad(L, L, &m, &D, &P);
    if (!iv_zero(L, L) || dbl(w64(m)) != 0.0 || D != 0 || w64(P) != 0) ++bad;
  }
  const double no[][2] = {{1.0, 2.0}, {-1.0, 1.0}, {0.0, 1.0}, {1e-300, 1e-300 * 3},
                          {INFINITY, INFINITY}, {NAN, NAN}, {5e-324, 5e-324}, {-0.0, 1.0},
                          {-0.0, 0.0}, {0.0, -0.0}};
  for (auto& p : no)
    if (iv_narrow(words_of(bits(p[0])), words_of(bits(p[1]))) ||
        iv_zero(words_of(bits(p[0])), words_of(bits(p[1])))) ++bad;
  std::printf("%ld %ld %ld\n", n, wide, bad);
  return bad != 0;
}
"""


def test_entry_arithmetic_against_directed_doubles(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    src = tmp_path / "prep.cpp"
    src.write_text(HARNESS)
    exe = tmp_path / "prep"
    subprocess.run([gxx, "-O1", "-frounding-math", "-std=c++17", "-I", str(CSRC), str(src), "-o",
                    str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    n, wide, bad = (int(x) for x in r.stdout.split())
    assert r.returncode == 0 and bad == 0
    assert n == 2000000 and wide > 1000000
