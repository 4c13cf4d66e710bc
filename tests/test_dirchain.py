"""CPU test of the integer chains of directed sums (vcp_gb300/csrc/dirchain.cuh,
host-callable): every step of a sum chain (up and down) and of an upward FMA
chain has the bits of the directed double operation -- random magnitudes and
spreads, zeros, subnormals, sums that pass the largest double, infinities,
NaN and negative terms."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "vcp_gb300" / "csrc"

HARNESS = r"""
#include "dirchain.cuh"
#include <cstdio>
#include <random>
using namespace vcpcu;
static std::mt19937_64 g(9);
static double dbl(uint64_t b) { double d; memcpy(&d, &b, 8); return d; }
static bool same(double a, double b) {
  return oz_bits(a) == oz_bits(b) || (a != a && b != b);
}
// a non-negative double with exponent field lo .. lo + span, or a special one
static double draw(int lo, int span, int special) {
  if (special && g() % special == 0) {
    switch (g() % 6) {
      case 0: return 0.0;
      case 1: return dbl(g() & ((1ULL << 52) - 1));   // subnormal
      case 2: return dbl((1ULL << 52) - 1 + (g() % 3));
      case 3: return 0.0;
      case 4: return dbl((uint64_t)(lo + span) << 52);
      default: return 1.0;
    }
  }
  uint64_t m = g();
  if (g() % 8 == 0) m = 0;
  if (g() % 8 == 0) m = ~0ULL;
  return dbl(((uint64_t)(lo + g() % (span + 1)) << 52) | (m >> 12));
}
int main() {
  long steps = 0, bad = 0;
  const int starts[] = {1, 1000, 1020, 2000, 2040, 30, 500};
  for (int rep = 0; rep < 4000; ++rep) {
    const int lo = starts[rep % 7];
    int span = (int)(g() % 40);
    if (lo + span > 2046) span = 2046 - lo;
    const int special = rep % 3 == 0 ? 4 : (rep % 3 == 1 ? 50 : 0);
    DirChain u = chain_zero(), d = chain_zero(), f = chain_zero();
    double cu = 0.0, cd = 0.0, cf = 0.0;
    const int flo = lo > 1500 ? 1530 : (lo < 600 ? 400 : lo);
    // the same terms in batches of 8
    DirChain bu = chain_zero(), bd = chain_zero(), bf = chain_zero();
    double vx[8], va[8], vb[8];
    for (int k = 0; k < 304; ++k) {
      double x = draw(lo, span, special);
      if (rep % 40 == 7 && k == 200) x = INFINITY;
      if (rep % 40 == 8 && k == 200) x = NAN;
      if (rep % 40 == 9 && k == 200) x = -1.0;
      long long M;
      int e;
      chain_split(oz_bits(x), &M, &e);
      chain_add<true>(u, x, M, e);
      chain_add<false>(d, x, M, e);
      cu = chain_add_dir(cu, x, true);
      cd = chain_add_dir(cd, x, false);
      if (!same(chain_value(u), cu) || !same(chain_value(d), cd)) ++bad;
      double a = draw(flo, span / 2, special), b = draw(flo, span / 2, special);
      if (rep % 40 == 10 && k == 200) a = INFINITY;
      if (rep % 40 == 11 && k == 200) b = NAN;
      chain_fma(f, chain_factor(a), chain_factor(b));
      if (oz_bits(chain_factor_value(chain_factor(a))) != oz_bits(a)) ++bad;
      cf = chain_fma_ru(a, b, cf);
      if (!same(chain_value(f), cf)) ++bad;
      vx[k % 8] = x;
      va[k % 8] = a;
      vb[k % 8] = b;
      if (k % 8 == 7) {
        auto get = [&](int p, long long* m, int* y) { chain_split(oz_bits(vx[p]), m, y); };
        auto value = [&](int p) { return vx[p]; };
        chain_add_n<true, 8>(bu, get, value);
        chain_add_n<false, 8>(bd, get, value);
        auto factors = [&](int p, ChainFactor* x, ChainFactor* y) {
          *x = chain_factor(va[p]);
          *y = chain_factor(vb[p]);
        };
        chain_fma_n<8>(bf, factors, factors);
        if (!same(chain_value(bu), cu) || !same(chain_value(bd), cd) ||
            !same(chain_value(bf), cf)) ++bad;
      }
      ++steps;
    }
  }
  std::printf("%ld %ld\n", steps, bad);
  return bad != 0;
}
"""


def test_chains_against_directed_doubles(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    src = tmp_path / "chain.cpp"
    src.write_text(HARNESS)
    exe = tmp_path / "chain"
    subprocess.run([gxx, "-O1", "-frounding-math", "-std=c++17", "-I", str(CSRC), str(src), "-o",
                    str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    steps, bad = (int(x) for x in r.stdout.split())
    assert r.returncode == 0 and bad == 0
    assert steps == 4000 * 304
