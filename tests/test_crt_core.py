"""CPU test of the remaindering core that the reassembly kernels run
(vcp_gb300/csrc/ozaki_crt.cuh, host-callable): for every modulus count, the
value rebuilt from the residues of X is X itself -- random X, X next to the
plan's limit M / 4, small and zero X, both signs, and residues whose group
values are the largest -- and the directed conversion gives the truncated and
the next 53-bit significand."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "vcp_gb300" / "csrc"

HARNESS = r"""
#include "ozaki_crt.cuh"
#include <cmath>
#include <cstdio>
#include <random>
using namespace vcpcu;
typedef unsigned __int128 u128;
static u128 join(const uint32_t (&w)[4]) {
  u128 v = 0;
  for (int t = 3; t >= 0; --t) v = (v << 32) | w[t];
  return v;
}
static double dbl(const uint32_t (&w)[2]) {
  uint64_t b = ((uint64_t)w[0] << 32) | w[1];
  double d;
  memcpy(&d, &b, 8);
  return d;
}
int main() {
  std::mt19937_64 g(1);
  long values = 0, conversions = 0, bad = 0;
  for (int L = 3; L <= OZ_MAX_MODULI_128; ++L) {
    CrtBasis b;
    crt_basis(L, &b);
    u128 M = 1;
    for (int l = 0; l < L; ++l) M *= (u128)OZ_MODULI[l];
    const __int128 lim = (__int128)(M / 4);
    for (long it = 0; it < 40000; ++it) {
      const u128 r = ((u128)g() << 64) | g();
      __int128 X;
      switch (it % 4) {
        case 0: X = (__int128)(r % (u128)lim); break;
        case 1: X = lim - 1 - (__int128)(g() % 1000); break;
        case 2: X = (__int128)(g() % 1000); break;
        default: X = (__int128)((r >> (g() % 126)) % (u128)lim); break;
      }
      if (it & 8) X = -X;
      uint32_t V[OZ_CRT_GROUPS] = {}, w[4];
      for (int l = 0; l < L; ++l) {
        int c = (int)(X % OZ_MODULI[l]);
        if (c < 0) c += OZ_MODULI[l];
        V[l / 3] += (uint32_t)c * b.a[l / 3][l % 3];
      }
      crt_reduce(V, b, w);
      ++values;
      if (join(w) != (u128)X << b.z) ++bad;
      const int neg = crt_abs(w);
      const u128 mag = join(w);
      if (neg != (X < 0) || mag != (u128)(X < 0 ? -X : X) << b.z) ++bad;
      int bl = 0;
      while (bl < 128 && (mag >> bl)) ++bl;
      uint32_t dn[2], up[2];
      const int e = (int)(g() % 801) - 400;
      crt_to_dir(w, (e + 1149) << 20, dn, up);
      ++conversions;
      const int sh = bl > 53 ? bl - 53 : 0;
      const u128 top = mag >> sh;
      const bool rem = (top << sh) != mag;
      if (dbl(dn) != std::ldexp((double)(uint64_t)top, sh + e)) ++bad;
      if (dbl(up) != std::ldexp((double)((uint64_t)top + rem), sh + e)) ++bad;
    }
    // every residue m - 1 (X = -1): the largest group values
    uint32_t V[OZ_CRT_GROUPS] = {}, w[4];
    for (int l = 0; l < L; ++l) V[l / 3] += (uint32_t)(OZ_MODULI[l] - 1) * b.a[l / 3][l % 3];
    crt_reduce(V, b, w);
    if (join(w) != (u128)(__int128)-1 << b.z) ++bad;
  }
  std::printf("%ld %ld %ld\n", values, conversions, bad);
  return bad != 0;
}
"""


def test_crt_core_against_128_bit_integers(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    src = tmp_path / "core.cpp"
    src.write_text(HARNESS)
    exe = tmp_path / "core"
    subprocess.run([gxx, "-O2", "-std=c++17", "-I", str(CSRC), str(src), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    values, conversions, bad = (int(x) for x in r.stdout.split())
    assert r.returncode == 0 and bad == 0
    assert values == conversions == 14 * 40000
