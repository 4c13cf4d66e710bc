"""The steps of a young radius chain (vcp_gb300/csrc/dirchain.cuh
chain_fma_steps): on the CPU, chains whose first batches are the FP64
instructions and whose later ones go whole or step by step have the bits of the
upward FMA chain; on the GPU, interval products around the stages where the
kernel changes over equal the oracle bit for bit."""
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parent.parent / "vcp_gb300" / "csrc"

HARNESS = r"""
#include "dirchain.cuh"
#include <cstdio>
#include <random>
using namespace vcpcu;
static std::mt19937_64 g(5);
static double draw(int mid, int span) {
  const uint64_t r = g();
  if (r % 61 == 0) return 0.0;
  const uint64_t e = (uint64_t)(mid - span + (int)(g() % (2 * span + 1)));
  return chain_from_bits((e << 52) | (r >> 12));
}
int main() {
  long bad = 0, batches = 0;
  for (int rep = 0; rep < 3000; ++rep) {
    const int mids[] = {1023, 530, 1500, 512, 1535};
    const int mid = mids[rep % 5], span = rep % 4 == 0 ? 0 : (rep % 4 == 1 ? 4 : (rep % 4 == 2 ? 40 : 300));
    const int young = rep % 6;
    DirChain x = chain_zero();
    double c = 0.0;
    for (int t = 0; t < 12; ++t) {
      double a[8], b[8];
      for (int p = 0; p < 8; ++p) {
        a[p] = draw(mid, span);
        b[p] = draw(mid, span);
        if (rep % 50 == 3 && t == rep % 7 && p == 5) a[p] = rep & 64 ? INFINITY : NAN;
        c = chain_fma_ru(a[p], b[p], c);
      }
      auto get = [&](int p, ChainFactor* u, ChainFactor* v) {
        *u = chain_factor(a[p]);
        *v = chain_factor(b[p]);
      };
      if (t < young / 2 || !chain_fma_batch<8>(x, get)) chain_fma_steps<8>(x, get, t < young);
      const double v = chain_value(x);
      if (oz_bits(v) != oz_bits(c) && !(v != v && c != c)) ++bad;
      ++batches;
    }
  }
  std::printf("%ld %ld\n", batches, bad);
  return bad != 0;
}
"""


def test_young_chains_against_directed_doubles(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    src = tmp_path / "young.cpp"
    src.write_text(HARNESS)
    exe = tmp_path / "young"
    subprocess.run([gxx, "-O1", "-frounding-math", "-std=c++17", "-I", str(CSRC), str(src), "-o",
                    str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    batches, bad = (int(x) for x in r.stdout.split())
    assert r.returncode == 0 and bad == 0
    assert batches == 3000 * 12


@pytest.mark.gpu
@pytest.mark.parametrize("phi", [0, 8, 250])
@pytest.mark.parametrize("m,n,k", [(33, 17, 15), (64, 40, 16), (33, 65, 17), (40, 33, 31),
                                   (300, 130, 32), (70, 18, 33), (31, 129, 41), (1100, 1030, 40)])
def test_products_of_short_inner_dimension(cuda_lib, oracle, m, n, k, phi):
    from vcp_gb300 import pidcuda
    from vcp_gb300 import workloads as W
    rng = np.random.default_rng(m + n + k + phi)
    A = W.interval_ephi(rng, m, k, phi, 2.0 ** -12)
    B = W.interval_ephi(rng, k, n, phi, 2.0 ** -12)
    C = np.asarray(pidcuda.mulmm(A, B, m, n, k))
    ref = np.asarray(oracle.pidblas_mulmm(m, n, k, A, B))
    assert np.array_equal(C.view(np.int64), ref.view(np.int64))
