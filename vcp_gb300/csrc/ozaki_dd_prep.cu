// ozaki_dd_prep.cu -- operand preparation of the dd product (ozaki_dd.cu) in
// two launches over both factors, in the manner of the interval product's
// (ozaki_prep.cu): the exponents of the largest |a1| of every row of A and
// column of B, then the residue planes (oz_tile_off) of the w-bit integers of
// their entries, bf16, k padded with zeros.
//
// Bound: DRAM (16 bytes read, 2 L written per entry of the split) and the FP32
// pipe (10 paired instructions per residue and pair of entries).  n = 2048, L =
// 28: maxima and exponents 52 -> 29 us, splits 214 -> 128 us (89 at the copy
// bandwidth), against one pass per factor with 12-bit limbs and 128-bit
// shifts in the general form.
#include "common.cuh"
#include "ozaki.cuh"
#include "ozaki_common.cuh"
#include "ozaki_dd.cuh"
#include "ozaki_prep.cuh"
#include "ozaki_residue.cuh"
#include "swfp.cuh"

namespace vcpcu {

namespace {

constexpr int NT = 256;
constexpr int DD_LIMBS = 8;  // 14-bit limbs: w <= 112

struct DdSide {
  const double* X;  // dd pairs, ld in pairs
  long ld;
  int lines;
  size_t pstride;
  uint16_t* planes;
  uint32_t* e;  // encoded exponent of the largest |a1| of a line
};
struct DdPrepArgs {
  DdSide a, b;
  int K, Kp, L, w;
  int* flag;
  int nA;            // blocks of the left factor
  int spanA, spanB;  // maxima: k range of a block
};

struct DdMax {
  uint32_t e = 0;
  bool bad = false;
  __device__ __forceinline__ void add(double2 v) {
    const uint32_t h = words_of(sw_bits(v.x)).hi;
    const int f = (int)((h >> 20) & 0x7ffu);
    if (f == 0) {  // zero or subnormal
      e = max(e, exp_enc(oz_exponent(oz_abs(v.x))));
    } else {
      e = max(e, (uint32_t)(f - 1021 + OZ_EXP_BIAS));
      bad = bad || f == 0x7ff;
    }
    bad = bad || !sw_finite(v.y);
  }
};

__device__ __forceinline__ void dd_max_left(const DdSide& s, int K, int rb, int k0, int* flag) {
  __shared__ uint32_t red[32];
  const int lane = threadIdx.x & 31, ph = threadIdx.x >> 5;
  const int i = rb * 32 + lane;
  if (threadIdx.x < 32) red[lane] = 0;
  __syncthreads();
  DdMax x;
  if (i < s.lines) {
    constexpr int U = 8;
    for (int c = k0 + ph; c < K; c += 8 * U) {
      double2 v[U];
#pragma unroll
      for (int u = 0; u < U; ++u)
        v[u] = c + 8 * u < K ? reinterpret_cast<const double2*>(
                                   s.X)[(size_t)i + (size_t)(c + 8 * u) * s.ld]
                             : make_double2(0.0, 0.0);
#pragma unroll
      for (int u = 0; u < U; ++u) x.add(v[u]);
    }
  }
  if (x.bad) atomicOr(flag, 1);
  atomicMax(&red[lane], x.e);
  __syncthreads();
  if (threadIdx.x < 32 && i < s.lines && red[lane]) atomicMax(&s.e[i], red[lane]);
}

__device__ __forceinline__ void dd_max_right(const DdSide& s, int k0, int k1, int cb, int* flag) {
  const int lane = threadIdx.x & 31;
  const int j = cb * 8 + (threadIdx.x >> 5);
  if (j >= s.lines) return;  // whole warps only
  const double2* col = reinterpret_cast<const double2*>(s.X) + (size_t)j * s.ld;
  DdMax x;
  constexpr int U = 8;
  for (int k = k0 + lane; k < k1; k += 32 * U) {
    double2 v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = k + 32 * u < k1 ? col[k + 32 * u] : make_double2(0.0, 0.0);
#pragma unroll
    for (int u = 0; u < U; ++u) x.add(v[u]);
  }
  const bool bad = __any_sync(0xffffffffu, x.bad);
  const uint32_t e = __reduce_max_sync(0xffffffffu, x.e);
  if (lane == 0) {
    if (bad) atomicOr(flag, 1);
    if (e) atomicMax(&s.e[j], e);
  }
}

__global__ void __launch_bounds__(NT) dd_maxima(const __grid_constant__ DdPrepArgs p) {
  dep_ready();
  int local = blockIdx.x;
  if (local < p.nA) {
    const int nrb = (p.a.lines + 31) >> 5;
    const int k0 = (local / nrb) * p.spanA;
    dd_max_left(p.a, min(p.K, k0 + p.spanA), local % nrb, k0, p.flag);
  } else {
    local -= p.nA;
    const int ncb = (p.b.lines + 7) >> 3;
    const int k0 = (local / ncb) * p.spanB;
    dd_max_right(p.b, k0, min(p.K, k0 + p.spanB), local % ncb, p.flag);
  }
}

// Eight consecutive k of one line (E its exponent, OZ_ZERO_EXP: all zero).
__device__ __forceinline__ void dd_split8(const double2 (&v)[8], int E, const DdPrepArgs& p,
                                          const DdSide& s, size_t off) {
  unsigned long long h[4][DD_LIMBS];
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    __int128 a[2] = {0, 0};
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const double2 x = v[2 * t + u];
      // (a non-finite entry makes the whole result NaN: any integer will do)
      if (E != OZ_ZERO_EXP && sw_finite(x.x) && sw_finite(x.y)) {
        dd_add_int(x.x, E, p.w, a[u]);
        dd_add_int(x.y, E, p.w, a[u]);
      }
    }
    limbs_pair<DD_LIMBS>(a[0], a[1], h[t]);
  }
#pragma unroll
  for (int l = 0; l < OZ_MAX_MODULI; ++l) {
    if (l >= p.L) break;
    uint32_t x[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) x[t] = res_pair<DD_LIMBS>(h[t], l);
    *reinterpret_cast<uint4*>(s.planes + l * s.pstride + off) = make_uint4(x[0], x[1], x[2], x[3]);
  }
}

// Columns: as split_right of ozaki_prep.cu (coalesced reads turned to 8
// consecutive k per lane through shared memory).
__host__ __device__ __forceinline__ int dd_right_lanes(int Kp) {
  return Kp <= 64 ? 8 : (Kp <= 128 ? 16 : 32);
}

// Left blocks: rows [32 rb, + 32) x 64 k, a warp 8 rows x 32 k (lane =
// k-group + 4 row, as ozaki_prep.cu); right blocks as above.  Both end in the same dd_split8: its 32
// unrolled residues are most of the kernel's code, and two copies of it
// overran the instruction cache (160 us against 128 at n = 2048).
__global__ void __launch_bounds__(NT, 3) dd_split(const __grid_constant__ DdPrepArgs p) {
  __shared__ double2 turn[NT / 32][288];
  dep_wait();
  dep_ready();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool left = (int)blockIdx.x < p.nA;
  const DdSide& s = left ? p.a : p.b;
  int line, k;  // of the lane's first entry
  double2 v[8];
  if (left) {
    const int nrb = (s.lines + 31) >> 5;
    line = (blockIdx.x % nrb) * 32 + (warp & 3) * 8 + (lane >> 2);
    k = (blockIdx.x / nrb) * 64 + (warp >> 2) * 32 + (lane & 3) * 8;
#pragma unroll
    for (int t = 0; t < 8; ++t)
      v[t] = line < s.lines && k + t < p.K
                 ? reinterpret_cast<const double2*>(s.X)[(size_t)line + (size_t)(k + t) * s.ld]
                 : make_double2(0.0, 0.0);
  } else {
    const int lanes = dd_right_lanes(p.Kp), per = 8 * lanes, nkb = (p.Kp + per - 1) / per;
    const int local = blockIdx.x - p.nA;
    const int col0 = ((local / nkb) * 8 + warp) * (32 / lanes), k0 = (local % nkb) * per;
    double2* T = turn[warp];
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      const int x = 32 * t + lane, j = col0 + x / per, kk = k0 + (x & (per - 1));
      v[t] = j < s.lines && kk < p.K
                 ? reinterpret_cast<const double2*>(s.X)[(size_t)kk + (size_t)j * s.ld]
                 : make_double2(0.0, 0.0);
    }
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      const int x = 32 * t + lane;
      T[x + (x >> 3)] = v[t];
    }
    __syncwarp();
#pragma unroll
    for (int t = 0; t < 8; ++t) v[t] = T[9 * lane + t];
    line = col0 + lane / lanes;
    k = k0 + (lane & (lanes - 1)) * 8;
  }
  if (line >= s.lines || k >= p.Kp) return;
  dd_split8(v, dd_line_exp(s.e[line]), p, s, oz_tile_off(line, left ? OZ_BM : OZ_BN, k, p.Kp));
}

inline int cdiv(long a, long b) { return (int)((a + b - 1) / b); }

}  // namespace

int dd_prepare(int M, int N, int K, int Mp, int Np, int Kp, int L, int w, const double* A,
               long lda, const double* B, long ldb, uint32_t* eA, uint32_t* eB,
               uint16_t* planesA, uint16_t* planesB, int* flag, cudaStream_t st) {
  DdPrepArgs p;
  p.a = DdSide{A, lda, M, (size_t)Mp * Kp, planesA, eA};
  p.b = DdSide{B, ldb, N, (size_t)Np * Kp, planesB, eB};
  p.K = K;
  p.Kp = Kp;
  p.L = L;
  p.w = w;
  p.flag = flag;
  const int nrb = cdiv(M, 32), ncb = cdiv(N, 8);
  if (K > 0) {
    auto span = [&](int line_blocks, int least) {  // as ozaki_prep.cu
      int x = 1024;
      while (x > least && (long)line_blocks * cdiv(K, x) < 608) x >>= 1;
      return x;
    };
    p.spanA = span(nrb, 64);
    p.spanB = span(ncb, 256);
    p.nA = nrb * cdiv(K, p.spanA);
    dd_maxima<<<p.nA + ncb * cdiv(K, p.spanB), NT, 0, st>>>(p);
    VCPCU_LAUNCH_CHECK("dd_maxima");
  }
  p.nA = nrb * cdiv(Kp, 64);
  const int lanes = dd_right_lanes(Kp);
  const int blocks = p.nA + cdiv(N, 8 * (32 / lanes)) * cdiv(Kp, 8 * lanes);
  VCPCU_CUDA_TRY(launch_dep(K > 0, 1, dd_split, dim3(blocks), dim3(NT), 0, st, p));
  VCPCU_LAUNCH_CHECK("dd_split");
  return VCPCU_OK;
}

}  // namespace vcpcu
