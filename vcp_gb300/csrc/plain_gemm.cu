// plain_gemm.cu -- FP64 CUDA-core GEMMs with per-instruction directed
// rounding: the "plain form" of the verified product.
//
// Result definition (vblas/README.md, "packing layout"; the AVX-512 micro
// kernel vblas/rmatmul_avx512.hpp:195-242 keeps the C tile in registers and
// continues the chain across k blocks): entry C(i,j) is the sequential chain
//     c = +0.0;  for p = 0..K-1:  c = fma_dir(A(i,p), B(p,j), c)
// in ascending p.  Every thread here owns whole C entries and runs exactly
// that chain, so the kernels are bit-identical to vblas rmatmul/udmatmul for
// any tiling.  K tails are padded with +0.0 * +0.0 = +0.0 products, which
// leave every chain value unchanged in all three rounding modes (a -0.0
// accumulator can only arise under round-down, where -0.0 + +0.0 = -0.0).
//
// The interval kernel follows pidblas::mulmm (vcp/pidblas.hpp:239-294): its
// four dgemm_ calls become four chains per entry in one pass over A and B:
//     lo = chain_rd(mA*mB)          (:264-266)
//     up = chain_ru(mA*mB)          (:269-271)
//     t1 = chain_ru((|mA|+rA)*rB)   (:273-279; |mA|+rA rounded up)
//     t2 = chain_ru(rA*|mB|)        (:281)
//     T  = t1 +ru t2 ; up = up +ru T ; lo = lo -rd T   (:283-286)
// with mA, rA, mB, rB from kv-style midrad (pidblas.hpp:43-51).
#include <mutex>

#include "common.cuh"
#include "dirchain.cuh"
#include "plain_gemm.cuh"
#include "swfp.cuh"

namespace vcpcu {

namespace {

constexpr int BM = 64, BN = 64, BK = 16, NT = 256, BKI = 8;

// Kinds of chains a kernel runs per C entry.
enum Kind { K_RN = 0, K_RU = 1, K_RD = 2, K_UD = 3 };

template <int KIND>
__device__ __forceinline__ double fma_k(double a, double b, double c) {
  if (KIND == K_RU) return __fma_ru(a, b, c);
  if (KIND == K_RD) return __fma_rd(a, b, c);
  return __fma_rn(a, b, c);
}

// Tiles of the two products below: 32 rows (a row per lane) x 4 CW columns;
// each of four warps -- one per SM sub-partition -- owns CW columns.  Both are
// bound by the FP64 pipe (64 cycles per warp instruction), so what counts is
// that the SMs' sub-partitions get the same number of (32-row, column) chain
// sets: CW = 8, 4 or 2, whichever leaves the fullest one the least to do,
// the widest of equals.
constexpr int TROWS = 32;
// The cost of a width in blocks on the fullest SM x CW, with `penalty` 32nds
// more at CW = 4 and twice that at CW = 2 (a narrower block stages as much of
// A), and a quarter more for a single block on an SM (nothing runs while it
// waits at its barriers).  Interval product, us at CW = 8 / 4 / 2: 512^3 659 /
// 683 / 684, 256^3 254 / 142 / 119, 300 x 200 x 700 591 / 321 / 271.
inline int tile_cols(int M, int N, int penalty) {
  const long mt = (M + TROWS - 1) / TROWS;
  int best = 8;
  double cost = 0.0;
  for (int cw = 8, f = 32; cw >= 2; cw >>= 1, f += penalty) {
    const long rounds = (mt * ((N + 4 * cw - 1) / (4 * cw)) + 151) / 152;
    const double c = (rounds == 1 ? 1.25 : 1.0) * (double)rounds * cw * f;
    if (cw == 8 || c < cost) {
      best = cw;
      cost = c;
    }
  }
  return best;
}

// One-direction (KIND RN/RU/RD) or up+down (K_UD) point GEMM.
// GEMM naming: C(M x N) = A(M x K) * B(K x N), column-major.  n = 1024, both
// directions: 64 x 64 tiles 4.12 ms, these 3.47 ms (the FP64 rate).
template <int KIND, int CW>
__global__ void __launch_bounds__(128)
point_gemm_kernel(int M, int N, int K, const double* __restrict__ A, long lda,
                  const double* __restrict__ B, long ldb, double* __restrict__ C0,
                  double* __restrict__ C1, long ldc) {
  constexpr int NCH = (KIND == K_UD) ? 2 : 1, COLS = 4 * CW;
  constexpr int QA = TROWS * BK / 128, QB = COLS * BK / 128;
  __shared__ double As[2][BK][TROWS];
  __shared__ double Bs[2][BK][COLS];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int mt = (M + TROWS - 1) / TROWS;
  const int row0 = (blockIdx.x % mt) * TROWS, col0 = (blockIdx.x / mt) * COLS;
  const int b_k = tid % BK, b_j = tid / BK;

  double acc[NCH][CW];
#pragma unroll
  for (int c = 0; c < NCH; ++c)
#pragma unroll
    for (int j = 0; j < CW; ++j) acc[c][j] = 0.0;

  double ra[QA], rb[QB];
  auto load_tile = [&](int k0) {
#pragma unroll
    for (int q = 0; q < QA; ++q) {
      const int gi = row0 + lane, gk = k0 + warp + 4 * q;
      ra[q] = (gi < M && gk < K) ? A[gi + gk * lda] : 0.0;
    }
#pragma unroll
    for (int q = 0; q < QB; ++q) {
      const int hk = k0 + b_k, hj = col0 + b_j + (128 / BK) * q;
      rb[q] = (hk < K && hj < N) ? B[hk + hj * ldb] : 0.0;
    }
  };
  auto store_tile = [&](int buf) {
#pragma unroll
    for (int q = 0; q < QA; ++q) As[buf][warp + 4 * q][lane] = ra[q];
#pragma unroll
    for (int q = 0; q < QB; ++q) Bs[buf][b_k][b_j + (128 / BK) * q] = rb[q];
  };

  const int nk = (K + BK - 1) / BK;
  load_tile(0);
  store_tile(0);
  __syncthreads();
  for (int t = 0; t < nk; ++t) {
    const int buf = t & 1;
    if (t + 1 < nk) load_tile((t + 1) * BK);
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      const double a = As[buf][kk][lane];
#pragma unroll
      for (int j = 0; j < CW; ++j) {
        const double b = Bs[buf][kk][warp * CW + j];
        if (KIND == K_UD) {
          acc[0][j] = __fma_ru(a, b, acc[0][j]);
          acc[NCH - 1][j] = __fma_rd(a, b, acc[NCH - 1][j]);
        } else {
          acc[0][j] = fma_k<KIND>(a, b, acc[0][j]);
        }
      }
    }
    if (t + 1 < nk) store_tile(buf ^ 1);
    __syncthreads();
  }

  const int gi = row0 + lane;
#pragma unroll
  for (int j = 0; j < CW; ++j) {
    const int gj = col0 + warp * CW + j;
    if (gi < M && gj < N) {
      C0[gi + gj * ldc] = acc[0][j];
      if (KIND == K_UD) C1[gi + gj * ldc] = acc[NCH - 1][j];
    }
  }
}

template <int KIND>
void point_launch(int M, int N, int K, const double* A, long lda, const double* B, long ldb,
                  double* C0, double* C1, long ldc, cudaStream_t s) {
  const int cw = tile_cols(M, N, 0);
  const unsigned grid = (unsigned)((M + TROWS - 1) / TROWS) * (unsigned)((N + 4 * cw - 1) / (4 * cw));
  if (cw == 8)
    point_gemm_kernel<KIND, 8><<<grid, 128, 0, s>>>(M, N, K, A, lda, B, ldb, C0, C1, ldc);
  else if (cw == 4)
    point_gemm_kernel<KIND, 4><<<grid, 128, 0, s>>>(M, N, K, A, lda, B, ldb, C0, C1, ldc);
  else
    point_gemm_kernel<KIND, 2><<<grid, 128, 0, s>>>(M, N, K, A, lda, B, ldb, C0, C1, ldc);
}

// C = 0 for the n <= 0 (empty inner dimension) case of vblas rmatmul.
__global__ void zero_kernel(int M, int N, double* C, long ldc) {
  long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  long total = (long)M * N;
  for (; idx < total; idx += (long)gridDim.x * blockDim.x) {
    long i = idx % M, j = idx / M;
    C[i + j * ldc] = 0.0;
  }
}

}  // namespace

// kv-style midpoint/radius of [lo, up]: m = fl((lo + up) / 2) to nearest
// (halves taken separately when lo + up overflows), r = max(m - lo, up - m)
// rounded up, so that [m - r, m + r] contains [lo, up].  Explicit _rn
// intrinsics keep the compiler from contracting into an FMA.
__device__ __forceinline__ void midrad_dev(double lo, double up, double& m, double& r) {
  double s = __dadd_rn(lo, up);
  if (isfinite(s))
    m = __dmul_rn(s, 0.5);
  else
    m = __dadd_rn(__dmul_rn(lo, 0.5), __dmul_rn(up, 0.5));
  r = fmax(__dsub_ru(m, lo), __dsub_ru(up, m));
}

// Left factor: interval A (m x k, ld in intervals) -> planes mA, pA = |mA| +ru rA, rA
// (ld = M).  Right factor: interval B -> planes mB, rB (ld = K).
// With plus_rad == 0 the middle plane is |mA| itself (the Aᵀ[A] kernel).
__global__ void interval_prep_left(int M, int K, const double* __restrict__ A, long lda,
                                   double* __restrict__ mA, double* __restrict__ pA,
                                   double* __restrict__ rA, int plus_rad = 1) {
  long total = (long)M * K;
  for (long idx = (long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (long)gridDim.x * blockDim.x) {
    long i = idx % M, p = idx / M;
    const double* e = A + 2 * (i + p * lda);
    double m, r;
    midrad_dev(e[0], e[1], m, r);
    mA[idx] = m;
    rA[idx] = r;
    pA[idx] = plus_rad ? __dadd_ru(fabs(m), r) : fabs(m);
  }
}

__global__ void interval_prep_right(int K, int N, const double* __restrict__ B, long ldb,
                                    double* __restrict__ mB, double* __restrict__ rB) {
  long total = (long)K * N;
  for (long idx = (long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (long)gridDim.x * blockDim.x) {
    long p = idx % K, j = idx / K;
    const double* e = B + 2 * (p + j * ldb);
    double m, r;
    midrad_dev(e[0], e[1], m, r);
    mB[idx] = m;
    rB[idx] = r;
  }
}

namespace {

// Fused mid-rad interval GEMM over prepped planes (ld = M for A planes,
// ld = K for B planes).  Writes C as {inf, sup} pairs (ld in intervals).
//
// The two midpoint chains of an entry run on the FP64 pipe (warps 0 .. 3), the
// two radius chains -- sums of non-negative products rounded up -- on the
// integer pipe beside it (warps 4 .. 7 and 8 .. 11, dirchain.cuh, eight steps
// at a time), each warp on CW columns of the block's 32 rows, a row per lane.  The FP64
// pipe then has 2 instead of 4 instructions per entry and step: it is the
// bound, the integer warps take about half the issue slots beside it.  The
// radius chains' states live in shared memory between batches (their code is
// one loop over the columns).  n = 512: 64 x 64 tiles with four FP64 chains
// 2.07 ms, this 0.64; n = 1024 8.24 and
// 4.4 ms (3.5 at the FP64 rate).
constexpr int ITN = 384;  // threads
// Stages of BKI steps in which a radius chain takes the FP64 instructions:
// always (some lane's terms outgrow its unit), and where a batch does not go
// through.  With the single steps instead, one of them in FP64 for the warp at
// nearly every k, short inner dimensions were slower than four FP64 chains:
// 3000 x 3000, exponents over +-8, k = 16 / 32 / 64 / 256 1372 / 2490 / 4442 /
// 12603 us, now 1066 / 2036 / 3670 / 11649 (four FP64 chains 1063 / 2022 / 3940 /
// 15457); n = 1000 1152 us at k = 256 and narrow exponents, now 1136.  Batches
// tried in the second stage: 1073 / 2116 / 3776; FP64 up to stage 8: 3970 at 64.
constexpr int INEW = 2, IYOUNG = 4;
template <int CW>
struct ITile {
  struct Stage {
    double am[BKI][TROWS];
    ChainFactor ap[BKI][TROWS], ar[BKI][TROWS];
    double bm[BKI][4 * CW];
    ChainFactor br[BKI][4 * CW], bs[BKI][4 * CW];
  } st[2];
  long long c[2][4 * CW][TROWS];
  int U[2][4 * CW][TROWS];
};

// A stage's steps of a chain one by one; out of line, for the registers of the
// batches.
template <int COLS>
static __device__ __noinline__ DirChain chain_steps(DirChain x, const ChainFactor* a,
                                                    const ChainFactor* b, bool young) {
  chain_fma_steps<BKI>(
      x,
      [&](int p, ChainFactor* u, ChainFactor* v) {
        *u = a[p * TROWS];
        *v = b[p * COLS];
      },
      young);
  return x;
}

template <int CW>
__global__ void __launch_bounds__(ITN, 2)
interval_gemm_kernel(int M, int N, int K, const double* __restrict__ mA,
                     const double* __restrict__ pA, const double* __restrict__ rA,
                     const double* __restrict__ mB, const double* __restrict__ rB,
                     double* __restrict__ C, long ldc) {
  extern __shared__ __align__(16) uint8_t plain_smem[];
  ITile<CW>& sm = *reinterpret_cast<ITile<CW>*>(plain_smem);
  constexpr int COLS = 4 * CW;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int mt = (M + TROWS - 1) / TROWS;
  const int row0 = (blockIdx.x % mt) * TROWS, col0 = (blockIdx.x / mt) * COLS;
  const int b_k = tid % BKI, b_j = tid / BKI;

  double ram, rap, rar, rbm = 0.0, rbr = 0.0;
  auto load_tile = [&](int k0) {  // by the first 256 threads
    if (warp < 8) {
      const int gi = row0 + lane, gk = k0 + warp;
      const bool ok = gi < M && gk < K;
      const long o = gi + (long)gk * M;
      ram = ok ? mA[o] : 0.0;
      rap = ok ? pA[o] : 0.0;
      rar = ok ? rA[o] : 0.0;
    }
    if (b_j < COLS) {  // (COLS <= 32)
      const int hk = k0 + b_k, hj = col0 + b_j;
      const bool ok = hk < K && hj < N;
      const long o = hk + (long)hj * K;
      rbm = ok ? mB[o] : 0.0;
      rbr = ok ? rB[o] : 0.0;
    }
  };
  auto store_tile = [&](int buf) {
    auto& t = sm.st[buf];
    if (warp < 8) {
      t.am[warp][lane] = ram;
      t.ap[warp][lane] = chain_factor(rap);
      t.ar[warp][lane] = chain_factor(rar);
    }
    if (b_j < COLS) {
      t.bm[b_k][b_j] = rbm;
      t.br[b_k][b_j] = chain_factor(rbr);
      t.bs[b_k][b_j] = chain_factor(oz_abs(rbm));
    }
  };

  double lo[CW], up[CW];
#pragma unroll
  for (int j = 0; j < CW; ++j) lo[j] = up[j] = 0.0;
  const int w0 = (warp & 3) * CW;  // the warp's first column
  const int h = warp >= 8;               // the radius product of a chain warp
  if (warp >= 4) {
    for (int j = w0; j < w0 + CW; ++j) {
      sm.c[h][j][lane] = 0;
      sm.U[h][j][lane] = 1;
    }
  }
  const int nk = (K + BKI - 1) / BKI;
  load_tile(0);
  store_tile(0);
  __syncthreads();
  for (int t = 0; t < nk; ++t) {
    const auto& st = sm.st[t & 1];
    if (t + 1 < nk) load_tile((t + 1) * BKI);
    if (warp < 4) {
#pragma unroll
      for (int kk = 0; kk < BKI; ++kk) {
        const double a = st.am[kk][lane];
#pragma unroll
        for (int j = 0; j < CW; ++j) {
          const double b = st.bm[kk][w0 + j];
          lo[j] = __fma_rd(a, b, lo[j]);
          up[j] = __fma_ru(a, b, up[j]);
        }
      }
    } else {
      // (|mA| + rA) rB or rA |mB|
      const ChainFactor* a = (h ? &st.ar[0][0] : &st.ap[0][0]) + lane;
      const ChainFactor(*fb)[COLS] = h ? st.bs : st.br;
      ChainFactor fa[BKI];
#pragma unroll
      for (int kk = 0; kk < BKI; ++kk) fa[kk] = a[kk * TROWS];
#pragma unroll 1
      for (int j = w0; j < w0 + CW; ++j) {
        DirChain x{sm.c[h][j][lane], sm.U[h][j][lane]};
        if (t < INEW || !chain_fma_batch<BKI>(x, [&](int p, ChainFactor* u, ChainFactor* v) {
              *u = fa[p];
              *v = fb[p][j];
            }))
          x = chain_steps<COLS>(x, a, &fb[0][j], t < IYOUNG);
        sm.c[h][j][lane] = x.c;
        sm.U[h][j][lane] = x.U;
      }
    }
    if (t + 1 < nk) store_tile((t + 1) & 1);
    __syncthreads();
  }

  const int gi = row0 + lane;
  if (warp >= 4 || gi >= M) return;
#pragma unroll
  for (int j = 0; j < CW; ++j) {
    const int gj = col0 + w0 + j;
    if (gj >= N) break;
    const DirChain t1{sm.c[0][w0 + j][lane], sm.U[0][w0 + j][lane]},
        t2{sm.c[1][w0 + j][lane], sm.U[1][w0 + j][lane]};
    const double T = __dadd_ru(chain_value(t1), chain_value(t2));
    double* e = C + 2 * (gi + (long)gj * ldc);
    e[0] = __dsub_rd(lo[j], T);
    e[1] = __dadd_ru(up[j], T);
  }
}

template <int CW>
int interval_launch(int M, int N, int K, const double* mA, const double* pA, const double* rA,
                    const double* mB, const double* rB, double* C, long ldc, cudaStream_t s) {
  static std::mutex mu;
  static bool done[64] = {false};
  int dev = 0;
  VCPCU_CUDA_TRY(cudaGetDevice(&dev));
  {
    std::lock_guard<std::mutex> lk(mu);
    if (dev < 0 || dev >= 64 || !done[dev]) {
      VCPCU_CUDA_TRY(cudaFuncSetAttribute(interval_gemm_kernel<CW>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)sizeof(ITile<CW>)));
      if (dev >= 0 && dev < 64) done[dev] = true;
    }
  }
  const unsigned grid = (unsigned)((M + TROWS - 1) / TROWS) * (unsigned)((N + 4 * CW - 1) / (4 * CW));
  interval_gemm_kernel<CW><<<grid, ITN, sizeof(ITile<CW>), s>>>(M, N, K, mA, pA, rA, mB, rB, C, ldc);
  VCPCU_LAUNCH_CHECK("interval_gemm_kernel");
  return VCPCU_OK;
}

// R = Y [C] with imats::mul_m_im's own loop (vcp/imats.hpp:203-213), the
// product the base class runs on its local interval matrices (imats::eigsymge
// forms R = Y (A X - B X Lambda) with it): per entry c = [0, 0], then
// c = c + [y, y] * C(j, k) for j ascending, every step with kv's interval
// operations -- the product as the first smallest of RD(y cl), RD(y cu) and
// the first largest of RU(y cl), RU(y cu) (std::min_element / max_element
// over kv's four candidates), the sum rounded outward.  Eight FP64
// operations per term.  Padding terms are [+0, +0] and leave c unchanged.
__global__ void __launch_bounds__(NT)
imats_mulmm_kernel(int M, int N, int K, const double* __restrict__ Y, long ldy,
                   const double* __restrict__ C, long ldc, double* __restrict__ R, long ldr) {
  __shared__ double Ys[2][BKI][BM], Cl[2][BKI][BN], Cu[2][BKI][BN];
  const int tid = threadIdx.x;
  const int tr = tid / 16, tc = tid % 16;
  const int row0 = blockIdx.x * BM, col0 = blockIdx.y * BN;
  const int a_i = tid % BM, a_k = tid / BM;
  const int b_k = tid % BKI, b_j = tid / BKI;
  constexpr int QA = BKI / (NT / BM), QB = BN / (NT / BKI);
  double lo[4][4], up[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) lo[i][j] = up[i][j] = 0.0;
  double ry[QA], rl[QB], ru[QB];
  auto load_tile = [&](int k0) {
#pragma unroll
    for (int q = 0; q < QA; ++q) {
      const int gi = row0 + a_i, gk = k0 + a_k + (NT / BM) * q;
      ry[q] = (gi < M && gk < K) ? Y[gi + (long)gk * ldy] : 0.0;
    }
#pragma unroll
    for (int q = 0; q < QB; ++q) {
      const int hk = k0 + b_k, hj = col0 + b_j + (NT / BKI) * q;
      const bool ok = hk < K && hj < N;
      const double* e = C + 2 * (hk + (long)hj * ldc);
      rl[q] = ok ? e[0] : 0.0;
      ru[q] = ok ? e[1] : 0.0;
    }
  };
  auto store_tile = [&](int buf) {
#pragma unroll
    for (int q = 0; q < QA; ++q) Ys[buf][a_k + (NT / BM) * q][a_i] = ry[q];
#pragma unroll
    for (int q = 0; q < QB; ++q) {
      Cl[buf][b_k][b_j + (NT / BKI) * q] = rl[q];
      Cu[buf][b_k][b_j + (NT / BKI) * q] = ru[q];
    }
  };
  const int nk = (K + BKI - 1) / BKI;
  load_tile(0);
  store_tile(0);
  __syncthreads();
  for (int t = 0; t < nk; ++t) {
    const int buf = t & 1;
    if (t + 1 < nk) load_tile((t + 1) * BKI);
#pragma unroll 2
    for (int kk = 0; kk < BKI; ++kk) {
      double y[4], cl[4], cu[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) y[i] = Ys[buf][kk][tr + 16 * i];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        cl[j] = Cl[buf][kk][tc + 16 * j];
        cu[j] = Cu[buf][kk][tc + 16 * j];
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const double p1 = __dmul_rd(y[i], cl[j]), p2 = __dmul_rd(y[i], cu[j]);
          const double q1 = __dmul_ru(y[i], cl[j]), q2 = __dmul_ru(y[i], cu[j]);
          lo[i][j] = __dadd_rd(lo[i][j], p2 < p1 ? p2 : p1);
          up[i][j] = __dadd_ru(up[i][j], q1 < q2 ? q2 : q1);
        }
    }
    if (t + 1 < nk) store_tile(buf ^ 1);
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int gi = row0 + tr + 16 * i, gj = col0 + tc + 16 * j;
      if (gi < M && gj < N) {
        double* e = R + 2 * (gi + (long)gj * ldr);
        e[0] = lo[i][j];
        e[1] = up[i][j];
      }
    }
}

// [A]ᵀ[A] with pidblas::mulltmm semantics (vcp/pidblas.hpp:296-358) over
// prepped planes: X = Aᵀ (n x k: mX, aX = |mX|, rX), Y = A (k x n: mY, rY).
// Five chains per entry (i, j):
//   lo = RD Σ mX mY, up = RU Σ mX mY          (dsyrk under RD / RU)
//   t1 = RU Σ aX rY   = (|mA|ᵀ rA)(i,j)       (the dgemm temp)
//   t2 = RU Σ rX |mY| = (|mA|ᵀ rA)(j,i)
//   t3 = RU Σ rX rY   = (rAᵀ rA)(i,j)          (dsyrk of rA)
// temp = t1 +ru (t2 +ru t3) for i <= j; C(i,j) = C(j,i) =
// [lo -rd temp, up +ru temp] taken from the upper triangle.
__global__ void __launch_bounds__(NT)
syrk_interval_kernel(int N, int K, const double* __restrict__ mX, const double* __restrict__ aX,
                     const double* __restrict__ rX, const double* __restrict__ mY,
                     const double* __restrict__ rY, double* __restrict__ C, long ldc) {
  __shared__ double Xm[2][BKI][BM], Xa[2][BKI][BM], Xr[2][BKI][BM];
  __shared__ double Ym[2][BKI][BN], Yr[2][BKI][BN];
  const int row0 = blockIdx.x * BM, col0 = blockIdx.y * BN;
  if (col0 + BN <= row0) return;  // tile entirely below the diagonal
  const int tid = threadIdx.x;
  const int tr = tid / 16, tc = tid % 16;
  const int a_i = tid % BM, a_k = tid / BM;
  const int b_k = tid % BKI, b_j = tid / BKI;
  constexpr int QA = BKI / (NT / BM), QB = BN / (NT / BKI);
  double lo[4][4], up[4][4], t1[4][4], t2[4][4], t3[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) lo[i][j] = up[i][j] = t1[i][j] = t2[i][j] = t3[i][j] = 0.0;
  double ram[QA], raa[QA], rar[QA], rbm[QB], rbr[QB];
  auto load_tile = [&](int k0) {
#pragma unroll
    for (int q = 0; q < QA; ++q) {
      int gi = row0 + a_i, gk = k0 + a_k + (NT / BM) * q;
      bool ok = gi < N && gk < K;
      long o = gi + (long)gk * N;
      ram[q] = ok ? mX[o] : 0.0;
      raa[q] = ok ? aX[o] : 0.0;
      rar[q] = ok ? rX[o] : 0.0;
    }
#pragma unroll
    for (int q = 0; q < QB; ++q) {
      int hk = k0 + b_k, hj = col0 + b_j + (NT / BKI) * q;
      bool okb = hk < K && hj < N;
      long ob = hk + (long)hj * K;
      rbm[q] = okb ? mY[ob] : 0.0;
      rbr[q] = okb ? rY[ob] : 0.0;
    }
  };
  auto store_tile = [&](int buf) {
#pragma unroll
    for (int q = 0; q < QA; ++q) {
      Xm[buf][a_k + (NT / BM) * q][a_i] = ram[q];
      Xa[buf][a_k + (NT / BM) * q][a_i] = raa[q];
      Xr[buf][a_k + (NT / BM) * q][a_i] = rar[q];
    }
#pragma unroll
    for (int q = 0; q < QB; ++q) {
      Ym[buf][b_k][b_j + (NT / BKI) * q] = rbm[q];
      Yr[buf][b_k][b_j + (NT / BKI) * q] = rbr[q];
    }
  };
  const int nk = (K + BKI - 1) / BKI;
  load_tile(0);
  store_tile(0);
  __syncthreads();
  for (int t = 0; t < nk; ++t) {
    const int buf = t & 1;
    if (t + 1 < nk) load_tile((t + 1) * BKI);
#pragma unroll 2
    for (int kk = 0; kk < BKI; ++kk) {
      double xm[4], xa[4], xr[4], ym[4], yr[4], ya[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        xm[i] = Xm[buf][kk][tr + 16 * i];
        xa[i] = Xa[buf][kk][tr + 16 * i];
        xr[i] = Xr[buf][kk][tr + 16 * i];
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        ym[j] = Ym[buf][kk][tc + 16 * j];
        yr[j] = Yr[buf][kk][tc + 16 * j];
        ya[j] = fabs(ym[j]);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          lo[i][j] = __fma_rd(xm[i], ym[j], lo[i][j]);
          up[i][j] = __fma_ru(xm[i], ym[j], up[i][j]);
          t1[i][j] = __fma_ru(xa[i], yr[j], t1[i][j]);
          t2[i][j] = __fma_ru(xr[i], ya[j], t2[i][j]);
          t3[i][j] = __fma_ru(xr[i], yr[j], t3[i][j]);
        }
    }
    if (t + 1 < nk) store_tile(buf ^ 1);
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      int gi = row0 + tr + 16 * i, gj = col0 + tc + 16 * j;
      if (gi < N && gj < N && gi <= gj) {
        const double temp = __dadd_ru(t1[i][j], __dadd_ru(t2[i][j], t3[i][j]));
        const double u = __dadd_ru(up[i][j], temp);
        const double l = __dsub_rd(lo[i][j], temp);
        double* e = C + 2 * (gi + (long)gj * ldc);
        e[0] = l;
        e[1] = u;
        double* f = C + 2 * (gj + (long)gi * ldc);
        f[0] = l;
        f[1] = u;
      }
    }
}

inline int grid_1d(long total) {
  long b = (total + 255) / 256;
  if (b > 152 * 32) b = 152 * 32;
  if (b < 1) b = 1;
  return (int)b;
}

}  // namespace

int launch_point_gemm(int M, int N, int K, const double* A, long lda, const double* B,
                      long ldb, double* C0, double* C1, long ldc, int kind,
                      cudaStream_t s) {
  if (M <= 0 || N <= 0) return VCPCU_OK;
  if (K <= 0) {
    zero_kernel<<<grid_1d((long)M * N), 256, 0, s>>>(M, N, C0, ldc);
    VCPCU_LAUNCH_CHECK("zero_kernel");
    if (C1) {
      zero_kernel<<<grid_1d((long)M * N), 256, 0, s>>>(M, N, C1, ldc);
      VCPCU_LAUNCH_CHECK("zero_kernel");
    }
    return VCPCU_OK;
  }
  switch (kind) {
    case PK_UP:
      point_launch<K_RU>(M, N, K, A, lda, B, ldb, C0, nullptr, ldc, s);
      break;
    case PK_DOWN:
      point_launch<K_RD>(M, N, K, A, lda, B, ldb, C0, nullptr, ldc, s);
      break;
    case PK_UPDOWN:
      point_launch<K_UD>(M, N, K, A, lda, B, ldb, C0, C1, ldc, s);
      break;
    default:
      point_launch<K_RN>(M, N, K, A, lda, B, ldb, C0, nullptr, ldc, s);
      break;
  }
  VCPCU_LAUNCH_CHECK("point_gemm_kernel");
  return VCPCU_OK;
}

int launch_interval_gemm_plain(int M, int N, int K, const double* A, long lda,
                               const double* B, long ldb, double* C, long ldc,
                               double* ws, cudaStream_t s) {
  if (N <= kThinN)
    return launch_interval_gemm_thin(M, N, K, A, lda, THIN_INTERVAL, B, ldb, false, C, ldc, ws, s);
  // ws holds 3*M*K + 2*K*N doubles.
  double* mA = ws;
  double* pA = mA + (size_t)M * K;
  double* rA = pA + (size_t)M * K;
  double* mB = rA + (size_t)M * K;
  double* rB = mB + (size_t)K * N;
  interval_prep_left<<<grid_1d((long)M * K), 256, 0, s>>>(M, K, A, lda, mA, pA, rA);
  VCPCU_LAUNCH_CHECK("interval_prep_left");
  interval_prep_right<<<grid_1d((long)K * N), 256, 0, s>>>(K, N, B, ldb, mB, rB);
  VCPCU_LAUNCH_CHECK("interval_prep_right");
  switch (tile_cols(M, N, 3)) {
    case 8:
      return interval_launch<8>(M, N, K, mA, pA, rA, mB, rB, C, ldc, s);
    case 4:
      return interval_launch<4>(M, N, K, mA, pA, rA, mB, rB, C, ldc, s);
    default:
      return interval_launch<2>(M, N, K, mA, pA, rA, mB, rB, C, ldc, s);
  }
}

// (A k x n interval, lda) -> Aᵀ (n x k, ld = n) interval.
__global__ void transpose_interval(int K, int N, const double* __restrict__ A, long lda,
                                   double* __restrict__ At) {
  long total = (long)K * N;
  for (long idx = (long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (long)gridDim.x * blockDim.x) {
    long j = idx % N, p = idx / N;  // At(j, p) = A(p, j), writes coalesced
    const double* e = A + 2 * (p + j * lda);
    At[2 * idx] = e[0];
    At[2 * idx + 1] = e[1];
  }
}

int launch_isyrk_plain(int N, int K, const double* A, long lda, double* C, long ldc, double* ws,
                       cudaStream_t s) {
  // ws: At (2 N K) + mX, aX, rX (3 N K) + mY, rY (2 K N)
  double* At = ws;
  double* mX = At + 2 * (size_t)N * K;
  double* aX = mX + (size_t)N * K;
  double* rX = aX + (size_t)N * K;
  double* mY = rX + (size_t)N * K;
  double* rY = mY + (size_t)N * K;
  if (K > 0) {
    transpose_interval<<<grid_1d((long)N * K), 256, 0, s>>>(K, N, A, lda, At);
    VCPCU_LAUNCH_CHECK("transpose_interval");
    interval_prep_left<<<grid_1d((long)N * K), 256, 0, s>>>(N, K, At, N, mX, aX, rX, 0);
    VCPCU_LAUNCH_CHECK("interval_prep_left");
    interval_prep_right<<<grid_1d((long)K * N), 256, 0, s>>>(K, N, A, lda, mY, rY);
    VCPCU_LAUNCH_CHECK("interval_prep_right");
  }
  dim3 grid((N + BM - 1) / BM, (N + BN - 1) / BN);
  syrk_interval_kernel<<<grid, NT, 0, s>>>(N, K, mX, aX, rX, mY, rY, C, ldc);
  VCPCU_LAUNCH_CHECK("syrk_interval_kernel");
  return VCPCU_OK;
}

size_t isyrk_plain_ws_bytes(int N, int K) { return sizeof(double) * 7 * (size_t)N * K; }

int launch_imats_mulmm(int M, int N, int K, const double* Y, long ldy, const double* C, long ldc,
                       double* R, long ldr, cudaStream_t s) {
  if (M <= 0 || N <= 0) return VCPCU_OK;
  dim3 grid((M + BM - 1) / BM, (N + BN - 1) / BN);
  imats_mulmm_kernel<<<grid, NT, 0, s>>>(M, N, K > 0 ? K : 0, Y, ldy, C, ldc, R, ldr);
  VCPCU_LAUNCH_CHECK("imats_mulmm_kernel");
  return VCPCU_OK;
}

size_t interval_gemm_plain_ws_bytes(int M, int N, int K) {
  if (N <= kThinN) return interval_gemm_thin_ws_bytes(N, K);
  return sizeof(double) * (3 * (size_t)M * K + 2 * (size_t)K * N);
}

}  // namespace vcpcu
