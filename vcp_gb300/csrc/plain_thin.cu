// plain_thin.cu -- sequential directed chains over the rows of a matrix: the
// plain interval product with a thin right factor (N <= kThinN columns: the
// matrix-vector products of imats::linearsolve, vcp/imats.hpp:305-309, which
// pdblas hands to dgemv_, vcp/pdblas.hpp:96-100) and the row sums of |X| of
// its norms (vcp/mats.hpp:1583-1597).
//
// Both are bound by their chains, one per row and kind, in ascending column
// order: GB300's FP64 pipe takes 64 cycles for a warp instruction whatever
// its active lanes, and 64 for the next one of the same chain.  So every
// chain has a lane of its own and the chains of a kind share a warp.  The four
// chains of a product run in FP64, one kind on each sub-partition of an SM; the
// row sums, of non-negative terms, on the integer pipe (dirchain.cuh).
// Everything that is not the chain -- midrad, kv |.|, significands and
// exponents -- is done ahead of it by four producer warps, which stream the
// matrix through a ring of cp.async stages and leave one processed stage of 16
// columns for the chain warps per barrier.  Measured at n = 4096, against two
// FP64 chains per lane (two lanes a row) and separate midrad, shift and |.|
// passes: interval x point vector 658 -> 224 us, point x interval vector
// 361 -> 208, |E| x vector 867 -> 221, norm 311 -> 128; at n = 1225 the norm
// and the interval sums of |X| 230 -> 47 us (three passes before).  (About 105
// cycles a step; bare chains on all four sub-partitions take 76 with operands
// in registers and 82 with loads from shared memory.  Twice the producer warps,
// or a stage's operands loaded ahead of its first step, left the time as it is.)
//   With the radius chains of the product on the integer pipe a chain's terms
// that outgrow its unit cost steps of their own, one lane's for all 32: an inner
// dimension of 64 (100000 x 16) took 2653 us where two lanes a row had taken 940
// and this form takes 724, exponents over +-600 (4000 x 3, k = 4000) 2099 for
// 1954 and now 410.  Narrow spreads at k = 4096: 3 columns 535 and 418 us, 8
// columns 917 and 1057, 16 columns 1965 and 1912.
#include "common.cuh"
#include "dirchain.cuh"
#include "ozaki_prep.cuh"
#include "plain_gemm.cuh"
#include "swfp.cuh"

#include <mutex>

namespace vcpcu {

namespace {

constexpr int TR = 32;      // rows of a block: one per lane
constexpr int TG = 16;      // columns of a stage
constexpr int TSTAGES = 6;  // 8 KB each
constexpr int TB = 8;       // steps of a batch

__device__ __forceinline__ void cp16(void* dst, const void* src, bool ok) {
  const int bytes = ok ? 16 : 0;  // 0: zero fill
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void cp8(void* dst, const void* src, bool ok) {
  const int bytes = ok ? 8 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Producer threads (0 .. 127): each copies and later processes its own four
// entries of a stage, x = thread + 128 q: row x % 32, column x / 32 -- no
// barrier between copy and use.  Entries past the ends become zeros; an
// 8-byte aligned matrix goes in halves.
constexpr int PT = 128, QE = TG * TR / PT;
__device__ __forceinline__ void stage_intervals(double2* stage, int t, const double* X, long ld,
                                                int i0, int rows, int c0, int cols, bool al16) {
#pragma unroll
  for (int q = 0; q < QE; ++q) {
    const int x = t + PT * q, r = x % TR, c = x / TR;
    const bool ok = i0 + r < rows && c0 + c < cols;
    const double* src = ok ? X + 2 * ((size_t)(i0 + r) + (size_t)(c0 + c) * ld) : X;
    if (al16) {
      cp16(&stage[x], src, ok);
    } else {
      cp8(&stage[x].x, src, ok);
      cp8(&stage[x].y, src + (ok ? 1 : 0), ok);
    }
  }
}
__device__ __forceinline__ void stage_points(double* stage, int t, const double* X, long ld,
                                             int i0, int rows, int c0, int cols) {
#pragma unroll
  for (int q = 0; q < QE; ++q) {
    const int x = t + PT * q, r = x % TR, c = x / TR;
    const bool ok = i0 + r < rows && c0 + c < cols;
    cp8(&stage[x], ok ? X + (size_t)(i0 + r) + (size_t)(c0 + c) * ld : X, ok);
  }
}

// kv midrad of an entry: m, P = RU(|m| + r) and r.  Narrow entries, zeros and
// the [0, u] that kv |.| makes of an entry around zero (m = r = u / 2, P = u)
// in integer operations.
struct Mid {
  double m, P, r;
};
static __device__ __noinline__ Mid entry_mid_general(double lo, double up) {
  Mid x;
  if (!sw_midrad_wide(lo, up, x.m, x.r, x.P)) sw_midrad_hw(lo, up, x.m, x.r, x.P);
  return x;
}
__device__ __forceinline__ Mid entry_mid(double2 v) {
  const Words lo = words_of(sw_bits(v.x)), up = words_of(sw_bits(v.y));
  const bool from0 = (lo.hi | lo.lo) == 0 && up.hi - 0x00200000u < 0x7fe00000u - 0x00200000u;
  if (from0) {
    const double half = sw_double(w64(up) - (1ULL << 52));
    return Mid{half, v.y, half};
  }
  if (!iv_narrow(lo, up) && !iv_zero(lo, up)) return entry_mid_general(v.x, v.y);
  Words m, P;
  uint64_t D;
  iv_midrad(lo, up, &m, &D, &P);
  // D 2^(e - 1075), a normal double or 0
  const int bl = iv_bitlen64(D);
  const uint64_t r = D ? ((uint64_t)(iv_exp(lo) + bl - 54) << 52) + (D << ((53 - bl) & 63)) : 0ULL;
  return Mid{sw_double(w64(m)), sw_double(w64(P)), sw_double(r)};
}

// E - 1 (outward); out of line, since FP64 instructions in the loop over the
// entries would take the FP64 pipe's time even predicated off.
static __device__ __noinline__ double2 minus_one(double2 e) {
  return make_double2(__dsub_rd(e.x, 1.0), __dsub_ru(e.y, 1.0));
}
// kv |E| of an entry.
__device__ __forceinline__ double2 entry_abs(double2 e) {
  double lo, up;
  sw_abs_iv(e.x, e.y, lo, up);
  return make_double2(lo, up);
}

// -------------------------------------------------------------- thin product
// Block: 32 rows x NB columns of C; four chain warps, a row per lane, by role
//   0  the round-down midpoint chain, negated into a round-up one
//      (RD(a b + c) = -RU((-a) b + (-c)), signed zeros included)
//   1  the round-up midpoint chain
//   2  RU((|mA| +ru rA) rB)
//   3  RU(rA |mB|)
// and T = 2 +ru 3, C = [1st -rd T, 2nd +ru T] as pidblas::mulmm combines them;
// four producer warps.  A step past K multiplies zeros and leaves every chain
// unchanged.
template <int NB>
struct ThinStage {
  double m[TG * TR];
  double f[2][TG * TR];  // P, r
  double bm[TG][NB];
  double fb[2][TG][NB];  // rB, |mB|
};
template <int NB>
struct ThinSmem {
  double2 ring[TSTAGES][TG * TR];
  ThinStage<NB> st[2];
  double T[2][TR][NB + 1];
};

template <int NB, int LEFT>
__global__ void __launch_bounds__(256)
interval_gemm_thin_kernel(int M, int N, int K, const double* __restrict__ A, long lda,
                          const double* __restrict__ mB, const double* __restrict__ rB,
                          double* __restrict__ C, long ldc) {
  extern __shared__ __align__(16) uint8_t thin_smem[];
  ThinSmem<NB>& sm = *reinterpret_cast<ThinSmem<NB>*>(thin_smem);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i0 = blockIdx.x * TR, i = i0 + lane, j0 = blockIdx.y * NB;
  const int ng = (K + TG - 1) / TG;
  if (warp >= 4) {
    const int t = threadIdx.x - PT;
    const bool al16 = ((uintptr_t)A & 15) == 0;
    auto issue = [&](int g) {
      if (g < ng) {
        double2* S = sm.ring[g % TSTAGES];
        if (LEFT == THIN_POINT)
          stage_points(reinterpret_cast<double*>(S), t, A, lda, i0, M, g * TG, K);
        else
          stage_intervals(S, t, A, lda, i0, M, g * TG, K, al16);
      }
      cp_commit();
    };
    constexpr int QB = (TG * NB + PT - 1) / PT;  // right entries per thread and stage
    double bm[QB], br[QB];
    auto load_b = [&](int g) {
#pragma unroll
      for (int q = 0; q < QB; ++q) {
        const int x = t + PT * q, k = g * TG + x % TG, j = j0 + x / TG;
        const bool ok = x < TG * NB && k < K && j < N;
        bm[q] = ok ? mB[k + (size_t)j * K] : 0.0;
        br[q] = ok ? rB[k + (size_t)j * K] : 0.0;
      }
    };
    for (int g = 0; g < TSTAGES - 1; ++g) issue(g);
    load_b(0);
    for (int g = 0; g <= ng; ++g) {
      if (g < ng) {
        cp_wait<TSTAGES - 2>();
        ThinStage<NB>& st = sm.st[g & 1];
#pragma unroll
        for (int q = 0; q < QB; ++q) {
          const int x = t + PT * q;
          if (x < TG * NB) {
            st.bm[x % TG][x / TG] = bm[q];
            st.fb[0][x % TG][x / TG] = br[q];
            st.fb[1][x % TG][x / TG] = oz_abs(bm[q]);
          }
        }
        load_b(g + 1);
        const double2* S = sm.ring[g % TSTAGES];
#pragma unroll
        for (int q = 0; q < QE; ++q) {
          const int x = t + PT * q;
          Mid v;
          if (LEFT == THIN_POINT) {
            const double a = reinterpret_cast<const double*>(S)[x];
            v = Mid{a, oz_abs(a), 0.0};
          } else {
            double2 e = S[x];
            if (LEFT == THIN_ABS_SHIFT) {
              if (g * TG + x / TR == i0 + x % TR) e = minus_one(e);
              e = entry_abs(e);
            }
            v = entry_mid(e);
          }
          st.m[x] = v.m;
          st.f[0][x] = v.P;
          st.f[1][x] = v.r;
        }
        issue(g + TSTAGES - 1);  // (into the slot of stage g - 1, this thread's own)
      }
      __syncthreads();  // stage g is there; stage g - 1 has been used
    }
  } else {
    const int role = warp;
    double c[NB];
#pragma unroll
    for (int j = 0; j < NB; ++j) c[j] = role == 0 ? -0.0 : 0.0;
    for (int g = 0; g <= ng; ++g) {
      if (g > 0) {
        const ThinStage<NB>& st = sm.st[(g - 1) & 1];
        const double* fa = (role < 2 ? st.m : st.f[role - 2]) + lane;
        const double(*fb)[NB] = role < 2 ? st.bm : st.fb[role - 2];
        const uint64_t neg = role == 0 ? 1ULL << 63 : 0ULL;
#pragma unroll
        for (int p = 0; p < TG; ++p) {
          const double a = sw_double(sw_bits(fa[p * TR]) ^ neg);
#pragma unroll
          for (int j = 0; j < NB; ++j) c[j] = __fma_ru(a, fb[p][j], c[j]);
        }
      }
      __syncthreads();
    }
    if (role >= 2) {
#pragma unroll
      for (int j = 0; j < NB; ++j) sm.T[role - 2][lane][j] = c[j];
    }
    asm volatile("bar.sync 1, 128;" ::: "memory");  // the four chain warps
    if (role < 2 && i < M) {
#pragma unroll
      for (int j = 0; j < NB; ++j) {
        if (j0 + j >= N) break;
        const double T = __dadd_ru(sm.T[0][lane][j], sm.T[1][lane][j]);
        double* e = C + 2 * ((size_t)i + (size_t)(j0 + j) * ldc);
        e[role] = role == 0 ? __dsub_rd(sw_neg(c[j]), T) : __dadd_ru(c[j], T);
      }
    }
  }
}

// Planes of the thin right factor (K x N, ld = K): kv midrad of an interval
// B, or the point entries with zero radii (the midrad of [b, b]).
template <bool B_POINT>
__global__ void thin_prep_right(int K, int N, const double* __restrict__ B, long ldb,
                                double* __restrict__ mB, double* __restrict__ rB) {
  const long total = (long)K * N;
  for (long idx = (long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (long)gridDim.x * blockDim.x) {
    const long p = idx % K, j = idx / K;
    if (B_POINT) {
      mB[idx] = B[p + j * ldb];
      rB[idx] = 0.0;
    } else {
      const double* e = B + 2 * (p + j * ldb);
      double m, r, P;
      sw_midrad_hw(e[0], e[1], m, r, P);
      mB[idx] = m;
      rB[idx] = r;
    }
  }
}

// ------------------------------------------------------------------ row sums
// Sums of kv |X| (SHIFT: |X - I|) along the rows: chain warp 0 the upper ends
// rounded up, chain warp 1 (BOTH) the lower ends rounded down, integer chains;
// four producer warps after them.
struct SumStage {
  long long M[TG * TR];
  int e[TG * TR];
  double v[TG * TR];
};
template <bool BOTH>
struct SumSmem {
  double2 ring[TSTAGES][TG * TR];
  SumStage st[2][BOTH ? 2 : 1];
};

template <bool SHIFT, bool BOTH>
__global__ void __launch_bounds__(BOTH ? 192 : 160)
abs_row_sums_kernel(int n, const double* __restrict__ X, long ldx, double* __restrict__ rows,
                    double* __restrict__ sums) {
  extern __shared__ __align__(16) uint8_t thin_smem[];
  SumSmem<BOTH>& sm = *reinterpret_cast<SumSmem<BOTH>*>(thin_smem);
  constexpr int CW = BOTH ? 2 : 1;  // chain warps
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i0 = blockIdx.x * TR, i = i0 + lane;
  const int ng = (n + TG - 1) / TG;
  if (warp >= CW) {
    const int t = threadIdx.x - 32 * CW;
    auto issue = [&](int g) {
      if (g < ng)
        stage_intervals(sm.ring[g % TSTAGES], t, X, ldx, i0, n, g * TG, n, true);
      cp_commit();
    };
    for (int g = 0; g < TSTAGES - 1; ++g) issue(g);
    for (int g = 0; g <= ng; ++g) {
      if (g < ng) {
        cp_wait<TSTAGES - 2>();
        const double2* S = sm.ring[g % TSTAGES];
#pragma unroll
        for (int q = 0; q < QE; ++q) {
          const int x = t + PT * q;
          double2 e = S[x];
          if (SHIFT && g * TG + x / TR == i0 + x % TR) e = minus_one(e);
          e = entry_abs(e);
#pragma unroll
          for (int w = 0; w < CW; ++w) {
            SumStage& st = sm.st[g & 1][w];
            const double v = w == 0 ? e.y : e.x;
            long long M;
            int f;
            chain_split(sw_bits(v), &M, &f);
            st.M[x] = M;
            st.e[x] = f;
            st.v[x] = v;
          }
        }
        issue(g + TSTAGES - 1);
      }
      __syncthreads();
    }
  } else {
    DirChain c = chain_zero();
    for (int g = 0; g <= ng; ++g) {
      if (g > 0) {
        const SumStage& st = sm.st[(g - 1) & 1][warp];
        // the chain starts as its first term (0 + x would lose a -0); entries
        // past the last column are zeros and add nothing
        if (g == 1) c = chain_of(st.v[lane]);
#pragma unroll 1
        for (int p0 = 0; p0 < TG; p0 += TB) {
          auto get = [&](int p, long long* M, int* e) {
            const int x = (p0 + p) * TR + lane;
            const bool first = g == 1 && p0 + p == 0;
            *M = first ? 0 : st.M[x];
            *e = first ? CHAIN_ZERO : st.e[x];
          };
          auto value = [&](int p) { return st.v[(p0 + p) * TR + lane]; };
          if (BOTH && warp == 1)
            chain_add_n<false, TB>(c, get, value);
          else
            chain_add_n<true, TB>(c, get, value);
        }
      }
      __syncthreads();
    }
    if (i < n) {
      const double v = chain_value(c);
      if (BOTH) sums[2 * i + (warp == 1 ? 0 : 1)] = v;
      if (warp == 0) rows[i] = v;
    }
  }
}

// The dynamic shared memory of a kernel, opted into once per device.
template <auto KERNEL>
int smem_optin(size_t bytes) {
  static std::mutex mu;
  static bool done[64] = {false};
  int dev = 0;
  VCPCU_CUDA_TRY(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  if (dev >= 0 && dev < 64 && done[dev]) return VCPCU_OK;
  VCPCU_CUDA_TRY(
      cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  if (dev >= 0 && dev < 64) done[dev] = true;
  return VCPCU_OK;
}

template <int NB, int LEFT>
int thin_launch(int M, int N, int K, const double* A, long lda, const double* mB,
                const double* rB, double* C, long ldc, cudaStream_t s) {
  constexpr size_t bytes = sizeof(ThinSmem<NB>);
  if (int e = smem_optin<interval_gemm_thin_kernel<NB, LEFT>>(bytes)) return e;
  const dim3 grid((M + TR - 1) / TR, (N + NB - 1) / NB);
  interval_gemm_thin_kernel<NB, LEFT><<<grid, 256, bytes, s>>>(M, N, K, A, lda, mB, rB, C, ldc);
  VCPCU_LAUNCH_CHECK("interval_gemm_thin_kernel");
  return VCPCU_OK;
}

// Columns of a block (1, 2, 4, 8 or 16) from an estimate of the cycles: a
// block keeps each sub-partition's FP64 pipe for 64 cycles a step and column,
// the pipes are shared by the up to three blocks of an SM (two from four columns
// on: shared memory), and the blocks of a last wave land together on the SMs that
// are free first; a wave's fill and end take about 4000 cycles.  Single columns
// come out up to a quarter better than that: a tenth in their favour.  us for 1 /
// 2 / 4 / 8 / 16 columns, the estimate's choice in brackets: 4096 x 16, k = 4096
// [1914] 2373 2086 2071 2478; 4096 x 8 1089 1585 [1051] 1255; 8192 x 2, k = 8192
// 1260 [1077]; 5000 x 3, k = 5000 [783] 973 1279; 10000 x 16, k = 1000 [1123]
// 1184 1196 1398 1650; 100000 x 16, k = 16 341 271 253 226 [224].
inline int thin_cols(int M, int N, int K) {
  const long rb = (M + TR - 1) / TR;
  int best = 1;
  double cost = 0.0;
  for (int nb = 1; nb < 2 * N && nb <= kThinN; nb <<= 1) {
    const long blocks = rb * ((N + nb - 1) / nb), per = nb <= 2 ? 3 : 2;
    const long waves = (blocks + 152 * per - 1) / (152 * per);
    const long depth = waves == 1 ? (blocks + 151) / 152 : per * waves;
    const double c =
        (nb == 1 ? 64.0 : 70.4 * nb) * (double)depth * K + 4000.0 * (double)waves;
    if (nb == 1 || c < cost) {
      best = nb;
      cost = c;
    }
  }
  return best;
}

template <int NB>
int thin_launch_left(ThinLeft left, int M, int N, int K, const double* A, long lda,
                     const double* mB, const double* rB, double* C, long ldc, cudaStream_t s) {
  switch (left) {
    case THIN_POINT:
      return thin_launch<NB, THIN_POINT>(M, N, K, A, lda, mB, rB, C, ldc, s);
    case THIN_ABS_SHIFT:
      return thin_launch<NB, THIN_ABS_SHIFT>(M, N, K, A, lda, mB, rB, C, ldc, s);
    default:
      return thin_launch<NB, THIN_INTERVAL>(M, N, K, A, lda, mB, rB, C, ldc, s);
  }
}

template <bool SHIFT, bool BOTH>
int row_sums_launch(int n, const double* X, long ldx, double* rows, double* sums, cudaStream_t s) {
  constexpr size_t bytes = sizeof(SumSmem<BOTH>);
  if (int e = smem_optin<abs_row_sums_kernel<SHIFT, BOTH>>(bytes)) return e;
  abs_row_sums_kernel<SHIFT, BOTH>
      <<<(n + TR - 1) / TR, BOTH ? 192 : 160, bytes, s>>>(n, X, ldx, rows, sums);
  VCPCU_LAUNCH_CHECK("abs_row_sums_kernel");
  return VCPCU_OK;
}

}  // namespace

int launch_interval_gemm_thin(int M, int N, int K, const double* A, long lda, ThinLeft left,
                              const double* B, long ldb, bool b_point, double* C, long ldc,
                              double* ws, cudaStream_t s) {
  if (M <= 0 || N <= 0) return VCPCU_OK;
  if (N > kThinN) {
    set_error("interval_gemm_thin: N = %d exceeds %d", N, kThinN);
    return VCPCU_ERR_INVALID_ARG;
  }
  if (K < 0) K = 0;
  // The kernel reads A while blocks of the same rows and other columns store C:
  // where the two overlap (a product in place), it reads a copy.
  Scratch copy;
  if (K > 0) {
    const size_t esz = left == THIN_POINT ? 8 : 16;
    const uintptr_t a0 = (uintptr_t)A, a1 = a0 + esz * ((size_t)(K - 1) * lda + M);
    const uintptr_t c0 = (uintptr_t)C, c1 = c0 + 16 * ((size_t)(N - 1) * ldc + M);
    if (a0 < c1 && c0 < a1) {
      if (int e = copy.alloc(esz * (size_t)M * K, s)) return e;
      VCPCU_CUDA_TRY(cudaMemcpy2DAsync(copy.ptr, esz * M, A, esz * lda, esz * M, K,
                                       cudaMemcpyDeviceToDevice, s));
      A = (const double*)copy.ptr;
      lda = M;
    }
  }
  double* mB = ws;
  double* rB = mB + (size_t)K * N;
  if (K > 0) {
    const long total = (long)K * N;
    const int blocks = (int)((total + 255) / 256 < 1216 ? (total + 255) / 256 : 1216);
    if (b_point)
      thin_prep_right<true><<<blocks, 256, 0, s>>>(K, N, B, ldb, mB, rB);
    else
      thin_prep_right<false><<<blocks, 256, 0, s>>>(K, N, B, ldb, mB, rB);
    VCPCU_LAUNCH_CHECK("thin_prep_right");
  }
  const int nb = thin_cols(M, N, K);
  if (nb == 1) return thin_launch_left<1>(left, M, N, K, A, lda, mB, rB, C, ldc, s);
  if (nb == 2) return thin_launch_left<2>(left, M, N, K, A, lda, mB, rB, C, ldc, s);
  if (nb == 4) return thin_launch_left<4>(left, M, N, K, A, lda, mB, rB, C, ldc, s);
  if (nb == 8) return thin_launch_left<8>(left, M, N, K, A, lda, mB, rB, C, ldc, s);
  return thin_launch_left<16>(left, M, N, K, A, lda, mB, rB, C, ldc, s);
}

size_t interval_gemm_thin_ws_bytes(int N, int K) {
  return sizeof(double) * 2 * (size_t)(K > 0 ? K : 1) * (N > 0 ? N : 1);
}

int launch_abs_row_sums(int n, const double* X, long ldx, bool shift, double* rows, double* sums,
                        cudaStream_t s) {
  if (n <= 0) return VCPCU_OK;
  if (sums)
    return shift ? row_sums_launch<true, true>(n, X, ldx, rows, sums, s)
                 : row_sums_launch<false, true>(n, X, ldx, rows, sums, s);
  return shift ? row_sums_launch<true, false>(n, X, ldx, rows, sums, s)
               : row_sums_launch<false, false>(n, X, ldx, rows, sums, s);
}

}  // namespace vcpcu
