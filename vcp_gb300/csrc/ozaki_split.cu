// ozaki_split.cu -- operand preparation of the slice form of the interval
// product (the CRT form's: ozaki_prep.cu): kv-style midrad of every interval entry (the
// same arithmetic as the plain form and as pidblas_assist::midrad,
// vcp/pidblas.hpp:43-51), per-row / per-column power-of-two exponents, and
// the bf16 digit planes that the tcgen05 slice GEMM consumes.
//
// Operands of C = [A]*[B] (A m x k, B k x n, kv layout, column-major):
//   left  (per row i):    mA  -> s   digits, round-to-nearest, exponent Em_i
//                         P = |mA| +ru rA -> sr digits, upward, exponent Ep_i
//                         rA  -> sr digits, upward, exponent Er_i
//                         delta_i = sum over slices and k of |digit|
//   right (per column j): mB  -> s   digits, round-to-nearest, exponent Fm_j
//                         rB  -> sr digits, upward, exponent Fr_j
//                         S = |mB| -> sr digits, upward, exponent Fm_j
//                         beta_j = sum_k |mB(k,j)| rounded upward
// Digit planes are K-major bf16: plane[p][row][k], row < Mp (or Np), k < Kp;
// the padding is zero.
#include "common.cuh"
#include "ozaki.cuh"
#include "ozaki_common.cuh"
#include "ozaki_residue.cuh"
#include "swfp.cuh"

namespace vcpcu {

__device__ __forceinline__ unsigned long long dbits(double x) {
  return (unsigned long long)__double_as_longlong(x);
}

template <int S>
__device__ __forceinline__ void digits_of(double x, int E, int up, int (&d)[S]) {
  if (E == OZ_ZERO_EXP || oz_zero(x)) {
#pragma unroll
    for (int q = 0; q < S; ++q) d[q] = 0;
    return;
  }
  if (S <= 7) {
    long long n = oz_scaled_int64(x, E, 8 * S, up);
#pragma unroll
    for (int p = S - 1; p >= 1; --p) {
      const int lo = (int)((unsigned long long)(n + 128) & 255ULL) - 128;
      d[p] = lo;
      n = (n - lo) >> 8;
    }
    d[0] = (int)n;
  } else {
    __int128 n = oz_scaled_int(x, E, S, up);
#pragma unroll
    for (int p = S - 1; p >= 1; --p) {
      const int lo = (int)((unsigned long long)(n + 128) & 255ULL) - 128;
      d[p] = lo;
      n = (n - lo) >> 8;
    }
    d[0] = (int)n;
  }
}

// ---------------------------------------------------------------- left factor
// Pass 1: kv midrad of every entry, stored as the planes mA, rA (column-major,
// ld = ldm), and the row maxima of |mA|, P = |mA| +ru rA and rA as double bit
// patterns (non-negative doubles order like their bit patterns).  One entry
// in four takes the FP64 instructions (sw_midrad_hw, the same bits), the
// others the integer-pipe form: the FP64 pipe then runs beside the integer
// one (at half, the FP64 pipe became the bound).
// Block: 32 rows x 8 column phases over a column range.
__global__ void __launch_bounds__(256)
oz_rowmax_left(int M, int K, const double* __restrict__ A, long lda, int cols_per_block,
               double* __restrict__ mA, double* __restrict__ rA, long ldm,
               unsigned long long* __restrict__ mx, int* __restrict__ flag) {
  __shared__ unsigned long long red[3][32];
  const int lane = threadIdx.x & 31, ph = threadIdx.x >> 5;
  const int i = blockIdx.x * 32 + lane;
  if (threadIdx.x < 32) red[0][lane] = red[1][lane] = red[2][lane] = 0;
  __syncthreads();
  unsigned long long am = 0, ap = 0, ar = 0;
  bool bad = false;
  if (i < M) {
    const int c0 = blockIdx.y * cols_per_block;
    const int c1 = min(K, c0 + cols_per_block);
    constexpr int U = 4;  // loads in flight per thread (see oz_colmax_right)
    for (int cb = c0 + ph; cb < c1; cb += 8 * U) {
      double2 e[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int c = cb + 8 * u;
        e[u] = c < c1 ? *reinterpret_cast<const double2*>(A + 2 * (i + (long)c * lda))
                      : make_double2(0.0, 0.0);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int c = cb + 8 * u;
        if (c >= c1) break;
        double m = 0.0, r = 0.0, p;
        if (sw_finite(e[u].x) && sw_finite(e[u].y)) {
          if (u == U - 1)
            sw_midrad_hw(e[u].x, e[u].y, m, r, p);
          else
            sw_midrad(e[u].x, e[u].y, m, r, p);
          am = max(am, dbits(oz_abs(m)));
          ap = max(ap, dbits(p));
          ar = max(ar, dbits(r));
        } else {
          bad = true;
        }
        mA[i + (long)c * ldm] = m;
        rA[i + (long)c * ldm] = r;
      }
    }
  }
  if (bad) atomicOr(flag, 1);
  atomicMax(&red[0][lane], am);
  atomicMax(&red[1][lane], ap);
  atomicMax(&red[2][lane], ar);
  __syncthreads();
  if (threadIdx.x < 32 && i < M) {
    atomicMax(&mx[3 * i + 0], red[0][lane]);
    atomicMax(&mx[3 * i + 1], red[1][lane]);
    atomicMax(&mx[3 * i + 2], red[2][lane]);
  }
}

// Exponents from the maxima (one thread per row or column).
__global__ void oz_exponents(int R, const unsigned long long* __restrict__ mx, int nper,
                             int* __restrict__ E) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= R) return;
  for (int t = 0; t < nper; ++t)
    E[nper * i + t] = oz_exponent(__longlong_as_double((long long)mx[nper * i + t]));
}

// Pass 2: digit planes of the left factor from the stored mA, rA.  Block:
// 32 rows x 64 k, 256 threads; digits are staged in shared memory and
// written K-contiguous (a transpose), 16 bytes per store.
constexpr int LT_R = 32, LT_K = 64, LT_KS = LT_K + 2;  // padded row: no bank conflicts
template <int S, int SR>
__global__ void __launch_bounds__(256)
oz_split_left(int M, int K, int Mp, int Kp, const double* __restrict__ mA,
              const double* __restrict__ rA, const int* __restrict__ E3,
              uint16_t* __restrict__ planes_m, uint16_t* __restrict__ planes_p,
              uint16_t* __restrict__ planes_r, unsigned long long* __restrict__ delta) {
  extern __shared__ int16_t sd[];  // digits [plane][LT_R][LT_KS], values in [-128, 128]
  constexpr int s = S, sr = SR, np = S + 2 * SR;
  const int tid = threadIdx.x;
  const int r = tid % LT_R, kph = tid / LT_R;  // 8 k phases
  const int i = blockIdx.y * LT_R + r;
  const int k0 = blockIdx.x * LT_K;
  int Em = OZ_ZERO_EXP, Ep = OZ_ZERO_EXP, Er = OZ_ZERO_EXP;
  if (i < M) {
    Em = E3[3 * i + 0];
    Ep = E3[3 * i + 1];
    Er = E3[3 * i + 2];
  }
  unsigned dsum = 0;
  int d[S], dr[SR];
  for (int kk = kph; kk < LT_K; kk += 8) {
    const int k = k0 + kk;
    double m = 0.0, rr = 0.0, p = 0.0;
    if (i < M && k < K) {
      m = mA[i + (long)k * M];
      rr = rA[i + (long)k * M];
      p = __dadd_ru(oz_abs(m), rr);
    }
    digits_of<S>(m, Em, 0, d);
#pragma unroll
    for (int q = 0; q < s; ++q) {
      sd[(q * LT_R + r) * LT_KS + kk] = (int16_t)d[q];
      dsum += (unsigned)abs(d[q]);
    }
    digits_of<SR>(p, Ep, 1, dr);
#pragma unroll
    for (int q = 0; q < sr; ++q) sd[((s + q) * LT_R + r) * LT_KS + kk] = (int16_t)dr[q];
    digits_of<SR>(rr, Er, 1, dr);
#pragma unroll
    for (int q = 0; q < sr; ++q) sd[((s + sr + q) * LT_R + r) * LT_KS + kk] = (int16_t)dr[q];
  }
  // per-row digit magnitude sum (midpoint slices)
  __shared__ unsigned rsum[LT_R];
  if (tid < LT_R) rsum[tid] = 0;
  __syncthreads();
  atomicAdd(&rsum[r], dsum);
  __syncthreads();
  if (tid < LT_R && blockIdx.y * LT_R + tid < M && rsum[tid])
    atomicAdd(&delta[blockIdx.y * LT_R + tid], (unsigned long long)rsum[tid]);
  // write-out: per plane, 32 rows x 64 k = 2048 bf16; thread -> 8 consecutive k
  const int wr = tid / 8, wk = (tid % 8) * 8;
  const int gi = blockIdx.y * LT_R + wr;
  for (int q = 0; q < np; ++q) {
    uint16_t* base;
    int pl;
    if (q < s) {
      base = planes_m;
      pl = q;
    } else if (q < s + sr) {
      base = planes_p;
      pl = q - s;
    } else {
      base = planes_r;
      pl = q - s - sr;
    }
    const int16_t* src = sd + (q * LT_R + wr) * LT_KS + wk;
    uint4 v;
    v.x = bf16_bits(src[0]) | (bf16_bits(src[1]) << 16);
    v.y = bf16_bits(src[2]) | (bf16_bits(src[3]) << 16);
    v.z = bf16_bits(src[4]) | (bf16_bits(src[5]) << 16);
    v.w = bf16_bits(src[6]) | (bf16_bits(src[7]) << 16);
    if (gi < Mp) *reinterpret_cast<uint4*>(base + ((size_t)pl * Mp + gi) * Kp + k0 + wk) = v;
  }
}

// --------------------------------------------------------------- right factor
// One block per column j < Np.  Pass 1 (thread t takes k = t, t+256, ...):
// midrad into the planes mB, rB (k contiguous), the column maxima and
// beta_j = RU sum |mB| (per-thread chains, then a pairwise tree).  Pass 2
// (thread t takes 8 consecutive k): digits from the stored planes, 16-byte
// stores.
template <int S, int SR>
__global__ void __launch_bounds__(256)
oz_split_right(int K, int N, int Kp, int Np, const double* __restrict__ B, long ldb,
               double* __restrict__ mBp, double* __restrict__ rBp,
               uint16_t* __restrict__ planes_m, uint16_t* __restrict__ planes_r,
               uint16_t* __restrict__ planes_s, int* __restrict__ F2,
               double* __restrict__ beta, int* __restrict__ flag) {
  const int j = blockIdx.x;
  const int tid = threadIdx.x;
  __shared__ unsigned long long smax[2];
  __shared__ double ssum[256];
  if (tid == 0) smax[0] = smax[1] = 0;
  __syncthreads();
  unsigned long long am = 0, ar = 0;
  double bsum = 0.0;
  bool bad = false;
  double* mcol = mBp + (size_t)j * Kp;
  double* rcol = rBp + (size_t)j * Kp;
  if (j < N) {
    for (int k = tid; k < K; k += 256) {
      const double2 e = *reinterpret_cast<const double2*>(B + 2 * (k + (long)j * ldb));
      double m = 0.0, r = 0.0, p;
      if (sw_finite(e.x) && sw_finite(e.y)) {
        sw_midrad(e.x, e.y, m, r, p);
        am = max(am, dbits(oz_abs(m)));
        ar = max(ar, dbits(r));
        bsum = __dadd_ru(bsum, fabs(m));
      } else {
        bad = true;
      }
      mcol[k] = m;
      rcol[k] = r;
    }
  }
  if (bad) atomicOr(flag, 1);
  atomicMax(&smax[0], am);
  atomicMax(&smax[1], ar);
  ssum[tid] = bsum;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (tid < w) ssum[tid] = __dadd_ru(ssum[tid], ssum[tid + w]);
    __syncthreads();
  }
  const int Fm = oz_exponent(__longlong_as_double((long long)smax[0]));
  const int Fr = oz_exponent(__longlong_as_double((long long)smax[1]));
  if (tid == 0 && j < N) {
    F2[2 * j + 0] = Fm;
    F2[2 * j + 1] = Fr;
    beta[j] = ssum[0];
  }
  // pass 2: the planes written above by this block are visible after the
  // barriers of the reduction
  constexpr int s = S, sr = SR;
  int d[S], dr[SR];
  uint32_t hm[S][4], hr[SR][4], hs[SR][4];
  for (int k0 = tid * 8; k0 < Kp; k0 += 256 * 8) {
#pragma unroll
    for (int h = 0; h < 8; ++h) {
      const int k = k0 + h;
      double m = 0.0, r = 0.0;
      if (j < N && k < K) {
        m = mcol[k];
        r = rcol[k];
      }
      digits_of<S>(m, Fm, 0, d);
#pragma unroll
      for (int q = 0; q < s; ++q) {
        const uint32_t b = bf16_bits(d[q]);
        if (h & 1) hm[q][h >> 1] |= b << 16; else hm[q][h >> 1] = b;
      }
      digits_of<SR>(r, Fr, 1, dr);
#pragma unroll
      for (int q = 0; q < sr; ++q) {
        const uint32_t b = bf16_bits(dr[q]);
        if (h & 1) hr[q][h >> 1] |= b << 16; else hr[q][h >> 1] = b;
      }
      digits_of<SR>(oz_abs(m), Fm, 1, dr);
#pragma unroll
      for (int q = 0; q < sr; ++q) {
        const uint32_t b = bf16_bits(dr[q]);
        if (h & 1) hs[q][h >> 1] |= b << 16; else hs[q][h >> 1] = b;
      }
    }
#pragma unroll
    for (int q = 0; q < s; ++q)
      *reinterpret_cast<uint4*>(planes_m + ((size_t)q * Np + j) * Kp + k0) =
          make_uint4(hm[q][0], hm[q][1], hm[q][2], hm[q][3]);
#pragma unroll
    for (int q = 0; q < sr; ++q) {
      *reinterpret_cast<uint4*>(planes_r + ((size_t)q * Np + j) * Kp + k0) =
          make_uint4(hr[q][0], hr[q][1], hr[q][2], hr[q][3]);
      *reinterpret_cast<uint4*>(planes_s + ((size_t)q * Np + j) * Kp + k0) =
          make_uint4(hs[q][0], hs[q][1], hs[q][2], hs[q][3]);
    }
  }
}

// ------------------------------------------------------------------ launchers
template <int S, int SR>
int launch_splits(const OzProblem& pb, const double* B, long ldb, OzWorkspace& ws,
                  cudaStream_t st) {
  dim3 g2(pb.Kp / LT_K, pb.Mp / LT_R);
  const size_t shm = sizeof(int16_t) * (size_t)(S + 2 * SR) * LT_R * LT_KS;
  VCPCU_CUDA_TRY(cudaFuncSetAttribute(oz_split_left<S, SR>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm));
  oz_split_left<S, SR><<<g2, 256, shm, st>>>(pb.M, pb.K, pb.Mp, pb.Kp, ws.midA, ws.radA, ws.E3,
                                             ws.a_mid, ws.a_p, ws.a_r, ws.delta);
  VCPCU_LAUNCH_CHECK("oz_split_left");
  oz_split_right<S, SR><<<pb.Np, 256, 0, st>>>(pb.K, pb.N, pb.Kp, pb.Np, B, ldb, ws.midB,
                                               ws.radB, ws.b_mid, ws.b_r, ws.b_s, ws.F2,
                                               ws.beta, ws.flag);
  VCPCU_LAUNCH_CHECK("oz_split_right");
  return VCPCU_OK;
}

int oz_prepare_slices(const OzProblem& pb, const double* A, long lda, const double* B, long ldb,
                      OzWorkspace& ws, cudaStream_t st) {
  VCPCU_CUDA_TRY(cudaMemsetAsync(ws.rowmax, 0, sizeof(unsigned long long) * 3 * (size_t)pb.Mp, st));
  VCPCU_CUDA_TRY(cudaMemsetAsync(ws.delta, 0, sizeof(unsigned long long) * (size_t)pb.Mp, st));
  VCPCU_CUDA_TRY(cudaMemsetAsync(ws.flag, 0, 4 * sizeof(int), st));  // every status word
  if (pb.sr != 2) {
    set_error("Ozaki form: radius slice count %d is not built (2 is)", pb.sr);
    return VCPCU_ERR_UNSUPPORTED;
  }
  if (pb.M > 0 && pb.K > 0) {
    const int cpb = 256;
    dim3 g1((pb.M + 31) / 32, (pb.K + cpb - 1) / cpb);
    oz_rowmax_left<<<g1, 256, 0, st>>>(pb.M, pb.K, A, lda, cpb, ws.midA, ws.radA, pb.M,
                                       ws.rowmax, ws.flag);
    VCPCU_LAUNCH_CHECK("oz_rowmax_left");
  }
  oz_exponents<<<(pb.Mp + 255) / 256, 256, 0, st>>>(pb.Mp, ws.rowmax, 3, ws.E3);
  VCPCU_LAUNCH_CHECK("oz_exponents");
  int st_ = VCPCU_OK;
  switch (pb.s) {
#define OZ_SPLIT_CASE(S)                                                          \
  case S:                                                                         \
    st_ = launch_splits<S, 2>(pb, B, ldb, ws, st);                                \
    break;
    OZ_SPLIT_CASE(2) OZ_SPLIT_CASE(3) OZ_SPLIT_CASE(4) OZ_SPLIT_CASE(5) OZ_SPLIT_CASE(6)
    OZ_SPLIT_CASE(7) OZ_SPLIT_CASE(8) OZ_SPLIT_CASE(9) OZ_SPLIT_CASE(10) OZ_SPLIT_CASE(11)
    OZ_SPLIT_CASE(12)
#undef OZ_SPLIT_CASE
    default:
      set_error("Ozaki form: slice count %d outside [2, 12]", pb.s);
      return VCPCU_ERR_INVALID_ARG;
  }
  return st_;
}

}  // namespace vcpcu
