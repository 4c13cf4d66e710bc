// ozaki_dd.cu -- double-double GEMM (the vcp::pddcuda policy, pddblas
// semantics: vcp/pddblas.hpp:318-409) on the tensor cores.
//
// pddblas splits each dd operand into double slices, multiplies every slice
// pair with dgemm and accumulates the exact products in dd
// (pddblas_assist::split_row / split_col / ozaki_acc, vcp/pddblas.hpp:82-193).
// Here each dd entry hi + lo is scaled per row (A) / column (B) to a w-bit
// integer (w = 8 * slices, default 112 bits), the integer product A'B' is
// formed exactly from its residues modulo L <= 32 pairwise-coprime moduli
// <= 256 (one bf16 tensor-core GEMM per modulus, exact fp32 chunks, their
// residues summed in fp32), recovered by Chinese remaindering in 256-bit arithmetic, and
// rounded to a dd midpoint C = chi + clo.  A rigorous upward-rounded bound
//   |A B - C| <= K 2^(E+F-w) (1 + 2^-40) + ulp-level conversion error
// is returned alongside (Cerr).  Inputs and outputs use kv::dd layout:
// pairs {a1, a2} of doubles, column-major.
#include "common.cuh"
#include "ozaki.cuh"
#include "ozaki_common.cuh"
#include "ozaki_dd.cuh"
#include "swfp.cuh"

#include <cmath>
#include <cstring>

namespace vcpcu {

int dd_prepare(int M, int N, int K, int Mp, int Np, int Kp, int L, int w, const double* A,
               long lda, const double* B, long ldb, uint32_t* eA, uint32_t* eB,
               uint16_t* planesA, uint16_t* planesB, int* flag, cudaStream_t st);

namespace {

// The width w (lowered for very long K) and the number of moduli L: prod m_l >
// 2 |A'B'|max.
void dd_plan(int K, int* w, int* L) {
  const int Keff = K > 1 ? K : 1;
  for (;; --*w) {
    const double need = (2.0 * *w - 1.0) + std::log2((double)Keff) + 0.01;
    double bits = 0.0;
    int l = 0;
    while (l < OZ_MAX_MODULI && bits <= need) bits += std::log2((double)OZ_MODULI[l++]);
    if (bits > need) {
      *L = l;
      return;
    }
  }
}

// ---- device ---------------------------------------------------------------
// All the reassembly arithmetic runs on the integer and FP32 pipes; the few
// FP64 instructions left sit on paths taken only near the ends of the
// double range.
__device__ __forceinline__ double bits_to_d(unsigned long long b) {
  return __longlong_as_double((long long)b);
}
__device__ __forceinline__ unsigned long long d_to_bits(double x) {
  return (unsigned long long)__double_as_longlong(x);
}

// Highest set bit + 1 of a DDL-limb magnitude (0 for zero).
__device__ __forceinline__ int bitlen(const uint32_t (&mag)[DDL]) {
  int bl = 0;
#pragma unroll
  for (int t = 0; t < DDL; ++t)
    if (mag[t]) bl = 32 * t + (32 - __clz(mag[t]));
  return bl;
}

// The top 64 bits of mag (bit length bl > 0) with a sticky bit for anything
// below, and the shift: mag ~ T 2^sh.  Also the exact top bits without the
// sticky bit (Tx) and whether the remainder below them is nonzero.
__device__ __forceinline__ unsigned long long top64(const uint32_t (&mag)[DDL], int bl, int& sh,
                                                    unsigned long long& Tx) {
  sh = bl > 64 ? bl - 64 : 0;
  const int wq = sh >> 5, bq = sh & 31;
  unsigned long long w0 = 0, w1 = 0, w2 = 0;
  uint32_t below = 0;
#pragma unroll
  for (int q = 0; q < DDL; ++q) {
    const uint32_t v = mag[q];
    if (q == wq) w0 = v;
    if (q == wq + 1) w1 = v;
    if (q == wq + 2) w2 = v;
    if (q < wq) below |= v;
  }
  const unsigned long long lo64 = w0 | (w1 << 32);
  const unsigned long long t = bq ? ((lo64 >> bq) | (w2 << (64 - bq))) : lo64;
  if (bq) below |= (uint32_t)w0 & ((1u << bq) - 1u);
  Tx = t;
  return below ? (t | 1ULL) : t;
}

// RN of an integer t > 0 to 53 bits: significand Mh in [2^52, 2^53) and
// shift g with RN(t) = Mh 2^g.
__device__ __forceinline__ unsigned long long u64_rn(unsigned long long t, int& g) {
  const int b = 64 - __clzll(t);
  if (b <= 53) {
    g = b - 53;
    return t << (53 - b);
  }
  const int s = b - 53;
  unsigned long long Mh = t >> s;
  const unsigned long long rem = t & ((1ULL << s) - 1), half = 1ULL << (s - 1);
  if (rem > half || (rem == half && (Mh & 1ULL))) ++Mh;
  g = s;
  if (Mh >> 53) {
    Mh >>= 1;
    ++g;
  }
  return Mh;
}

// dd_words of any magnitude: where the remainder's leading bit lies below the
// words that the direct form looks at.  Out of line.
static __device__ __noinline__ void dd_words_general(const uint32_t* m, DdWords* w) {
  uint32_t mag[DDL], y[DDL];
#pragma unroll
  for (int t = 0; t < DDL; ++t) mag[t] = m[t];
  w->Mh = w->Ml = 0;
  w->eh = w->el = w->lbl = 0;
  w->lneg = false;
  const int bl = w->bl = bitlen(mag);
  if (bl == 0) return;
  int sh, g;
  unsigned long long Tx;
  const unsigned long long t = top64(mag, bl, sh, Tx);
  w->Mh = u64_rn(t, g);
  w->eh = g + sh;
  // remainder Y = mag - RN(t) 2^sh = D 2^sh + (mag mod 2^sh), with
  // D = Tx - RN(t) (|D| <= 2^10; the u64 difference wraps exactly)
  const long long D = (long long)(Tx - (g >= 0 ? (w->Mh << g) : (w->Mh >> -g)));
  const unsigned long long Dm = (unsigned long long)(D < 0 ? -D : D);
  const int wq = sh >> 5, bq = sh & 31;
  const unsigned long long ds = Dm << bq;  // < 2^42
  unsigned long long b = 0;
#pragma unroll
  for (int q = 0; q < DDL; ++q) {  // y = |Y|: Dm 2^sh + low (D >= 0) or - low
    uint32_t low = q < wq ? mag[q] : 0u;
    if (q == wq && bq) low = mag[q] & ((1u << bq) - 1u);
    const uint32_t dq = q == wq ? (uint32_t)ds : (q == wq + 1 ? (uint32_t)(ds >> 32) : 0u);
    if (D >= 0) {
      y[q] = dq | low;  // disjoint bit ranges
    } else {
      const unsigned long long v = (unsigned long long)dq - low - b;
      y[q] = (uint32_t)v;
      b = (v >> 63) & 1ULL;
    }
  }
  w->lneg = D < 0;
  w->lbl = bitlen(y);
  if (w->lbl == 0) return;
  int ysh, yg;
  unsigned long long yTx;
  const unsigned long long yt = top64(y, w->lbl, ysh, yTx);
  w->Ml = u64_rn(yt, yg);
  w->el = yg + ysh;
}

// RU(x 2^e) for x > 0 through the range-safe FP64 steps.
__device__ double scale_ru_slow(double x, int e) {
  while (e > 1023) {
    x = __dmul_ru(x, 0x1p1023);
    e -= 1023;
  }
  while (e < -1022) {
    x = __dmul_ru(x, 0x1p-1022);
    e += 1022;
  }
  return __dmul_ru(x, __longlong_as_double((long long)(e + 1023) << 52));
}

// Reassembly: a thread owns 4 consecutive rows (their residue bytes are one
// 32-bit word per modulus) of every gridDim.y-th column.  Bound by integer
// instructions.  Three residues meet in one 32-bit value before the eight-limb
// products (ozaki_dd.cuh; one product per residue before), and the two words
// of the result come from five leading words picked by selections: n = 2048,
// L = 28, 250 -> 113 us.  (No __restrict__: the kernel may start while the ones
// before it still write res and flag, and read-only loads are not ordered by
// dep_wait().)
__global__ void __launch_bounds__(128, 6)
dd_crt_assemble_kernel(int M, int N, int K, int Mp, int L, int w, const uint8_t* res,
                       size_t plane, const uint32_t* eA, const uint32_t* eB, double* C, long ldc,
                       double* Cerr, long lde, const int* flag,
                       const __grid_constant__ DdBasis cc) {
  dep_wait();
  const bool bad = flag[0] != 0 || flag[1] != 0;
  const int i = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
  if (i >= M) return;
  // truncation of the operands to w-bit integers: K 2^(E+F-w) (1 + 2^-40)
  const double kf = __dmul_ru((double)(K > 0 ? K : 0), 1.0 + 0x1p-40);
  const unsigned long long kfb = d_to_bits(kf);
  const int kfe = (int)(kfb >> 52);
  int E[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) E[u] = i + u < M ? dd_line_exp(eA[i + u]) : OZ_ZERO_EXP;
  for (int j = blockIdx.y; j < N; j += gridDim.y) {
    const int Fj = dd_line_exp(eB[j]);
    const size_t e0 = (size_t)j * Mp + i;
    uint32_t pk[3 * DD_GROUPS];
#pragma unroll
    for (int l = 0; l < 3 * DD_GROUPS; ++l)
      pk[l] = l < L ? *reinterpret_cast<const uint32_t*>(res + (size_t)l * plane + e0) : 0u;
#pragma unroll 1
    for (int u = 0; u < 4; ++u) {
      if (i + u >= M) break;
      const int Ei = u == 0 ? E[0] : (u == 1 ? E[1] : (u == 2 ? E[2] : E[3]));
      double hi = 0.0, lo = 0.0, err = 0.0;
      if (Ei != OZ_ZERO_EXP && Fj != OZ_ZERO_EXP) {
        uint32_t V[DD_GROUPS], mag[DDL];
        const uint32_t sel = 0x4440u + (uint32_t)u;
#pragma unroll
        for (int g = 0; g < DD_GROUPS; ++g)
          V[g] = __byte_perm(pk[3 * g], 0u, sel) * cc.a[g][0] +
                 __byte_perm(pk[3 * g + 1], 0u, sel) * cc.a[g][1] +
                 __byte_perm(pk[3 * g + 2], 0u, sel) * cc.a[g][2];
        dd_reduce(V, cc, mag);
        const bool neg = dd_abs(mag, cc);
        DdWords wd;
        if (!dd_words(mag, &wd)) dd_words_general(mag, &wd);
        // mag = X 2^z: the exponents and bit lengths of X itself below
        const int ex = Ei + Fj - 2 * w, bl = wd.bl - cc.z, lbl = wd.lbl - cc.z;
        bool range_ok = true;
        if (wd.bl > 0) {
          const int sh = bl > 64 ? bl - 64 : 0;
          if (ex + sh < -1022 || ex + sh + 64 > 1023) range_ok = false;
          const double hval =
              range_ok ? bits_to_d(((unsigned long long)(wd.eh - cc.z + ex + 1074) << 52) + wd.Mh)
                       : 0.0;
          double lval = 0.0;
          if (wd.lbl > 0) {
            const int ye = ex + (lbl > 64 ? lbl - 64 : 0);
            if (ye < -1022 || ye + 64 > 1023)
              range_ok = false;
            else
              lval = bits_to_d(((unsigned long long)(wd.el - cc.z + ex + 1074) << 52) + wd.Ml);
            if (wd.lneg) lval = sw_neg(lval);
          }
          hi = neg ? sw_neg(hval) : hval;
          lo = neg ? sw_neg(lval) : lval;
          // conversion error <= ulp(lo) (<= |lo| 2^-52) + 2^-1074:
          // RU(|lo| 2^-52 + 2^-1074) is the successor of |lo| 2^-52 when
          // that is normal
          const unsigned long long lb = d_to_bits(lval) & 0x7fffffffffffffffULL;
          if ((lb >> 52) >= 53)
            err = bits_to_d(lb - (52ULL << 52) + 1);
          else
            err = __fma_ru(fabs(lo), 0x1p-52, 0x1p-1074);
        }
        const int et = Ei + Fj - w;
        double tr = 0.0;
        if (kfb != 0) {
          if (kfe + et >= 1 && kfe + et <= 2046)
            tr = bits_to_d(kfb + ((unsigned long long)(long long)et << 52));
          else
            tr = scale_ru_slow(kf, et);
        }
        err = __dadd_ru(err, tr);
        if (!range_ok) err = INFINITY;
      }
      if (bad) hi = lo = err = __longlong_as_double(0x7ff8000000000000LL);
      double* c = C + 2 * ((size_t)(i + u) + (size_t)j * ldc);  // perhaps 8-byte aligned only
      c[0] = hi;
      c[1] = lo;
      if (Cerr) Cerr[(size_t)(i + u) + (size_t)j * lde] = err;
    }
  }
}

size_t al256d(size_t x) { return (x + 255) & ~(size_t)255; }

}  // namespace

int dd_plan_bits(int k, int slices, int* w, int* L) {
  *w = 8 * slices;
  dd_plan(k, w, L);
  return 0;
}

int ozaki_ddgemm(int m, int n, int k, const double* A, long lda, const double* B, long ldb,
                 double* C, long ldc, double* Cerr, long lde, int slices, cudaStream_t s,
                 void* static_scratch, size_t static_bytes) {
  int w = 8 * (slices > 0 ? slices : 14), L = 0;
  dd_plan(k, &w, &L);
  DdBasis cc;
  dd_basis(L, &cc);
  OzPlan plan;
  memset(&plan, 0, sizeof(plan));
  OzProblem& pb = plan.pb;
  pb.M = m;
  pb.N = n;
  pb.K = k;
  pb.Mp = (m + OZ_BM - 1) / OZ_BM * OZ_BM;
  pb.Np = (n + OZ_BN - 1) / OZ_BN * OZ_BN;
  pb.Kp = k <= 0 ? OZ_BK : (k + OZ_BK - 1) / OZ_BK * OZ_BK;
  pb.crt = 1;
  pb.w = w;
  pb.L = L;
  pb.mplanes = L;
  pb.s = slices;
  pb.sr = 2;
  OzPairList& pl = plan.crt;
  for (int l = 0; l < L; ++l) {
    pl.pa[l] = pl.pb[l] = (int8_t)l;
    pl.gstart[l] = (int16_t)l;
    pl.gt[l] = (int8_t)l;
  }
  pl.gstart[L] = (int16_t)L;
  pl.npairs = pl.ngroups = L;
  // scratch: planes A, planes B, residues, and the words that the preparation
  // accumulates into (exponents of rows and columns, flag)
  const size_t bA = al256d((size_t)L * pb.Mp * pb.Kp * 2), bB = al256d((size_t)L * pb.Np * pb.Kp * 2),
               bR = al256d((size_t)L * pb.Np * pb.Mp), bE = al256d(4 * (size_t)pb.Mp),
               bF = al256d(4 * (size_t)pb.Np), bG = 256;
  const size_t total = bA + bB + bR + bE + bF + bG;
  Scratch buf;
  uint8_t* base;
  if (static_scratch) {
    if (total > static_bytes) {
      set_error("ddgemm: needs %zu bytes of scratch, more than the %zu available", total,
                static_bytes);
      return VCPCU_ERR_INVALID_ARG;
    }
    base = (uint8_t*)static_scratch;
  } else {
    int st = buf.alloc(total, s);
    if (st) return st;
    base = (uint8_t*)buf.ptr;
  }
  OzWorkspace ws;
  memset(&ws, 0, sizeof(ws));
  ws.a_mid = (uint16_t*)base;
  ws.b_mid = (uint16_t*)(base + bA);
  ws.res = base + bA + bB;
  uint8_t* zero = base + bA + bB + bR;
  uint32_t* eA = (uint32_t*)zero;
  uint32_t* eB = (uint32_t*)(zero + bE);
  ws.flag = (int*)(zero + bE + bF);
  VCPCU_CUDA_TRY(cudaMemsetAsync(zero, 0, bE + bF + bG, s));
  int st;
  {
    PhaseTimer t(0, s);
    st = dd_prepare(m, n, k, pb.Mp, pb.Np, pb.Kp, L, w, A, lda, B, ldb, eA, eB, ws.a_mid,
                    ws.b_mid, ws.flag, s);
    if (st) return st;
  }
  {
    PhaseTimer t(3, s);
    if ((st = oz_run_gemm(plan, OZ_CRT, ws, nullptr, 0, s, true))) return st;
  }
  oz_profile_add_flops(2LL * m * n * (long long)(k > 0 ? k : 0) * L);
  {
    PhaseTimer t(4, s);
    const int gx = (m + 511) / 512;
    const int gy = n < 65535 ? n : 65535;
    VCPCU_CUDA_TRY(launch_dep(true, 1, dd_crt_assemble_kernel, dim3(gx, gy), dim3(128), 0, s, m, n,
                              k, pb.Mp, L, w, ws.res, (size_t)pb.Np * pb.Mp, eA, eB, C, ldc, Cerr,
                              lde, ws.flag, cc));
    VCPCU_LAUNCH_CHECK("dd_crt_assemble_kernel");
  }
  oz_merge_status(ws.flag, s);
  return VCPCU_OK;
}

}  // namespace vcpcu
