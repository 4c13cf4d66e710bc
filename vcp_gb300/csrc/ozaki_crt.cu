// ozaki_crt.cu -- reassembly of the CRT (Ozaki-II) form of the midpoint
// product and the final enclosure.
//
// For each entry the slice GEMM left the residues c_l = (A'B')(i,j) mod m_l
// (l < L) of the exact integer product of the w-bit operands
// A' = round(mA 2^(w-E_i)), B' = round(mB 2^(w-F_j)).  Chinese remaindering
// gives X = sum_l c_l Q_l mod M (Q_l = (M/m_l) ((M/m_l)^-1 mod m_l)), taken
// in (-M/4, M/4); since prod m_l > 4 |A'B'|, X = (A'B')(i,j) exactly.  Then
//   mA mB = 2^(E+F-2w) X + ΔA mB + Â ΔB,   |ΔA| <= 2^(E-w-1), |ΔB| <= 2^(F-w-1),
//   |ΔA mB| <= 2^(E-w-1) beta_j,   |Â ΔB| <= 2^(E+F-2w-1) sum_k |A'(i,k)|,
// and the enclosure is [RD(2^(E+F-2w) X) - e, RU(2^(E+F-2w) X) + e] with
// e = RU(RU(trunc) + T(i,j)), T the upper bound of the radius term.
#include "common.cuh"
#include "ozaki.cuh"
#include "ozaki_common.cuh"
#include "ozaki_crt.cuh"
#include "ozaki_prep.cuh"
#include "swfp.cuh"

namespace vcpcu {

namespace {

// Sticky per-device status of the Ozaki form: bit 0 non-finite input, bit 1
// a bounded device wait timed out.  The reassembly kernels merge their
// product's status words; read and cleared by oz_take_status.
__device__ int g_oz_status;

__global__ void oz_status_merge(const int* flag) {
  int v = (flag[0] ? 1 : 0) | (flag[1] ? 2 : 0);
  if (v) atomicOr(&g_oz_status, v);
}

__device__ __forceinline__ double scale_dir2(double x, int e, bool up) {
  while (e > 1023) {
    x = up ? __dmul_ru(x, 0x1p1023) : __dmul_rd(x, 0x1p1023);
    e -= 1023;
  }
  while (e < -1022) {
    x = up ? __dmul_ru(x, 0x1p-1022) : __dmul_rd(x, 0x1p-1022);
    e += 1022;
  }
  const double p = __longlong_as_double((long long)(e + 1023) << 52);
  return up ? __dmul_ru(x, p) : __dmul_rd(x, p);
}

// x * 2^e rounded up (up) or down: the exponent field is moved on the
// integer pipe when x and the result are normal (then the product is exact
// and equals scale_dir2's); otherwise scale_dir2.
__device__ __forceinline__ double scale_pow2(double x, int e, bool up) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int be = (int)((b >> 52) & 0x7ff);
  if (be != 0 && be != 0x7ff && be + e >= 1 && be + e <= 2046)
    return __longlong_as_double((long long)(b + ((unsigned long long)(long long)e << 52)));
  if (oz_zero(x)) return x;
  return scale_dir2(x, e, up);
}

// RD and RU of t * 2^e for t > 0 (64 bits) built on the integer pipe: the
// top 53 bits of t are the truncated significand, any lower bit set makes
// RU one unit larger (a carry into the exponent field is the correct
// rounding).  Equal to scale_dir2(__ull2double_rd/ru(t), e) -- which runs
// when the result leaves the normal range.
__device__ __forceinline__ void u64_to_dir(unsigned long long t, int e, double& dn, double& upv) {
  const int lz = __clzll(t);
  const unsigned long long tn = t << lz;
  const int be = 1023 + 63 - lz + e;
  if (be >= 1 && be <= 2046) {
    const unsigned long long d =
        ((unsigned long long)be << 52) + ((tn >> 11) & ((1ULL << 52) - 1));
    dn = __longlong_as_double((long long)d);
    upv = __longlong_as_double((long long)(d + ((tn & 0x7ffULL) ? 1ULL : 0ULL)));
    return;
  }
  dn = scale_dir2(__ull2double_rd(t), e, false);
  upv = scale_dir2(__ull2double_ru(t), e, true);
}

// Directed conversion of (-1)^neg * mag * 2^e (mag: 4 limbs) to double.
// Limbs are picked by unrolled selects (no dynamically indexed array, which
// would live in local memory).
__device__ __forceinline__ void big_to_dir(const uint32_t (&mag)[4], int neg, int e, double& lo,
                                           double& up) {
  int bl = 0;  // bit length, 0..128
#pragma unroll
  for (int t = 0; t < 4; ++t)
    if (mag[t]) bl = 32 * t + (32 - __clz(mag[t]));
  if (bl == 0) {
    lo = up = 0.0;
    return;
  }
  const int sh = bl > 64 ? bl - 64 : 0;
  const int wq = sh >> 5, bq = sh & 31;
  unsigned long long w0 = 0, w1 = 0, w2 = 0;
  uint32_t below = 0;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    if (q == wq) w0 = mag[q];
    if (q == wq + 1) w1 = mag[q];
    if (q == wq + 2) w2 = mag[q];
    if (q < wq) below |= mag[q];
  }
  const unsigned long long lo64 = w0 | (w1 << 32);
  unsigned long long t = bq ? ((lo64 >> bq) | (w2 << (64 - bq))) : lo64;
  if (bq) below |= (uint32_t)w0 & ((1u << bq) - 1u);
  if (below) t |= 1ULL;
  double a_dn, a_up;
  u64_to_dir(t, e + sh, a_dn, a_up);
  if (!neg) {
    lo = a_dn;
    up = a_up;
  } else {
    lo = sw_neg(a_up);
    up = sw_neg(a_dn);
  }
}

// The radius sums of both products for 4 consecutive rows (e0 = j Mp + i0):
// one fp32 fold per product (slot 0 and slot nslot = 1), the slice GEMM
// epilogue's upward sum of every chunk weighted by its digit pair -- an
// upper bound of the exact integer W of the product.
__device__ __forceinline__ void rad_folds(const int32_t* P, size_t plane,
                                          size_t e0, const OzRadConst& rc, float (&S1)[4],
                                          float (&S2)[4]) {
  const float4 z = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  const float4 v1 = rc.run1 ? *reinterpret_cast<const float4*>(P + e0) : z;
  const float4 v2 =
      rc.run2 ? *reinterpret_cast<const float4*>(P + (size_t)rc.nslot * plane + e0) : z;
  S1[0] = v1.x;
  S1[1] = v1.y;
  S1[2] = v1.z;
  S1[3] = v1.w;
  S2[0] = v2.x;
  S2[1] = v2.y;
  S2[2] = v2.z;
  S2[3] = v2.w;
}

// RU(sqrt(RU(Q))) scale for a sum Q of squared low radius digits (0 for
// Q = 0; scale a power of two, so the product is exact).
__device__ __forceinline__ float lowpair_root(unsigned long long Q, float scale) {
  return Q ? __fmul_rn(__fsqrt_ru(__ull2float_ru(Q)), scale) : 0.0f;
}

// RU(RU(S + R) + b) 2^ex, 0 for a zero row or column.  S + R >= the exact
// W + R of the pairs that ran; b >= the left-out low x low pair (in the units
// of W: sum_k lo_A lo_B 2^-8 <= sqrt(sum lo_A^2) sqrt(sum lo_B^2) 2^-8,
// Cauchy-Schwarz), 0 when every pair ran.  The sum is >= 0 (the digits of
// both radius factors are upward, so every product of their reconstructions
// is non-negative) and is 0 or at least 2^-16: a normal float, whose double
// is built on the integer pipe.
__device__ __forceinline__ double rad_term(float S, bool zero, int ex, int R, float b) {
  if (zero) return 0.0;
  float s = R ? __fadd_ru(S, (float)R) : S;
  s = __fadd_ru(s, b);
  if (!(s > 0.0f)) return 0.0;
  const unsigned u = __float_as_uint(s);
  const double d = __longlong_as_double((long long)(((unsigned long long)((u >> 23) + 896) << 52) |
                                                    ((unsigned long long)(u & 0x7fffffu) << 29)));
  return scale_pow2(d, ex, true);
}

// T = RU(RU((|mA| + rA) rB) + RU(rA |mB|)) at (i, j), the products that ran;
// l1, l2 the bounds of their left-out pairs.
__device__ __forceinline__ double rad_T(float S1, float S2, int Ep, int Er, int Fm, int Fr,
                                        const OzRadConst& rc, float l1, float l2) {
  const double b1 = rc.run1 ? rad_term(S1, Ep == OZ_ZERO_EXP || Fr == OZ_ZERO_EXP,
                                       Ep + Fr - 8 * rc.t_ref, rc.R, l1)
                            : 0.0;
  if (!rc.run2) return b1;
  const double b2 =
      rad_term(S2, Er == OZ_ZERO_EXP || Fm == OZ_ZERO_EXP, Er + Fm - 8 * rc.t_ref, rc.R, l2);
  return rc.run1 ? __dadd_ru(b1, b2) : b2;
}

// Slice form: T (ld Mp) from the folds, before the midpoint product.
__global__ void __launch_bounds__(256)
oz_radius_T_kernel(int M, int N, int Mp, size_t plane, const int32_t* __restrict__ P,
                   const int* __restrict__ E3, const int* __restrict__ F2,
                   double* __restrict__ T, const __grid_constant__ OzRadConst rc) {
  const int Mq = (M + 3) >> 2;
  const long total = (long)Mq * N;
  for (long idx = (long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (long)gridDim.x * blockDim.x) {
    const int i0 = 4 * (int)(idx % Mq), j = (int)(idx / Mq);
    const size_t e0 = (size_t)j * Mp + i0;
    float W1[4], W2[4];
    rad_folds(P, plane, e0, rc, W1, W2);
    const int Fm = F2[2 * j], Fr = F2[2 * j + 1];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = i0 + u;
      if (i >= M) break;
      T[e0 + u] = rad_T(W1[u], W2[u], E3[3 * i + 1], E3[3 * i + 2], Fm, Fr, rc, 0.0f, 0.0f);
    }
  }
}

// ---------------------------------------------------------------- reassembly
//
// A block of 256 threads takes a tile of up to 128 rows and CB columns of one
// product; a thread owns 4 consecutive rows (their residue bytes are one
// 32-bit word per modulus, their folds one 16-byte load per product) of every
// CW-th column.  The per-row and per-column data -- exponents, sA = RU(sum_k
// |A'(i,k)|), beta_j = RU((sum_k |B'(k,j)| + ceil(K/2)) 2^(F - w)), the roots
// of the low radius digits' squares -- are formed once per block in shared
// memory.
//
// Bound: five FP64 additions per entry (64 cycles of a sub-partition's FP64
// unit per warp instruction) beside the integer arithmetic of the residues;
// DRAM moves 40 bytes per entry.  Values that every entry of a tile shares
// are scaled once (t1 and t2 below are an exponent add each), three residues
// meet in one 32-bit value before the multi-limb products (ozaki_crt.cuh),
// and the double results are put together from words.  Measured against one
// 128-bit product per residue, 8 columns a thread and a branch per entry:
// n = 8192 1.49 -> 0.76 ms, n = 512 48 -> 10 us (64 blocks before), 17 chunks
// of a 256-problem batch 1.30 -> 0.54 ms summed.  80 registers (three blocks
// per SM, a few words spilled) 752 us at n = 8192, 128 registers 815 us.

constexpr int ASM_ROWS = 128, ASM_COLS = 64, ASM_NT = 256;
// The direct path below adds to exponent fields without looking: every value of
// an entry has to be a normal double (or 0).  With |X| in [1, 2^(2w + 18)], sA in
// [2^(w - 2), 2^(w + 20)], beta in [2^(F - 2), 2^(F + 20)] (k <= 2^20) and folds in
// [2^-16, 2^52] that holds where the exponents of a factor pair sum up to
//   E + F in [2 w - 1020, ASM_HI],  Ep + Fr and Er + F in [ASM_RAD_LO, ASM_HI]
// and F, for beta itself, lies in [ASM_COL_LO, ASM_COL_HI].  A zero radius row or
// column has zero folds: any exponent gives its 0.  Entries of a zero row or column
// take the general path, which has little to do there.  (Limits of +-400 on each
// exponent, and the general path an entry at a time after the direct one: 3000 x
// 3000, k = 64, a zero row in four 605 us, now 351; factors over 2^450 690, now 267;
// rows and columns over 2^+-600 866, now 623.)
constexpr int ASM_HI = 990, ASM_RAD_LO = -970, ASM_COL_LO = -1020, ASM_COL_HI = 1003;

// (rows as one array per quantity: a thread reads its 4 as one vector, a
// warp's vectors lie side by side, free of bank conflicts)
struct alignas(16) AsmRows {
  double sA[ASM_ROWS];                       // RU(sum_k |A'(i,k)|)
  int E[ASM_ROWS], Ep[ASM_ROWS], Er[ASM_ROWS];  // exponents of mA, |mA| + rA, rA
  float qp[ASM_ROWS], qr[ASM_ROWS];          // 2^-8 roots of the low digits' squares of P, rA
};
struct AsmCol {
  double beta;
  int Fm, Fr;
  float q1, q2;     // roots of the low digits' squares of rB, |mB|
};
// What the entries of a product read and write.  res and P point at row /
// column 0 of the product (plane = Np Mp of its layout).
struct AsmArgs {
  int M, Mp, L, w;
  const uint8_t* res;
  size_t plane;
  const int32_t* P;
  double* C;
  double* Cup;  // not null: plain matrices, lower ends to C, upper ends to Cup
  long ldc;
  bool nonfinite, al16;
};
struct AsmTile {
  AsmRows row;
  // of each quad of rows: the column exponents that its direct path takes, Fm in
  // [x, y] and Fr in [z, w]; its zero rows (bits)
  int4 takes[ASM_ROWS / 4];
  int zero[ASM_ROWS / 4];
  AsmCol col[ASM_COLS];
  // of each warp's 32 columns: least and largest Fm, Fr of those that have one;
  // a zero column
  int minF[2], maxF[2], minR[2], maxR[2], zeroF[2];
  AsmArgs args;  // for the general path, which takes pointers
};

// RU of asum_hi 2^32 + asum_lo (exact below 2^96).
__device__ __forceinline__ double asum_ru(unsigned long long ah, unsigned long long al) {
  const unsigned __int128 sx = ((unsigned __int128)ah << 32) + al;
  if (!sx) return 0.0;
  double dn, up;
  const unsigned long long hi64 = (unsigned long long)(sx >> 64);
  if (hi64 == 0) {
    u64_to_dir((unsigned long long)sx, 0, dn, up);
  } else {
    const int sh = 64 - __clzll(hi64);
    unsigned long long t = (unsigned long long)(sx >> sh);
    if ((unsigned long long)sx & ((1ULL << sh) - 1)) t |= 1ULL;
    u64_to_dir(t, sh, dn, up);
  }
  return up;
}

// The rows [i0, i0 + nr) and columns [j0, j0 + nc) of the tile.  eA, asum, eB
// and bsum point at row / column 0 of the product.
__device__ __forceinline__ void asm_tile_setup(AsmTile& t, int i0, int nr, int j0, int nc, int K,
                                               int w, int lowb, const uint32_t* eA,
                                               const unsigned long long* asum, const uint32_t* eB,
                                               const unsigned long long* bsum) {
  const int x = threadIdx.x;
  if (x < ASM_ROWS) {
    double sA = 0.0;
    int E = OZ_ZERO_EXP, Ep = OZ_ZERO_EXP, Er = OZ_ZERO_EXP;
    float qp = 0.0f, qr = 0.0f;
    if (x < nr) {
      const int i = i0 + x;
      E = exp_dec(eA[3 * i]);
      Ep = exp_dec(eA[3 * i + 1]);
      Er = exp_dec(eA[3 * i + 2]);
      sA = asum_ru(asum[4 * i], asum[4 * i + 1]);
      if (lowb) {
        qp = lowpair_root(asum[4 * i + 2], 0x1p-8f);
        qr = lowpair_root(asum[4 * i + 3], 0x1p-8f);
      }
    }
    t.row.sA[x] = sA;
    t.row.E[x] = E;
    t.row.Ep[x] = Ep;
    t.row.Er[x] = Er;
    t.row.qp[x] = qp;
    t.row.qr[x] = qr;
    const unsigned all = 0xffffffffu;
    const bool z = E == OZ_ZERO_EXP;
    int loF = z ? ASM_COL_LO : max(ASM_COL_LO, 2 * w - 1020 - E),
        hiF = z ? ASM_COL_HI : min(ASM_COL_HI, ASM_HI - E), loR = OZ_ZERO_EXP, hiR = -OZ_ZERO_EXP;
    if (Er != OZ_ZERO_EXP) {
      loF = max(loF, ASM_RAD_LO - Er);
      hiF = min(hiF, ASM_HI - Er);
    }
    if (Ep != OZ_ZERO_EXP) {
      loR = ASM_RAD_LO - Ep;
      hiR = ASM_HI - Ep;
    }
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
      loF = max(loF, __shfl_xor_sync(all, loF, o));
      hiF = min(hiF, __shfl_xor_sync(all, hiF, o));
      loR = max(loR, __shfl_xor_sync(all, loR, o));
      hiR = min(hiR, __shfl_xor_sync(all, hiR, o));
    }
    const unsigned zb = __ballot_sync(all, z && x < nr);
    if ((x & 3) == 0) {
      t.takes[x >> 2] = make_int4(loF, hiF, loR, hiR);
      t.zero[x >> 2] = (zb >> (x & 28)) & 15;
    }
  } else if (x < ASM_ROWS + ASM_COLS) {  // two warps
    const int jc = x - ASM_ROWS, j = j0 + jc;
    const bool in = jc < nc;
    AsmCol c;
    c.Fm = in ? exp_dec(eB[2 * j]) : OZ_ZERO_EXP;
    c.Fr = in ? exp_dec(eB[2 * j + 1]) : OZ_ZERO_EXP;
    c.beta = 0.0;
    c.q1 = c.q2 = 0.0f;
    const bool zF = c.Fm == OZ_ZERO_EXP, zR = c.Fr == OZ_ZERO_EXP;
    if (!zF) {
      const double v = __fma_ru((double)bsum[4 * j], 0x1p32,
                                (double)(bsum[4 * j + 1] + (unsigned long long)(K + 1) / 2));
      c.beta = scale_dir2(v, c.Fm - w, true);
    }
    if (lowb && in) {
      c.q1 = lowpair_root(bsum[4 * j + 2], 1.0f);
      c.q2 = lowpair_root(bsum[4 * j + 3], 1.0f);
    }
    if (in) t.col[jc] = c;
    const unsigned all = 0xffffffffu;
    const int v0 = __reduce_min_sync(all, zF ? 30000 : c.Fm), v1 = __reduce_max_sync(all, c.Fm),
              v2 = __reduce_min_sync(all, zR ? 30000 : c.Fr), v3 = __reduce_max_sync(all, c.Fr),
              v4 = __any_sync(all, in && zF);
    if ((x & 31) == 0) {
      const int h = jc >> 5;
      t.minF[h] = v0;
      t.maxF[h] = v1;
      t.minR[h] = v2;
      t.maxR[h] = v3;
      t.zeroF[h] = v4;
    }
  }
  __syncthreads();
}

__device__ __forceinline__ void asm_store(const AsmArgs& a, size_t c, double2 r) {
  if (a.nonfinite) r.x = r.y = __longlong_as_double(0x7ff8000000000000LL);
  if (a.Cup) {
    a.C[c] = r.x;
    a.Cup[c] = r.y;
  } else if (a.al16) {
    reinterpret_cast<double2*>(a.C)[c] = r;
  } else {  // C may be only 8-byte aligned
    a.C[2 * c] = r.x;
    a.C[2 * c + 1] = r.y;
  }
}

// Entries of a column (rows i0 + q4 + u for the bits u of `rows`, column j, *col)
// that the direct path leaves out: the same operations with every range looked at.  Out
// of line, so that neither its registers nor its FP64 instructions weigh on the
// direct path; everything by pointers into shared memory and the parameters.
static __device__ __noinline__ void asm_quad_general(const AsmTile* t, int i0, int q4, int j,
                                                     int rows, const AsmCol* col,
                                                     const CrtBasis* cc, const OzRadConst* rc) {
  const AsmArgs& a = t->args;
  const int w = a.w, F = col->Fm;
  const size_t e0 = (size_t)j * a.Mp + i0 + q4;
  uint32_t pk[3 * OZ_CRT_GROUPS];
#pragma unroll
  for (int l = 0; l < 3 * OZ_CRT_GROUPS; ++l)
    pk[l] = l < a.L ? *reinterpret_cast<const uint32_t*>(a.res + (size_t)l * a.plane + e0) : 0u;
#pragma unroll 1
  for (int u = 0; u < 4; ++u) {
    if (!((rows >> u) & 1) || i0 + q4 + u >= a.M) continue;
    const int x = q4 + u, E = t->row.E[x];
    double lo = 0.0, up = 0.0, tr = 0.0;
    if (E != OZ_ZERO_EXP && F != OZ_ZERO_EXP) {
      uint32_t V[OZ_CRT_GROUPS], mag[4];
      const uint32_t sel = 0x4440u + (uint32_t)u;
#pragma unroll
      for (int g = 0; g < OZ_CRT_GROUPS; ++g)
        V[g] = __byte_perm(pk[3 * g], 0u, sel) * cc->a[g][0] +
               __byte_perm(pk[3 * g + 1], 0u, sel) * cc->a[g][1] +
               __byte_perm(pk[3 * g + 2], 0u, sel) * cc->a[g][2];
      crt_reduce(V, *cc, mag);
      const int neg = crt_abs(mag);
      big_to_dir(mag, neg, E + F - 2 * w - cc->z, lo, up);
      const double t1 = scale_pow2(col->beta, E - w - 1, true);
      const double t2 = scale_pow2(t->row.sA[x], E + F - 2 * w - 1, true);
      tr = __dadd_ru(t1, t2);
    }
    const float S1 = rc->run1 ? __int_as_float(a.P[e0 + u]) : 0.0f,
                S2 = rc->run2 ? __int_as_float(a.P[(size_t)rc->nslot * a.plane + e0 + u]) : 0.0f;
    const double T =
        rad_T(S1, S2, t->row.Ep[x], t->row.Er[x], F, col->Fr, *rc,
              __fmul_ru(t->row.qp[x], col->q1), __fmul_ru(t->row.qr[x], col->q2));
    const double err = __dadd_ru(tr, T);
    asm_store(a, (size_t)(i0 + x) + (size_t)j * a.ldc,
              make_double2(__dsub_rd(lo, err), __dadd_ru(up, err)));
  }
}

// RU(s) 2^x of a fold s >= 0 as a double (0 for 0): e20 = (x + 896) << 20.
__device__ __forceinline__ double asm_fold(float s, int e20) {
  const unsigned u = __float_as_uint(s);
  const bool pos = s > 0.0f;
  const int hi = (int)(u >> 3) + e20;
  return __hiloint2double(pos ? hi : 0, pos ? (int)(u << 29) : 0);
}

// All entries of a thread: rows i0 + 4 q .. + 3 (q = thread % Rq) of the
// columns j0 + thread / Rq + CW c of its block.  The 4 entries of a column run
// the direct path together without a branch between them (their FP64
// additions overlap).
// SPECIAL: some row or column of the thread's may leave the direct path.  A copy
// of its own and out of line (asm_entries_special), so that the loop of the others
// holds neither the tests nor a call: n = 4096, k = 64 196 us, 211 with the tests in
// one loop and 213 with the general path's calls at its end; the 256-problem batch
// 1687, 1765 and 1707.  (Inlined beside the other, its registers cost the loop 323.)
template <bool LOWB, bool SPECIAL>
__device__ __forceinline__ void asm_entries(const AsmTile& t, const AsmArgs& a, int i0,
                                            int q4, int slot, int CW, int j0, int nc,
                                            const CrtBasis& cc, const OzRadConst& rc) {
  const int i = i0 + q4;
  // per-row words of the direct path (those of a zero row or radius go unused)
  int E20[4], P20[4], R20[4], sAh[4], sAl[4];
  float qp[4], qr[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int E = t.row.E[q4 + u];
    E20[u] = E << 20;
    P20[u] = (t.row.Ep[q4 + u] - 8 * rc.t_ref + 896) << 20;
    R20[u] = (t.row.Er[q4 + u] - 8 * rc.t_ref + 896) << 20;
    const long long sb = __double_as_longlong(t.row.sA[q4 + u]);
    sAh[u] = (int)(sb >> 32) + ((E - 2 * a.w - 1) << 20);  // sA 2^(E - 2 w - 1)
    sAl[u] = (int)sb;
    qp[u] = LOWB ? t.row.qp[q4 + u] : 0.0f;
    qr[u] = LOWB ? t.row.qr[q4 + u] : 0.0f;
  }
  const int zero = SPECIAL ? t.zero[q4 >> 2] : 0;
  const int cX = (1149 - 2 * a.w - cc.z) << 20;
  for (int c = slot; c < nc; c += CW) {
    const int j = j0 + c;
    const AsmCol& col = t.col[c];
    const int Fm = col.Fm, Fr = col.Fr;
    if (SPECIAL) {
      const int4 f = t.takes[q4 >> 2];
      const bool direct = rc.R == 0 && Fm >= f.x && Fm <= f.y &&  // (a zero column's is below)
                          (Fr == OZ_ZERO_EXP || (Fr >= f.z && Fr <= f.w));
      const int redo = direct ? zero : 15;
      if (redo) asm_quad_general(&t, i0, q4, j, redo, &col, &cc, &rc);
      if (redo == 15) continue;
    }
    const size_t e0 = (size_t)j * a.Mp + i;
    uint32_t pk[3 * OZ_CRT_GROUPS];
#pragma unroll
    for (int l = 0; l < 3 * OZ_CRT_GROUPS; ++l)
      pk[l] = l < a.L ? *reinterpret_cast<const uint32_t*>(a.res + (size_t)l * a.plane + e0) : 0u;
    float S1[4], S2[4];
    rad_folds(a.P, a.plane, e0, rc, S1, S2);
    // group values of the 4 rows
    uint32_t V[4][OZ_CRT_GROUPS];
#pragma unroll
    for (int g = 0; g < OZ_CRT_GROUPS; ++g) {
      const uint32_t a0 = cc.a[g][0], a1 = cc.a[g][1], a2 = cc.a[g][2];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        V[u][g] = ((pk[3 * g] >> (8 * u)) & 255u) * a0 + ((pk[3 * g + 1] >> (8 * u)) & 255u) * a1 +
                  ((pk[3 * g + 2] >> (8 * u)) & 255u) * a2;
    }
    const int F20 = Fm << 20, Fr20 = Fr << 20;
    const long long bb = __double_as_longlong(col.beta);
    const int bh = (int)(bb >> 32) - ((a.w + 1) << 20), bl = (int)bb;  // beta 2^(-w - 1)
    double2 r[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      uint32_t mag[4], dn[2], up[2];
      crt_reduce(V[u], cc, mag);
      const int neg = crt_abs(mag);
      crt_to_dir(mag, E20[u] + F20 + cX, dn, up);
      // [lo, hi] = neg ? [-up, -dn] : [dn, up]
      const uint32_t sg = (uint32_t)neg << 31;
      const double lo = __hiloint2double((int)((neg ? up[0] : dn[0]) | sg),
                                         (int)(neg ? up[1] : dn[1])),
                   hi = __hiloint2double((int)((neg ? dn[0] : up[0]) | sg),
                                         (int)(neg ? dn[1] : up[1]));
      const double t1 = __hiloint2double(bh + E20[u], bl),
                   t2 = __hiloint2double(sAh[u] + F20, sAl[u]);
      double err = __dadd_ru(t1, t2);
      float s1 = S1[u], s2 = S2[u];
      if (LOWB) {
        s1 = __fadd_ru(s1, __fmul_ru(qp[u], col.q1));
        s2 = __fadd_ru(s2, __fmul_ru(qr[u], col.q2));
      }
      const double b1 = asm_fold(s1, P20[u] + Fr20), b2 = asm_fold(s2, R20[u] + F20);
      // (a product that did not run adds nothing)
      if (rc.run1 && rc.run2)
        err = __dadd_ru(err, __dadd_ru(b1, b2));
      else if (rc.run1)
        err = __dadd_ru(err, b1);
      else if (rc.run2)
        err = __dadd_ru(err, b2);
      r[u] = make_double2(__dsub_rd(lo, err), __dadd_ru(hi, err));
    }
    const size_t c0 = (size_t)i + (size_t)j * a.ldc;
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (i + u < a.M && !((zero >> u) & 1)) asm_store(a, c0 + u, r[u]);
  }
}

template <bool LOWB>
static __device__ __noinline__ void asm_entries_special(const AsmTile* t, int i0, int q4, int slot,
                                                        int CW, int j0, int nc, const CrtBasis* cc,
                                                        const OzRadConst* rc) {
  asm_entries<LOWB, true>(*t, t->args, i0, q4, slot, CW, j0, nc, *cc, *rc);
}
template <bool LOWB>
__device__ __forceinline__ void asm_tile(const AsmTile& t, const AsmArgs& a, int i0, int nr,
                                         int j0, int nc, const CrtBasis& cc,
                                         const OzRadConst& rc) {
  const int Rq = (nr + 3) >> 2, CW = ASM_NT / Rq;
  const int slot = (int)threadIdx.x / Rq, q4 = 4 * ((int)threadIdx.x - slot * Rq);
  if (slot >= CW) return;
  const int4 in = t.takes[q4 >> 2];
  if (t.zero[q4 >> 2] || t.zeroF[0] || t.zeroF[1] || rc.R != 0 ||
      min(t.minF[0], t.minF[1]) < in.x || max(t.maxF[0], t.maxF[1]) > in.y ||
      min(t.minR[0], t.minR[1]) < in.z || max(t.maxR[0], t.maxR[1]) > in.w)
    asm_entries_special<LOWB>(&t, i0, q4, slot, CW, j0, nc, &cc, &rc);
  else
    asm_entries<LOWB, false>(t, a, i0, q4, slot, CW, j0, nc, cc, rc);
}

// One product: blocks over the column ranges of CB columns, then over the
// 128-row tiles (one dimension: no limit on either).  Block 0 merges the
// status words.  (No __restrict__, here and in what it calls: the kernel may
// start while the ones before it still write res, P and flag, and read-only
// loads are not ordered by dep_wait().)
template <bool LOWB>
__global__ void __launch_bounds__(ASM_NT, 3)
oz_crt_assemble_kernel(int M, int N, int K, int Mp, int L, int w, int CB, const uint8_t* res,
                       size_t plane, const uint32_t* eA, const uint32_t* eB,
                       const unsigned long long* asum, const unsigned long long* bsum,
                       const int32_t* P, double* C, double* Cup, long ldc, const int* flag,
                       int merge,
                       const __grid_constant__ CrtBasis cc, const __grid_constant__ OzRadConst rc) {
  __shared__ AsmTile t;
  dep_wait();
  const int f0 = flag[0], f1 = flag[1];
  if (merge && (f0 | f1) && blockIdx.x == 0 && threadIdx.x == 0)
    atomicOr(&g_oz_status, (f0 ? 1 : 0) | (f1 ? 2 : 0));
  const int ncb = (N + CB - 1) / CB;
  const int i0 = (int)(blockIdx.x / ncb) * ASM_ROWS, nr = min(ASM_ROWS, M - i0);
  const int j0 = (int)(blockIdx.x % ncb) * CB, nc = min(CB, N - j0);
  const AsmArgs a{M, Mp, L, w, res, plane, P, C, Cup, ldc, f0 != 0 || f1 != 0,
                  (((uintptr_t)C) & 15) == 0};
  if (threadIdx.x == ASM_NT - 1) t.args = a;  // (no row or column of its own)
  asm_tile_setup(t, i0, nr, j0, nc, K, w, LOWB, eA, asum, eB, bsum);
  asm_tile<LOWB>(t, a, i0, nr, j0, nc, cc, rc);
}

// Grouped reassembly.  The problems of a bucket share one CRT plan (the
// bucket is keyed by modulus count, operand width, radius pairs and scaling), so
// the basis comes in the launch parameters as for one product.  A block takes a
// tile of up to 128 rows and OZ_GASM_COLS columns of one problem, found with
// one load (prob_asm); it stamps the problem's end and merges its status
// words into the sticky status.  A device-wait timeout of the slice
// GEMM (flag[1] of problem 0) poisons every output of the bucket.
template <bool LOWB>
__global__ void __launch_bounds__(ASM_NT, 3)
oz_crt_assemble_g(const __grid_constant__ OzGBucket b, const __grid_constant__ CrtBasis cc,
                  const __grid_constant__ OzRadConst rc) {
  __shared__ AsmTile t;
  const int p = b.prob_asm[blockIdx.x];
  const OzGProb& q = b.probs[p];
  const int m = q.m, n = q.n;
  const int tm = (m + ASM_ROWS - 1) / ASM_ROWS, local = blockIdx.x - b.blk_asm[p];
  const int i0 = (local % tm) * ASM_ROWS, nr = min(ASM_ROWS, m - i0);
  const int j0 = (local / tm) * OZ_GASM_COLS, nc = min(OZ_GASM_COLS, n - j0);
  const int f0 = b.flag[4 * p], f1 = b.flag[4 * p + 1];
  const AsmArgs a{m, q.Mp, q.L, q.w, b.res + q.res_off, (size_t)q.Np * q.Mp, b.P + q.P_off, q.C,
                  nullptr, q.ldc, f0 != 0 || b.flag[1] != 0, (((uintptr_t)q.C) & 15) == 0};
  if (threadIdx.x == ASM_NT - 1) t.args = a;  // (no row or column of its own)
  asm_tile_setup(t, i0, nr, j0, nc, q.k, q.w, LOWB, b.eA + 3 * (size_t)q.rowoff,
                 b.asum + 4 * (size_t)q.rowoff, b.eB + 2 * (size_t)q.coloff,
                 b.bsum + 4 * (size_t)q.coloff);
  asm_tile<LOWB>(t, a, i0, nr, j0, nc, cc, rc);
  if (threadIdx.x == 0 && (f0 | f1)) atomicOr(&g_oz_status, (f0 ? 1 : 0) | (f1 ? 2 : 0));
  if (b.t_last) {
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned long long now;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
      atomicMax(&b.t_last[q.orig], now);
    }
  }
}

static_assert(OZ_GASM_COLS <= ASM_COLS, "column data of a grouped tile");
static_assert(ASM_ROWS + ASM_COLS < ASM_NT && ASM_COLS == 64, "one thread a row or column");

}  // namespace

void oz_merge_status(const int* flag, cudaStream_t s) {
  oz_status_merge<<<1, 1, 0, s>>>(flag);
  count_launch();
}

int oz_take_status(cudaStream_t s, int* status) {
  int zero = 0;
  VCPCU_CUDA_TRY(cudaMemcpyFromSymbolAsync(status, g_oz_status, sizeof(int), 0,
                                           cudaMemcpyDeviceToHost, s));
  VCPCU_CUDA_TRY(cudaStreamSynchronize(s));
  VCPCU_CUDA_TRY(cudaMemcpyToSymbolAsync(g_oz_status, &zero, sizeof(int), 0,
                                         cudaMemcpyHostToDevice, s));
  VCPCU_CUDA_TRY(cudaStreamSynchronize(s));
  return VCPCU_OK;
}

int oz_crt_assemble(const OzPlan& plan, const OzWorkspace& ws, double* C, long ldc,
                    cudaStream_t st, bool merge_status, double* Cup, bool chained) {
  const OzProblem& pb = plan.pb;
  if (pb.M <= 0 || pb.N <= 0) return VCPCU_OK;
  const int tm = (pb.M + ASM_ROWS - 1) / ASM_ROWS;
  // columns per block: as many as leave four blocks for each of the 152 SMs
  // (a block's row and column data are formed once), 64 at most
  int CB = ASM_COLS;
  while (CB > 8 && (long)tm * ((pb.N + CB - 1) / CB) < 608) CB >>= 1;
  const unsigned grid = (unsigned)tm * (unsigned)((pb.N + CB - 1) / CB);
  const OzRadConst rc = oz_rad_const(plan);
  const auto kernel = rc.lowb ? oz_crt_assemble_kernel<true> : oz_crt_assemble_kernel<false>;
  VCPCU_CUDA_TRY(launch_dep(chained, 1, kernel, dim3(grid), dim3(ASM_NT), 0, st, pb.M, pb.N, pb.K,
                            pb.Mp, pb.L, pb.w, CB, ws.res, (size_t)pb.Np * pb.Mp, ws.eA, ws.eB,
                            ws.asum, ws.bsum, ws.P, C, Cup, ldc, ws.flag, merge_status ? 1 : 0,
                            plan.basis, rc));
  VCPCU_LAUNCH_CHECK("oz_crt_assemble_kernel");
  return VCPCU_OK;
}

int oz_gassemble(const OzGBucket& b, const OzPlan& shape, const OzRadConst& rc, int nblk,
                 cudaStream_t st) {
  if (nblk <= 0) return VCPCU_OK;
  if (rc.lowb)
    oz_crt_assemble_g<true><<<nblk, ASM_NT, 0, st>>>(b, shape.basis, rc);
  else
    oz_crt_assemble_g<false><<<nblk, ASM_NT, 0, st>>>(b, shape.basis, rc);
  VCPCU_LAUNCH_CHECK("oz_crt_assemble_g");
  return VCPCU_OK;
}

int oz_radius_T(const OzPlan& plan, const OzWorkspace& ws, cudaStream_t st) {
  const OzProblem& pb = plan.pb;
  const long total = (long)((pb.M + 3) / 4) * pb.N;
  long blocks = (total + 255) / 256;
  if (blocks > 152L * 64) blocks = 152L * 64;
  if (blocks < 1) blocks = 1;
  oz_radius_T_kernel<<<(int)blocks, 256, 0, st>>>(pb.M, pb.N, pb.Mp, (size_t)pb.Np * pb.Mp, ws.P,
                                                  ws.E3, ws.F2, ws.T, oz_rad_const(plan));
  VCPCU_LAUNCH_CHECK("oz_radius_T_kernel");
  return VCPCU_OK;
}

}  // namespace vcpcu
