// ozaki_prep.cu -- operand preparation of the CRT form of the interval
// product C = [A]*[B] (A m x k, B k x n, kv layout, column-major), in two
// launches over both factors:
//
//   1. oz_crt_maxima: the exponents of the largest |m|, P = |m| +ru r and r of
//      every row of A, of |m| and r of every column of B (kv midrad, as
//      pidblas_assist::midrad, vcp/pidblas.hpp:43-51).  Only the exponents are
//      wanted, so a narrow entry (ozaki_prep.cuh) takes about two dozen
//      integer instructions and nothing is stored but the maxima: the pass
//      reads each factor once, at memory speed.
//   2. oz_crt_split: midrad again, and the bf16 planes that the slice GEMM
//      consumes, in tiles (oz_tile_off), per line:
//        left  (per row i):    the L residues of A' = round(mA 2^(w - Em_i));
//                              two upward digits of P (exponent Ep_i) and of
//                              rA (Er_i)
//        right (per column j): the L residues of B' = round(mB 2^(w - Fm_j));
//                              two upward digits of rB (Fr_j) and of |mB| (Fm_j)
//      with the sums of |A'|, |B'| and of the squared low radius digits (they
//      bound the low x low radius pair left out of the slice GEMM).
//
// Midrad twice costs less than storing it (32 bytes of traffic per entry).
// Bound: DRAM (16 bytes read by the first pass; 16 read and 2 (L + 4) written
// by the second).  Measured at n = 8192, L = 16, against the passes they
// replace (midrad planes stored and read back, 204 and 317 integer
// instructions per entry): maxima 0.95 -> 0.32 ms (6.6 TB/s), splits 1.62 ->
// 1.26 ms (6.0 TB/s).  1225 x 1225 x 12544: 376 -> 82 us and 399 -> 280 us
// (one warp took a whole column before).  n = 512: 13 launches before the
// slice GEMM and after it, 5 now; the call 98 -> 47 us.
//
// A factor may also be given as plain doubles (a point matrix: m = x, r = 0).
// The digit planes of a radius product that does not run are not written.
// Lines past the last are not written either (their products are never
// read); k is padded to Kp with zeros.
#include "common.cuh"
#include "ozaki.cuh"
#include "ozaki_common.cuh"
#include "ozaki_prep.cuh"
#include "ozaki_residue.cuh"
#include "swfp.cuh"

#include <cstring>
#include <type_traits>

namespace vcpcu {

namespace {

constexpr int NT = 256;
// Exponents for which the split's direct path is exact (ozaki_prep.cuh).
constexpr int LINE_EXP_MIN = -900, LINE_EXP_MAX = 1000;

// One factor of one product.  Lines are rows of A or columns of B; pointers
// are at line 0 (the planes' rows line0 ..).
struct PrepSide {
  const double* X;  // intervals (ld in intervals) or, raw, plain doubles
  long ld;
  int raw;
  int lines;
  int line0;
  size_t pstride;
  uint16_t *pm, *p1, *p2;  // residue planes; digit planes of radius product 1, 2
  uint32_t* e;             // encoded exponents: 3 per row, 2 per column
  unsigned long long* sum;  // 4 per line
};

// One product (or a block of its rows and columns).
struct PrepArgs {
  PrepSide a, b;
  int K, Kp, L, w;
  int run1, run2;  // which radius products run
  int* flag;
  int nA;          // blocks of the left factor; the others are the right one's
  int spanA, spanB;  // maxima: k range of a block; split: 64-k steps of a left block
};

__device__ __forceinline__ Words words(double x) { return words_of(sw_bits(x)); }

// The three encoded exponents of an entry off the narrow path; false: it is
// not finite.
struct Exps {
  uint32_t m, p, r;
  bool ok;
};
static __device__ __noinline__ Exps entry_exponents_general(double lo, double up) {
  Exps x{0, 0, 0, false};
  if (!sw_finite(lo) || !sw_finite(up)) return x;
  double m, r, p;
  if (!sw_midrad_wide(lo, up, m, r, p)) sw_midrad_hw(lo, up, m, r, p);
  x.m = exp_enc(oz_exponent(oz_abs(m)));
  x.p = exp_enc(oz_exponent(p));
  x.r = exp_enc(oz_exponent(r));
  x.ok = true;
  return x;
}

// Running maxima of a thread: n (narrow entries: |m| and P share it), r, and
// m, p of the others.
struct Maxima {
  uint32_t n = 0, r = 0, m = 0, p = 0;
  bool bad = false;
  __device__ __forceinline__ void add(double2 v) {
    const Words lo = words(v.x), up = words(v.y);
    if (iv_narrow(lo, up) && !iv_all_ones(lo, up)) {
      uint32_t em, er;
      iv_exponents(lo, up, &em, &er);
      n = max(n, em);
      r = max(r, er);
    } else if (!iv_zero(lo, up)) {
      const Exps x = entry_exponents_general(v.x, v.y);
      m = max(m, x.m);
      p = max(p, x.p);
      r = max(r, x.r);
      bad = bad || !x.ok;
    }
  }
};

__device__ __forceinline__ double2 load_entry(const PrepSide& s, size_t at) {
  if (s.raw) {
    const double x = s.X[at];
    return make_double2(x, x);
  }
  return reinterpret_cast<const double2*>(s.X)[at];
}

// The largest high word (sign cleared) of a thread's plain doubles: the
// exponent of the largest of them, of |m| and P alike (r = 0), where it is
// that of a normal double with biased exponent >= 64; otherwise (all small or
// zero, or some not finite) the thread takes its entries again one by one.
// Two instructions an entry, where the interval rule takes two dozen: the
// pass over a 16384 x 16384 point factor 570 -> 320 us (6.7 TB/s).
__device__ __forceinline__ bool raw_exponent(uint32_t hi, uint32_t* em) {
  const uint32_t e = hi >> 20;
  if (e - 64u > 1982u) return false;
  *em = e - 1021 + OZ_EXP_BIAS;
  return true;
}

// Rows [32 rb, + 32) of A over k in [k0, k1): lane = row, the warps take
// every eighth k, eight loads in flight per thread.
__device__ __forceinline__ void maxima_left(const PrepSide& s, int K, int rb, int k0, int* flag) {
  __shared__ uint32_t red[3][32];
  const int lane = threadIdx.x & 31, ph = threadIdx.x >> 5;
  const int i = rb * 32 + lane;
  if (threadIdx.x < 96) red[threadIdx.x >> 5][lane] = 0;
  __syncthreads();
  Maxima x;
  bool each = i < s.lines;
  if (each && s.raw) {
    constexpr int U = 16;
    uint32_t hi = 0;
    for (int c = k0 + ph; c < K; c += 8 * U) {
      double v[U];
#pragma unroll
      for (int u = 0; u < U; ++u)
        v[u] = c + 8 * u < K ? s.X[(size_t)i + (size_t)(c + 8 * u) * s.ld] : 0.0;
#pragma unroll
      for (int u = 0; u < U; ++u) hi = max(hi, words(v[u]).hi & 0x7fffffffu);
    }
    each = !raw_exponent(hi, &x.n);
  }
  if (each) {
    constexpr int U = 8;
    for (int c = k0 + ph; c < K; c += 8 * U) {
      double2 v[U];
#pragma unroll
      for (int u = 0; u < U; ++u)
        v[u] = c + 8 * u < K ? load_entry(s, (size_t)i + (size_t)(c + 8 * u) * s.ld)
                             : make_double2(0.0, 0.0);
#pragma unroll
      for (int u = 0; u < U; ++u) x.add(v[u]);
    }
  }
  if (x.bad) atomicOr(flag, 1);
  atomicMax(&red[0][lane], max(x.n, x.m));
  atomicMax(&red[1][lane], max(x.n, x.p));
  atomicMax(&red[2][lane], x.r);
  __syncthreads();
  if (threadIdx.x < 96) {
    const int t = threadIdx.x >> 5;
    if (i < s.lines && red[t][lane]) atomicMax(&s.e[3 * i + t], red[t][lane]);
  }
}

// Columns [8 cb, + 8) of B over k in [k0, k1): one warp per column.
__device__ __forceinline__ void maxima_right(const PrepSide& s, int k0, int k1, int cb,
                                             int* flag) {
  const int lane = threadIdx.x & 31;
  const int j = cb * 8 + (threadIdx.x >> 5);
  if (j >= s.lines) return;  // whole warps only
  const size_t at = (size_t)j * s.ld;
  Maxima x;
  bool each = true;
  if (s.raw) {
    constexpr int U = 8;
    uint32_t hi = 0;
    for (int k = k0 + lane; k < k1; k += 32 * U) {
      double v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) v[u] = k + 32 * u < k1 ? s.X[at + k + 32 * u] : 0.0;
#pragma unroll
      for (int u = 0; u < U; ++u) hi = max(hi, words(v[u]).hi & 0x7fffffffu);
    }
    each = !raw_exponent(hi, &x.n);
  }
  if (each) {
    constexpr int U = 8;
    for (int k = k0 + lane; k < k1; k += 32 * U) {
      double2 v[U];
#pragma unroll
      for (int u = 0; u < U; ++u)
        v[u] = k + 32 * u < k1 ? load_entry(s, at + k + 32 * u) : make_double2(0.0, 0.0);
#pragma unroll
      for (int u = 0; u < U; ++u) x.add(v[u]);
    }
  }
  const bool bad = __any_sync(0xffffffffu, x.bad);
  const uint32_t em = __reduce_max_sync(0xffffffffu, max(x.n, x.m)),
                 er = __reduce_max_sync(0xffffffffu, x.r);
  if (lane == 0) {
    if (bad) atomicOr(flag, 1);
    if (em) atomicMax(&s.e[2 * j], em);
    if (er) atomicMax(&s.e[2 * j + 1], er);
  }
}

// Block `local` of a product: the left factor's blocks (row blocks fastest:
// neighbours read adjacent rows), then the right one's.
__device__ __forceinline__ void maxima_block(const PrepArgs& p, int local) {
  if (local < p.nA) {
    const int nrb = (p.a.lines + 31) >> 5;
    const int rb = local % nrb, k0 = (local / nrb) * p.spanA;
    maxima_left(p.a, min(p.K, k0 + p.spanA), rb, k0, p.flag);
  } else {
    local -= p.nA;
    const int ncb = (p.b.lines + 7) >> 3;
    const int cb = local % ncb, k0 = (local / ncb) * p.spanB;
    maxima_right(p.b, k0, min(p.K, k0 + p.spanB), cb, p.flag);
  }
}

__global__ void __launch_bounds__(NT) oz_crt_maxima(const __grid_constant__ PrepArgs p) {
  dep_ready();
  maxima_block(p, blockIdx.x);
}

// ----------------------------------------------------------------- split
// w-bit integer of x (|x| <= 2^(E-1)): round to nearest even, |result| <=
// 2^(w-1), for any E.  x 2^(w-E) is formed exactly by power-of-two
// multiplications (no overflow: it stays below 2^(w-1); a subnormal
// intermediate is below 2^-1022 and converts to 0 either way) and converted
// with one rounding.
__device__ __forceinline__ long long crt_int(double x, int E, int w) {
  if (E == OZ_ZERO_EXP || oz_zero(x)) return 0;
  int s = w - E;
  if (s < -1100) return 0;  // |x| 2^s < 2^-76
  double y = x;
  while (s > 1000) {
    y = __dmul_rn(y, 0x1p1000);
    s -= 1000;
  }
  while (s < -1000) {
    y = __dmul_rn(y, 0x1p-1000);
    s += 1000;
  }
  return __double2ll_rn(__dmul_rn(y, __longlong_as_double((long long)(s + 1023) << 52)));
}

// Per-line constants.  The digits that come from the bits of a double (P of
// a row, |mB| of a column) have exponent Eb, those of the radius Er.
struct Line {
  double scale;  // 2^(w - E): A' = RN(m scale)
  int E, Eb, Er;
  bool direct;   // every exponent in the direct path's range (or no such value)
};
__device__ __forceinline__ bool line_exp_ok(int E) {
  return E == OZ_ZERO_EXP || (E >= LINE_EXP_MIN && E <= LINE_EXP_MAX);
}
__device__ __forceinline__ Line make_line(int E, int Eb, int Er, int w) {
  Line x{0.0, E, Eb, Er, line_exp_ok(E) && line_exp_ok(Eb) && line_exp_ok(Er)};
  if (x.direct && E != OZ_ZERO_EXP)
    x.scale = __longlong_as_double((long long)(w - E + 1023) << 52);
  return x;
}

struct Ints {
  long long a;  // w-bit integer of the midpoint
  int nb, nr;   // 16-bit upward integers of P or |m|, and of r
};

// An entry off the direct path (not narrow, or exponents beyond its range).
template <bool LEFT>
static __device__ __noinline__ Ints entry_general(double lo, double up, int E, int Eb, int Er,
                                                  int w) {
  Ints x{0, 0, 0};
  if (!sw_finite(lo) || !sw_finite(up)) return x;  // the whole result is NaN then
  double m, r, p;
  if (!sw_midrad_wide(lo, up, m, r, p)) sw_midrad_hw(lo, up, m, r, p);
  x.a = crt_int(m, E, w);
  if (Eb != OZ_ZERO_EXP) x.nb = (int)oz_scaled_int64(LEFT ? p : oz_abs(m), Eb, 16, 1);
  if (Er != OZ_ZERO_EXP) x.nr = (int)oz_scaled_int64(r, Er, 16, 1);
  return x;
}

template <bool LEFT>
__device__ __forceinline__ Ints entry_ints(double2 v, const Line& ln, int w) {
  const Words lo = words(v.x), up = words(v.y);
  if (ln.direct && (iv_narrow(lo, up) || iv_zero(lo, up))) {
    Words m, P;
    uint64_t D;
    iv_midrad(lo, up, &m, &D, &P);
    Ints x;
    x.a = __double2ll_rn(__dmul_rn(sw_double(w64(m)), ln.scale));
    x.nb = LEFT ? up16_bits(P.hi, P.lo, ln.Eb + 1028)
                : up16_bits(m.hi & 0x7fffffffu, m.lo, ln.Eb + 1028);
    x.nr = up16_ulps(D, ln.Er + 1090 - iv_exp(lo));
    return x;
  }
  return entry_general<LEFT>(v.x, v.y, ln.E, ln.Eb, ln.Er, w);
}

// High and low digit of n <= 2^15: n = 256 d1 + d0, d0 in [-128, 127].
__device__ __forceinline__ void digits16(int n, int& d1, int& d0) {
  d0 = (int)(int8_t)n;
  d1 = (n + 128) >> 8;
}

// An entry of a point factor where no radius product runs: its integer alone.
static __device__ __noinline__ long long point_general(double x, int E, int w) {
  return sw_finite(x) ? crt_int(x, E, w) : 0;
}
__device__ __forceinline__ long long point_int(double x, const Line& ln, int w) {
  const Words b = words(x);
  if (ln.direct && ((uint32_t)iv_exp(b) - 64u <= 1982u || ((b.hi << 1) | b.lo) == 0))
    return __double2ll_rn(__dmul_rn(x, ln.scale));
  return point_general(x, ln.E, w);
}
__device__ __forceinline__ double load_split(const PrepSide& s, size_t at, double) {
  return s.X[at];
}
__device__ __forceinline__ double2 load_split(const PrepSide& s, size_t at, double2) {
  return load_entry(s, at);
}
__device__ __forceinline__ void zero_split(double& v) { v = 0.0; }
__device__ __forceinline__ void zero_split(double2& v) { v = make_double2(0.0, 0.0); }

// Sums of a thread's entries.
struct LineSums {
  unsigned long long hi = 0, lo = 0;  // sum |A'| = hi 2^32 + lo
  uint32_t qb = 0, qr = 0;            // squares of the low digits
};

// Eight consecutive k of one line: digit planes (dst1 / dst2: products 1 /
// 2), residue planes, sums.  off is the element offset of the first within a
// plane; store false (a line past the last) writes nothing.
// V: double2, or double (POINT kernels: both factors plain doubles and no
// radius product, so no digits).
template <int NL, bool LEFT, class V>
__device__ __forceinline__ void split8(const V (&v)[8], const Line& ln, const PrepArgs& p,
                                       const PrepSide& s, size_t off, bool store, LineSums& sums) {
  constexpr bool POINT = std::is_same_v<V, double>;
  unsigned long long h[4][NL];
  uint32_t b1[4] = {}, b0[4] = {}, r1[4] = {}, r0[4] = {};
  const bool digits = !POINT && (p.run1 | p.run2);  // (no radius product: both radii are zero)
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    Ints x, y;
    if constexpr (POINT) {
      x = Ints{point_int(v[2 * t], ln, p.w), 0, 0};
      y = Ints{point_int(v[2 * t + 1], ln, p.w), 0, 0};
    } else {
      x = entry_ints<LEFT>(v[2 * t], ln, p.w);
      y = entry_ints<LEFT>(v[2 * t + 1], ln, p.w);
    }
    limbs_pair<NL>(x.a, y.a, h[t]);
    const unsigned long long ax = (unsigned long long)(x.a < 0 ? -x.a : x.a),
                             ay = (unsigned long long)(y.a < 0 ? -y.a : y.a);
    if constexpr (NL == 4) {  // |A'| <= 2^55: plain 64-bit sums
      sums.lo += ax + ay;
    } else {
      sums.hi += (ax >> 32) + (ay >> 32);
      sums.lo += (ax & 0xffffffffULL) + (ay & 0xffffffffULL);
    }
    if (!digits) continue;
    int xb1, xb0, yb1, yb0, xr1, xr0, yr1, yr0;
    digits16(x.nb, xb1, xb0);
    digits16(y.nb, yb1, yb0);
    digits16(x.nr, xr1, xr0);
    digits16(y.nr, yr1, yr0);
    sums.qb += (uint32_t)(xb0 * xb0 + yb0 * yb0);
    sums.qr += (uint32_t)(xr0 * xr0 + yr0 * yr0);
    b1[t] = bf16_pair(xb1, yb1);
    b0[t] = bf16_pair(xb0, yb0);
    r1[t] = bf16_pair(xr1, yr1);
    r0[t] = bf16_pair(xr0, yr0);
  }
  if (!store) return;
  auto put = [&](uint16_t* plane, const uint32_t (&x)[4]) {
    *reinterpret_cast<uint4*>(plane + off) = make_uint4(x[0], x[1], x[2], x[3]);
  };
  if (!POINT && p.run1) {  // (|mA| + rA) rB
    put(s.p1, LEFT ? b1 : r1);
    put(s.p1 + s.pstride, LEFT ? b0 : r0);
  }
  if (!POINT && p.run2) {  // rA |mB|
    put(s.p2, LEFT ? r1 : b1);
    put(s.p2 + s.pstride, LEFT ? r0 : b0);
  }
#pragma unroll
  for (int l = 0; l < OZ_MAX_MODULI_128; ++l) {
    if (l >= p.L) break;
    uint32_t x[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) x[t] = res_pair<NL>(h[t], l);
    put(s.pm + l * s.pstride, x);
  }
}

// Adds a thread's sums, reduced over `lanes` lanes whose first is `first`, to
// the line's: sum_k |A'| as (bits >= 32, bits < 32), the squares of the low
// digits of (P, rA) or (rB, |mB|).
template <int NL, bool LEFT>
__device__ __forceinline__ void add_sums(LineSums x, int lanes, int step, bool first,
                                         unsigned long long* sum) {
  for (int o = step; o < lanes * step; o <<= 1) {
    x.lo += __shfl_xor_sync(0xffffffffu, x.lo, o);
    if (NL != 4) x.hi += __shfl_xor_sync(0xffffffffu, x.hi, o);
    x.qb += __shfl_xor_sync(0xffffffffu, x.qb, o);
    x.qr += __shfl_xor_sync(0xffffffffu, x.qr, o);
  }
  if (!first) return;
  if (NL == 4) {  // at most 2^55 per entry, 2^8 entries: below 2^64
    x.hi = x.lo >> 32;
    x.lo &= 0xffffffffULL;
  }
  if (x.hi | x.lo) {
    atomicAdd(&sum[0], x.hi);
    atomicAdd(&sum[1], x.lo);
  }
  const uint32_t q2 = LEFT ? x.qb : x.qr, q3 = LEFT ? x.qr : x.qb;
  if (q2) atomicAdd(&sum[2], (unsigned long long)q2);
  if (q3) atomicAdd(&sum[3], (unsigned long long)q3);
}

// Rows [32 rb, + 32), steps of 64 k from 64 kb0: a warp takes 8 rows x 32 k,
// lane = k-group + 4 row.  The eight lanes that a 16-byte store serves at a
// time then write two lines of a plane (with rows fastest they wrote eight,
// and the store pipe, 36 passes an instruction, was the bound: 1225x12544
// 332 -> 301 us, n = 8192 1441 -> 1311).
template <int NL, class V>
__device__ __forceinline__ void split_left(const PrepArgs& p, int rb, int kb0, int steps) {
  const PrepSide& s = p.a;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i = rb * 32 + (warp & 3) * 8 + (lane >> 2);
  const bool row = i < s.lines;
  const uint32_t* e = s.e + 3 * (size_t)i;
  const Line ln = row ? make_line(exp_dec(e[0]), exp_dec(e[1]), exp_dec(e[2]), p.w)
                      : make_line(OZ_ZERO_EXP, OZ_ZERO_EXP, OZ_ZERO_EXP, p.w);
  LineSums sums;
  for (int it = 0; it < steps; ++it) {
    const int k = (kb0 + it) * 64 + (warp >> 2) * 32 + (lane & 3) * 8;
    if ((kb0 + it) * 64 >= p.Kp) break;
    V v[8];
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      zero_split(v[t]);
      if (row && k + t < p.K) v[t] = load_split(s, (size_t)i + (size_t)(k + t) * s.ld, V());
    }
    split8<NL, true>(v, ln, p, s, oz_tile_off(s.line0 + i, OZ_BM, k, p.Kp), row, sums);
  }
  add_sums<NL, true>(sums, 4, 1, row && (lane & 3) == 0, s.sum + 4 * (size_t)i);
}

// Lanes per column of the right split: as many as its padded length fills
// with 8 k each, a power of two; a warp takes 32 / lanes columns.
__host__ __device__ __forceinline__ int right_lanes(int Kp) {
  return Kp <= 64 ? 8 : (Kp <= 128 ? 16 : 32);
}

// The columns of block cb over the k range kb (8 lanes-per-column k).  The
// warp's 256 entries are read coalesced and turned to 8 consecutive k per
// lane through shared memory (one 16-byte slot of padding per 8 entries: no
// bank conflicts), so that a plane's store is 16 bytes per lane, contiguous
// along each column.
template <int NL, class V>
__device__ __forceinline__ void split_right(const PrepArgs& p, int cb, int kb) {
  __shared__ V turn[NT / 32][288];
  const PrepSide& s = p.b;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int lanes = right_lanes(p.Kp), per = 8 * lanes;  // lanes and k per column
  const int col0 = (cb * 8 + warp) * (32 / lanes);
  if (col0 >= s.lines) return;  // whole warps only (no block barrier below)
  const int k0 = kb * per;
  V* T = turn[warp];
  {
    V v[8];
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      const int x = 32 * t + lane, j = col0 + x / per, k = k0 + (x & (per - 1));
      zero_split(v[t]);
      if (j < s.lines && k < p.K) v[t] = load_split(s, (size_t)k + (size_t)j * s.ld, V());
    }
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      const int x = 32 * t + lane;
      T[x + (x >> 3)] = v[t];
    }
  }
  __syncwarp();
  const int j = col0 + lane / lanes, k = k0 + (lane & (lanes - 1)) * 8;
  const bool col = j < s.lines;
  const uint32_t* e = s.e + 2 * (size_t)j;
  const int Fm = col ? exp_dec(e[0]) : OZ_ZERO_EXP, Fr = col ? exp_dec(e[1]) : OZ_ZERO_EXP;
  const Line ln = make_line(Fm, Fm, Fr, p.w);
  V v[8];
#pragma unroll
  for (int t = 0; t < 8; ++t) v[t] = T[9 * lane + t];
  LineSums sums;
  split8<NL, false>(v, ln, p, s, oz_tile_off(s.line0 + j, OZ_BN, k, p.Kp), col && k < p.Kp,
                    sums);
  add_sums<NL, false>(sums, lanes, 1, col && (lane & (lanes - 1)) == 0, s.sum + 4 * (size_t)j);
}

template <int NL, class V>
__device__ __forceinline__ void split_block(const PrepArgs& p, int local) {
  if (local < p.nA) {
    const int nrb = (p.a.lines + 31) >> 5;
    split_left<NL, V>(p, local % nrb, (local / nrb) * p.spanA, p.spanA);
  } else {
    local -= p.nA;
    const int nkb = (p.Kp + 8 * right_lanes(p.Kp) - 1) / (8 * right_lanes(p.Kp));
    split_right<NL, V>(p, local / nkb, local % nkb);
  }
}

// Two point factors without a radius product (the directed point product) hold
// one double an entry, no digits and no width test: 62 registers, so that a
// fourth block fits an SM, and 16384 x 16384 takes 1600 us where the general
// kernel took 2360 (10.7 GB: 6.7 TB/s; 4.5 before).  The general kernel at four
// blocks spills (n = 8192 1.25 -> 1.43 ms), at two it is 12 % slower.
template <int NL, class V>
__global__ void __launch_bounds__(NT, std::is_same_v<V, double> && NL < 6 ? 4 : 3)
oz_crt_split(const __grid_constant__ PrepArgs p) {
  dep_wait();
  dep_ready();
  split_block<NL, V>(p, blockIdx.x);
}

// ------------------------------------------------------ grouped products
// The problems of a bucket: block -> problem by a table, its PrepArgs from its
// descriptor.
__device__ __forceinline__ PrepArgs group_args(const OzGBucket& b, const OzGProb& q, int p) {
  PrepArgs a;
  const size_t psA = (size_t)b.Arows * 64, psB = (size_t)b.Brows * 64;
  uint16_t* pA = b.planesA + (size_t)q.arow * 64;
  uint16_t* pB = b.planesB + (size_t)q.brow * 64;
  a.a = PrepSide{q.A, q.lda, 0, q.m, 0, psA, pA, pA + b.Lmax * psA, pA + (b.Lmax + 2) * psA,
                 b.eA + 3 * (size_t)q.rowoff, b.asum + 4 * (size_t)q.rowoff};
  a.b = PrepSide{q.B, q.ldb, 0, q.n, 0, psB, pB, pB + b.Lmax * psB, pB + (b.Lmax + 2) * psB,
                 b.eB + 2 * (size_t)q.coloff, b.bsum + 4 * (size_t)q.coloff};
  a.K = q.k;
  a.Kp = q.Kp;
  a.L = q.L;
  a.w = q.w;
  a.run1 = a.run2 = 1;
  a.flag = b.flag + 4 * p;
  return a;
}

__device__ __forceinline__ unsigned long long g_timer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__global__ void __launch_bounds__(NT) oz_crt_maxima_g(const __grid_constant__ OzGBucket b) {
  const int p = b.prob_max[blockIdx.x];
  const OzGProb& q = b.probs[p];
  if (threadIdx.x == 0 && b.t_first) atomicMin(&b.t_first[q.orig], g_timer());
  PrepArgs a = group_args(b, q, p);
  a.nA = q.max_left;
  a.spanA = a.spanB = OZ_GMAX_SPAN;
  maxima_block(a, blockIdx.x - b.blk_max[p]);
}

template <int NL>
__global__ void __launch_bounds__(NT, 3) oz_crt_split_g(const __grid_constant__ OzGBucket b) {
  const int p = b.prob_split[blockIdx.x];
  const OzGProb& q = b.probs[p];
  PrepArgs a = group_args(b, q, p);
  a.nA = q.split_left;
  a.spanA = 1;
  split_block<NL, double2>(a, blockIdx.x - b.blk_split[p]);
}

inline int cdiv(long a, long b) { return (int)((a + b - 1) / b); }

// Launches both passes over the factors of p (either may have no lines).
int prepare(PrepArgs& p, cudaStream_t st) {
  bool after_maxima = false;  // a kernel of this call precedes the split
  const int nrb = cdiv(p.a.lines, 32), ncb = cdiv(p.b.lines, 8);
  if (p.K > 0) {
    // k range of a block: about eight blocks for each of the 152 SMs, so that
    // a small or a long and narrow factor spreads too
    auto span = [&](int line_blocks, int least) {
      int x = 1024;
      while (x > least && (long)line_blocks * cdiv(p.K, x) < 608) x >>= 1;
      return x;
    };
    p.spanA = span(nrb, 64);
    p.spanB = span(ncb, 256);
    p.nA = nrb * cdiv(p.K, p.spanA);
    const long blocks = (long)p.nA + (long)ncb * cdiv(p.K, p.spanB);
    if (blocks > 0) {
      oz_crt_maxima<<<(unsigned)blocks, NT, 0, st>>>(p);
      VCPCU_LAUNCH_CHECK("oz_crt_maxima");
      after_maxima = true;
    }
  }
  // 64-k steps of a left block: four (fewer additions to the row sums) where
  // that leaves enough blocks
  p.spanA = (long)nrb * cdiv(p.Kp, 256) >= 1216 ? 4 : 1;
  p.nA = nrb * cdiv(p.Kp, 64 * p.spanA);
  const int lanes = right_lanes(p.Kp);
  const long blocks = (long)p.nA + (long)cdiv(p.b.lines, 8 * (32 / lanes)) * cdiv(p.Kp, 8 * lanes);
  if (blocks <= 0) return VCPCU_OK;
  // |A'|, |B'| <= 2^(w-1): four 14-bit limbs up to w = 56, five 12-bit limbs
  // up to w = 61, six up to 73
  const bool point = p.a.raw && p.b.raw && !p.run1 && !p.run2;
  const auto split =
      point ? (p.w <= 56 ? oz_crt_split<4, double>
                         : (p.w <= 61 ? oz_crt_split<5, double> : oz_crt_split<6, double>))
            : (p.w <= 56 ? oz_crt_split<4, double2>
                         : (p.w <= 61 ? oz_crt_split<5, double2> : oz_crt_split<6, double2>));
  VCPCU_CUDA_TRY(launch_dep(after_maxima, 1, split, dim3((unsigned)blocks), dim3(NT), 0, st, p));
  VCPCU_LAUNCH_CHECK("oz_crt_split");
  return VCPCU_OK;
}

PrepSide left_side(const OzProblem& pb, const OzOperand& A, int i0, int rows, OzWorkspace& ws) {
  const int mv = pb.M - i0 < rows ? (pb.M - i0 > 0 ? pb.M - i0 : 0) : rows;
  return PrepSide{A.x + (size_t)(A.raw ? 1 : 2) * i0, A.ld, A.raw, mv, i0,
                  (size_t)pb.Mp * pb.Kp, ws.a_mid, ws.a_p, ws.a_r, ws.eA + 3 * (size_t)i0,
                  ws.asum + 4 * (size_t)i0};
}
PrepSide right_side(const OzProblem& pb, const OzOperand& B, int j0, int cols, OzWorkspace& ws) {
  const int nv = pb.N - j0 < cols ? (pb.N - j0 > 0 ? pb.N - j0 : 0) : cols;
  return PrepSide{B.x + (size_t)(B.raw ? 1 : 2) * j0 * B.ld, B.ld, B.raw, nv, j0,
                  (size_t)pb.Np * pb.Kp, ws.b_mid, ws.b_r, ws.b_s, ws.eB + 2 * (size_t)j0,
                  ws.bsum + 4 * (size_t)j0};
}
PrepArgs prep_args(const OzProblem& pb, int point_mask, OzWorkspace& ws) {
  PrepArgs p;
  memset(&p, 0, sizeof(p));
  p.K = pb.K;
  p.Kp = pb.Kp;
  p.L = pb.L;
  p.w = pb.w;
  p.run1 = !(point_mask & 2);
  p.run2 = !(point_mask & 1);
  p.flag = ws.flag;
  return p;
}

}  // namespace

int oz_prepare_begin(OzWorkspace& ws, cudaStream_t st) {
  VCPCU_CUDA_TRY(cudaMemsetAsync(ws.zero, 0, ws.zero_bytes, st));
  return VCPCU_OK;
}

int oz_prepare_left_rows(const OzProblem& pb, const OzOperand& A, int i0, int rows,
                         OzWorkspace& ws, cudaStream_t st) {
  PrepArgs p = prep_args(pb, 0, ws);
  p.a = left_side(pb, A, i0, rows, ws);
  return prepare(p, st);
}

int oz_prepare_right_cols(const OzProblem& pb, const OzOperand& B, int j0, int cols,
                          OzWorkspace& ws, cudaStream_t st) {
  PrepArgs p = prep_args(pb, 0, ws);
  p.b = right_side(pb, B, j0, cols, ws);
  return prepare(p, st);
}

int oz_prepare(const OzProblem& pb, int point_mask, const OzOperand& A, const OzOperand& B,
               OzWorkspace& ws, cudaStream_t st) {
  if (int e = oz_prepare_begin(ws, st)) return e;
  PrepArgs p = prep_args(pb, point_mask, ws);
  p.a = left_side(pb, A, 0, pb.M, ws);
  p.b = right_side(pb, B, 0, pb.N, ws);
  return prepare(p, st);
}

void oz_gprep_blocks(int m, int n, int k, int Kp, OzGProb* q, int* max_blocks, int* split_blocks) {
  const int lanes = right_lanes(Kp);
  q->max_left = cdiv(m, 32) * cdiv(k, OZ_GMAX_SPAN);
  *max_blocks = q->max_left + cdiv(n, 8) * cdiv(k, OZ_GMAX_SPAN);
  q->split_left = cdiv(m, 32) * (Kp / 64);
  *split_blocks = q->split_left + cdiv(n, 8 * (32 / lanes)) * cdiv(Kp, 8 * lanes);
}

int oz_gprep(const OzGBucket& b, int nblk_max, int nblk_split, int wmax, cudaStream_t st) {
  if (nblk_max > 0) {
    oz_crt_maxima_g<<<nblk_max, NT, 0, st>>>(b);
    VCPCU_LAUNCH_CHECK("oz_crt_maxima_g");
  }
  if (nblk_split <= 0) return VCPCU_OK;
  if (wmax <= 56)
    oz_crt_split_g<4><<<nblk_split, NT, 0, st>>>(b);
  else
    oz_crt_split_g<6><<<nblk_split, NT, 0, st>>>(b);
  VCPCU_LAUNCH_CHECK("oz_crt_split_g");
  return VCPCU_OK;
}

}  // namespace vcpcu
