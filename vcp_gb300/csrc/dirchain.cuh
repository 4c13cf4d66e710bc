// dirchain.cuh -- sequential directed-rounding chains of non-negative doubles
// on the integer pipe (host- and device-callable, so that the CPU tests run
// the very code of the kernels).
//
//     sum chain   c = RU(c + x)        or  c = RD(c + x)
//     FMA chain   c = RU(c + a b)                          (x, a, b >= 0)
//
// GB300's FP64 pipe takes 64 cycles for a warp instruction, and 64 more
// before the next instruction of the same chain; integer instructions issue
// beside it.  A chain of non-negative terms only grows, so its last place
// changes at most a few dozen times: c is held as an integer (below 2^53) in
// units u = 2^(U - 1075), and a step is
//     c += ceil(x / u)   (RU)      c += floor(x / u)   (RD),
// which is the correctly rounded sum while it stays below 2^53 units; from
// 2^53 on the unit doubles and c becomes ceil(c / 2) (floor(c / 2)) -- nested
// ceilings (floors) by integers are one ceiling (floor) of the exact sum.
// ceil(P / 2^s) = floor((P - 1) / 2^s) + 1 is an arithmetic shift and holds
// for P = 0.  U is a double's exponent field (1 for subnormals and zero:
// their unit is 2^-1074).
//
// Where a term is at least 2^53 units (the chain's first terms, growth in
// leaps) or anything is infinite, NaN or negative, the step is the FP64
// instruction itself on the chain's value; U = CHAIN_RAW then keeps a value
// that has no such form (c its bits) on that path.
#pragma once
#include "ozaki_common.cuh"

#ifndef __CUDA_ARCH__
#include <cfenv>
#include <cmath>
#endif

namespace vcpcu {

constexpr int CHAIN_RAW = -100000;

struct DirChain {
  long long c;
  int U;
};

OZ_HD DirChain chain_zero() { return DirChain{0, 1}; }

OZ_HD double chain_from_bits(uint64_t b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)b);
#else
  double d;
  memcpy(&d, &b, 8);
  return d;
#endif
}

OZ_HD double chain_value(const DirChain& x) {
  if (x.U == CHAIN_RAW) return chain_from_bits((uint64_t)x.c);
  // (the hidden bit, if any, adds 1 to the exponent field)
  return chain_from_bits(((uint64_t)(x.U - 1) << 52) + (uint64_t)x.c);
}

OZ_HD DirChain chain_of(double v) {
  const uint64_t b = oz_bits(v);
  const int e = (int)(b >> 52);  // the sign makes it 2048 or more
  if (e >= 2047) return DirChain{(long long)b, CHAIN_RAW};
  const uint64_t m = b & ((1ULL << 52) - 1);
  return e ? DirChain{(long long)(m | (1ULL << 52)), e} : DirChain{(long long)m, 1};
}

// Significand and exponent field of a non-negative double for the chains:
// value M 2^(e - 1075); e = CHAIN_BIG for an infinity, NaN or a negative value
// (no unit is small enough: the FP64 step), CHAIN_ZERO for zero (any unit is;
// times an infinity or NaN it is the FP64 step again).
constexpr int CHAIN_BIG = 20000, CHAIN_ZERO = -8000;
OZ_HD void chain_split(uint64_t b, long long* M, int* e) {
  const int f = (int)(b >> 52);
  const uint64_t m = b & ((1ULL << 52) - 1);
  *M = (long long)(f ? m | (1ULL << 52) : m);
  *e = f >= 2047 ? CHAIN_BIG : (f ? f : (m ? 1 : CHAIN_ZERO));
}

OZ_HD double chain_add_dir(double a, double b, bool up) {
#ifdef __CUDA_ARCH__
  return up ? __dadd_ru(a, b) : __dadd_rd(a, b);
#else
  fesetround(up ? FE_UPWARD : FE_DOWNWARD);
  volatile double x = a, y = b, z = x + y;
  fesetround(FE_TONEAREST);
  return z;
#endif
}
OZ_HD double chain_fma_ru(double a, double b, double c) {
#ifdef __CUDA_ARCH__
  return __fma_ru(a, b, c);
#else
  fesetround(FE_UPWARD);
  volatile double x = a, y = b, w = c, z = std::fma(x, y, w);
  fesetround(FE_TONEAREST);
  return z;
#endif
}

// The unit doubles once the sum has reached 2^53 units; past the largest
// exponent the value is infinity (RU) or stays the largest double (RD).
template <bool UP>
OZ_HD void chain_carry(DirChain& x) {
  if ((uint32_t)((uint64_t)x.c >> 32) >= (1u << 21)) {
    x.c = (x.c + (UP ? 1 : 0)) >> 1;
    x.U += 1;
    if (x.U > 2046) {
      if (UP)
        x = DirChain{(long long)0x7ff0000000000000ULL, CHAIN_RAW};
      else
        x = DirChain{(1LL << 53) - 1, 2046};
    }
  }
}

// The FP64 steps, out of line: rare, and a loop over chains stays small.
#ifdef __CUDACC__
#define CHAIN_SLOW static __host__ __device__ __noinline__
#else
#define CHAIN_SLOW inline
#endif
template <bool UP>
CHAIN_SLOW DirChain chain_add_slow(DirChain x, double v) {
  return chain_of(chain_add_dir(chain_value(x), v, UP));
}
CHAIN_SLOW DirChain chain_fma_slow(DirChain x, double a, double b) {
  return chain_of(chain_fma_ru(a, b, chain_value(x)));
}

// c = RU / RD (c + v) for v = M 2^(e - 1075) (chain_split).
template <bool UP>
OZ_HD void chain_add(DirChain& x, double v, long long M, int e) {
  int d = x.U - e;
  if (d < 0) {
    x = chain_add_slow<UP>(x, v);
    return;
  }
  d = d < 63 ? d : 63;
  x.c += UP ? ((M - 1) >> d) + 1 : M >> d;
  chain_carry<UP>(x);
}

// Factor of an FMA chain: M = h 2^26 + l, value M 2^(e - 1075); hi is the
// double's high word (its low one is in h and l), for the FP64 step.
struct alignas(16) ChainFactor {
  int h, l, e, hi;
};
OZ_HD ChainFactor chain_factor(double v) {
  long long M;
  int e;
  chain_split(oz_bits(v), &M, &e);
  return ChainFactor{(int)(M >> 26), (int)(M & 0x3ffffff), e, (int)(oz_bits(v) >> 32)};
}
OZ_HD double chain_factor_value(const ChainFactor& f) {
  const uint32_t lo = ((uint32_t)f.h << 26) | (uint32_t)f.l;
  return chain_from_bits(((uint64_t)(uint32_t)f.hi << 32) | lo);
}

// c = RU(c + a b) for the factors of a and b.  P = Ma Mb; t = floor((P -
// 1) / 2^52) comes out of three partial products of at most 2^54 with signed
// carries; P / u = P / 2^s, s = U + 1075 - ea - eb.
OZ_HD void chain_fma(DirChain& x, const ChainFactor& fa, const ChainFactor& fb) {
  int s = x.U + 1023 - fa.e - fb.e;  // s - 52
  if (s < 1) {
    x = chain_fma_slow(x, chain_factor_value(fa), chain_factor_value(fb));
    return;
  }
  s = s < 63 ? s : 63;
  const long long t0 = (long long)fa.l * fb.l - 1;
  const long long t1 = (long long)fa.h * fb.l + ((long long)fa.l * fb.h + (t0 >> 26));
  const long long t = (long long)fa.h * fb.h + (t1 >> 26);
  x.c += (t >> s) + 1;
  chain_carry<true>(x);
}

// x >> s for any s >= 0 (the device instruction takes more than 63 for 63; a
// negative s gives a value that its caller discards).
OZ_HD long long chain_shr(long long x, int s) {
#ifdef __CUDA_ARCH__
  long long r;
  asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(s));
  return r;
#else
  return x >> (s < 0 ? 0 : (s > 63 ? 63 : s));
#endif
}

// N steps at once.  With every term below 2^53 units, the terms in units are
// independent of one another, and where the sum with all of them stays below
// 2^53 units no step doubles the unit: one sum is the whole batch (the common
// case: a chain doubles its unit some dozen times).  Else the steps go one by
// one on the terms at hand, halved with every doubling (nested ceilings and
// floors again).  Away from both: one step after the other.
constexpr int CHAIN_TOP = 2000;  // exponents from here on step singly

// y[p]: floor of the term in units (RD), or one less than its ceiling (RU).
template <bool UP, int N>
OZ_HD void chain_batch(DirChain& x, const long long (&y)[N]) {
  long long S = x.c + (UP ? N : 0);
#pragma unroll
  for (int p = 0; p < N; ++p) S += y[p];
  if ((uint32_t)((uint64_t)S >> 32) < (1u << 21)) {
    x.c = S;
    return;
  }
  int k = 0;
#pragma unroll
  for (int p = 0; p < N; ++p) {
    x.c += (y[p] >> k) + (UP ? 1 : 0);
    if ((uint32_t)((uint64_t)x.c >> 32) >= (1u << 21)) {
      x.c = (x.c + (UP ? 1 : 0)) >> 1;
      ++k;
    }
  }
  x.U += k;
}

// c = RU / RD (c + M_p 2^(e_p - 1075)), p ascending; get(p, &M, &e), value(p)
// the double itself.
template <bool UP, int N, typename GET, typename VALUE>
OZ_HD void chain_add_n(DirChain& x, GET get, VALUE value) {
  long long y[N];
  int em = CHAIN_ZERO;
#pragma unroll
  for (int p = 0; p < N; ++p) {
    int e;
    get(p, &y[p], &e);
    em = em > e ? em : e;
    y[p] = chain_shr(UP ? y[p] - 1 : y[p], x.U - e);
  }
  if (x.U < em || x.U > CHAIN_TOP || x.U < 1) {
#pragma unroll 1
    for (int p = 0; p < N; ++p) {
      long long M;
      int e;
      get(p, &M, &e);
      chain_add<UP>(x, value(p), M, e);
    }
    return;
  }
  chain_batch<UP, N>(x, y);
}

// c = RU(c + a_p b_p), p ascending, get(p, &fa, &fb) the factors: the whole
// batch at once, or false and x as it was.
template <int N, typename GET>
OZ_HD bool chain_fma_batch(DirChain& x, GET get) {
  long long y[N];
  int sm = 1;
  const int U = x.U + 1023;
#pragma unroll
  for (int p = 0; p < N; ++p) {
    ChainFactor fa, fb;
    get(p, &fa, &fb);
    const int s = U - fa.e - fb.e;
    sm = sm < s ? sm : s;
    const long long t0 = (long long)fa.l * fb.l - 1;
    const long long t1 = (long long)fa.h * fb.l + ((long long)fa.l * fb.h + (t0 >> 26));
    y[p] = chain_shr((long long)fa.h * fb.h + (t1 >> 26), s);
  }
  if (sm < 1 || x.U > CHAIN_TOP || x.U < 1) return false;
  chain_batch<true, N>(x, y);
  return true;
}
// Its steps one by one (p not a constant: get from memory).  fp64: all of them
// the FP64 instruction, for a young chain -- a term outgrows its unit so often
// that some lane of a warp takes an FP64 step at nearly every p anyway.
template <int N, typename GET>
OZ_HD void chain_fma_steps(DirChain& x, GET get, bool fp64) {
  if (fp64) {
    double c = chain_value(x);
#pragma unroll
    for (int p = 0; p < N; ++p) {
      ChainFactor fa, fb;
      get(p, &fa, &fb);
      c = chain_fma_ru(chain_factor_value(fa), chain_factor_value(fb), c);
    }
    x = chain_of(c);
    return;
  }
#pragma unroll 1
  for (int p = 0; p < N; ++p) {
    ChainFactor fa, fb;
    get(p, &fa, &fb);
    chain_fma(x, fa, fb);
  }
}
template <int N, typename GET, typename AGAIN>
OZ_HD void chain_fma_n(DirChain& x, GET get, AGAIN again) {
  if (!chain_fma_batch<N>(x, get)) chain_fma_steps<N>(x, again, false);
}

}  // namespace vcpcu
