// ozaki_prep.cuh -- one interval entry of the CRT form's operand preparation,
// in integer operations on the words of its endpoints (host- and
// device-callable, so that the CPU tests run the very code of the kernels).
//
// The common entry is narrow: both endpoints normal, of one sign and one
// binary exponent e (64 <= e <= 2046, so that every result is normal).  Bit
// patterns of one sign and exponent are integers in units of the last place
// u = 2^(e - 1075), so with s = bits(up) - bits(lo):
//     kv midpoint  RN((lo + up) / 2): bits m = bits(lo) + floor(s / 2), one
//                  more where s and that sum are odd (ties to even),
//     kv radius    max(RU(m - lo), RU(up - m)) = D u, D = (|s| + 1) / 2 (exact),
//     P = RU(|m| + r): bits |m| + D (a carry into the exponent field is the
//                  power of two itself).
// An entry that is the same zero at both ends goes the same way (all of it
// zero).
// Other entries take sw_midrad_wide (swfp.cuh).
#pragma once
#include "ozaki_common.cuh"

namespace vcpcu {

struct Words {
  uint32_t hi, lo;
};

OZ_HD uint64_t w64(Words w) { return ((uint64_t)w.hi << 32) | w.lo; }
OZ_HD Words words_of(uint64_t b) { return Words{(uint32_t)(b >> 32), (uint32_t)b}; }

OZ_HD int iv_exp(Words lo) { return (int)((lo.hi >> 20) & 0x7ffu); }
// (both ends the same zero: bit differences of [-0, +0] mean nothing)
OZ_HD bool iv_zero(Words lo, Words up) {
  return ((lo.hi << 1) | (lo.hi ^ up.hi) | lo.lo | up.lo) == 0;
}
OZ_HD bool iv_narrow(Words lo, Words up) {
  return (lo.hi ^ up.hi) < 0x100000u && (uint32_t)iv_exp(lo) - 64u <= 1982u;
}

OZ_HD int iv_clz(uint32_t x) {
#ifdef __CUDA_ARCH__
  return __clz((int)x);
#else
  return x ? __builtin_clz(x) : 32;
#endif
}
OZ_HD int iv_bitlen64(uint64_t x) {
  const uint32_t h = (uint32_t)(x >> 32);
  return h ? 64 - iv_clz(h) : 32 - iv_clz((uint32_t)x);
}

// Midpoint bits, D (radius in units u) and the bits of P of a narrow or
// zero entry.
OZ_HD void iv_midrad(Words lo, Words up, Words* m, uint64_t* D, Words* P) {
  const int64_t s = (int64_t)(w64(up) - w64(lo));
  uint64_t a = w64(lo) + (uint64_t)(s >> 1);
  a += (uint64_t)((uint32_t)s & (uint32_t)a & 1u);
  *m = words_of(a);
  const uint64_t k = (uint64_t)(s >> 63);
  *D = (((uint64_t)s ^ k) - k + 1) >> 1;
  *P = words_of((a & 0x7fffffffffffffffULL) + *D);
}

// Exponents (E with |x| <= 2^(E-1), oz_exponent) travel through integer
// maxima as E + 2^15, 0 for "all zero" (OZ_ZERO_EXP).
constexpr int OZ_EXP_BIAS = 1 << 15;
OZ_HD uint32_t exp_enc(int E) { return E == OZ_ZERO_EXP ? 0u : (uint32_t)(E + OZ_EXP_BIAS); }
OZ_HD int exp_dec(uint32_t c) { return c ? (int)c - OZ_EXP_BIAS : OZ_ZERO_EXP; }

// The encoded exponents of |m| (which is that of P, too) and of r of a narrow
// entry.  P's exponent differs only where the larger end's significand is all
// ones (iv_all_ones: the caller takes the general path there).
OZ_HD bool iv_all_ones(Words lo, Words up) { return lo.lo == 0xffffffffu || up.lo == 0xffffffffu; }
OZ_HD void iv_exponents(Words lo, Words up, uint32_t* em, uint32_t* er) {
  const int e = iv_exp(lo);
  const int64_t s = (int64_t)(w64(up) - w64(lo));
  const uint64_t k = (uint64_t)(s >> 63);
  const int bl = iv_bitlen64(((uint64_t)s ^ k) - k + 1) - 1;  // bit length of D
  *em = (uint32_t)(e - 1021 + OZ_EXP_BIAS);
  *er = bl ? (uint32_t)(e + bl - 1074 + OZ_EXP_BIAS) : 0u;
}

// Upward 16-bit radius digits: n = ceil(x 2^(16 - E)) <= 2^15 for
// 0 <= x <= 2^(E-1), -900 <= E <= 1000, as minus the floor of -x: the leading
// bits of x with a sticky bit for the rest, shifted right arithmetically.
//
// x a normal double or 0 (words hi, lo); c = E + 1028.  A shift of 31 or
// more leaves n = 1.
OZ_HD int up16_bits(uint32_t hi, uint32_t lo, int c) {
  const int be = (int)(hi >> 20);
  int sh = c - be;
  sh = sh < 31 ? sh : 31;
  const int v = (int)((((hi & 0xfffffu) | 0x100000u) << 1) | (lo ? 1u : 0u));
  const int n = -((-v) >> sh);
  return be ? n : 0;
}
// x = D 2^(e - 1075), D < 2^53; c = E + 1090 - e.
OZ_HD int up16_ulps(uint64_t D, int c) {
  const uint32_t h = (uint32_t)(D >> 32), l = (uint32_t)D;
  const uint32_t w1 = h ? h : l, w0 = h ? l : 0u;
  const int lz = iv_clz(w1);
#ifdef __CUDA_ARCH__
  const uint32_t t1 = __funnelshift_l(w0, w1, lz);
#else
  const uint32_t t1 = lz == 0 ? w1 : (lz == 32 ? w0 : (w1 << lz) | (w0 >> (32 - lz)));
#endif
  const int v = (int)((t1 >> 1) | (t1 & 1u) | ((w0 << (lz & 31)) ? 1u : 0u));
  const int bl = (h ? 64 : 32) - lz;
  int sh = c - bl;
  sh = sh < 31 ? sh : 31;
  const int n = -((-v) >> sh);
  return w1 ? n : 0;
}

}  // namespace vcpcu
