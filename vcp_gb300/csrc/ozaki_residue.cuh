// ozaki_residue.cuh -- residues of scaled integers modulo the CRT moduli, on
// the FP32 pipe, as bf16 patterns (the operand planes of the slice GEMM).
#pragma once
#include "ozaki_common.cuh"

namespace vcpcu {

// The moduli, largest first (the list the host plan indexes).
#define OZ_MOD_LIST(F)                                                                   \
  F(256), F(255), F(253), F(251), F(247), F(241), F(239), F(233), F(229), F(227), F(223),     \
      F(217), F(211), F(199), F(197), F(193), F(191), F(181), F(179), F(173), F(167), F(163), \
      F(157), F(151), F(149), F(139), F(137), F(131), F(127), F(113), F(109), F(107)

// Residues on the FP32 pipe (the integer multiply pipe is half as wide).
// a is cut into b-bit limbs h_t, the last one signed (b = 12; b = 14 for the
// four-limb form, which holds magnitudes <= 2^55, and the eight-limb form of
// the dd product, magnitudes <= 2^111), exact as floats, and
// x = sum_t h_t c_lt with c_lt = 2^(b t) mod m_l taken in [-m_l/2, m_l/2]:
// |x| <= h_0 + 128 sum_{t>0} |h_t| <= 2^14 + 128 (6 2^14 + 2^13) < 2^24 in the
// longest form, an exact float.  The quotient q = rint(x RN(1/m)) is within
// 1/2 + |x / m| 2^-24 of x / m (|x| 2^-24 <= 0.82; exact for m = 256), so the
// integer r = x - q m (one exact FMA) has |r| <= m/2 + 0.82, i.e. |r| <= 128:
// a residue of a in the range the slice GEMM's exact chunk sums allow
// (|r_a r_b| <= 2^14 over 1024 terms), and exact in bf16.
__host__ __device__ constexpr int oz_limb_bits(int NL) {
  return NL == 4 || NL == 8 ? 14 : 12;
}
constexpr float oz_limb_c(unsigned long long m, int b, int t) {
  unsigned long long c = 1 % m;
  for (int i = 0; i < t; ++i) c = (c << b) % m;
  return 2 * c > m ? (float)c - (float)m : (float)c;
}
// (every constant twice: the two halves of a paired operand in one load)
struct alignas(8) OzPair {
  float a, b;
};
constexpr OzPair oz_dup(float c) { return {c, c}; }
constexpr OzPair oz_limb_cc(unsigned long long m, int b, int t) { return oz_dup(oz_limb_c(m, b, t)); }
#define OZ_LIMB_ROW(m)                                                                     \
  {oz_limb_cc(m, 12, 0), oz_limb_cc(m, 12, 1), oz_limb_cc(m, 12, 2), oz_limb_cc(m, 12, 3), \
   oz_limb_cc(m, 12, 4), oz_limb_cc(m, 12, 5)}
#define OZ_LIMB14_ROW(m)                                                                   \
  {oz_limb_cc(m, 14, 0), oz_limb_cc(m, 14, 1), oz_limb_cc(m, 14, 2), oz_limb_cc(m, 14, 3), \
   oz_limb_cc(m, 14, 4), oz_limb_cc(m, 14, 5), oz_limb_cc(m, 14, 6), oz_limb_cc(m, 14, 7)}
#define OZ_NEGM(m) oz_dup(-(float)(m))
#define OZ_INVF(m) oz_dup(1.0f / (float)(m))
static __constant__ OzPair c_limb[OZ_MAX_MODULI][6] = {OZ_MOD_LIST(OZ_LIMB_ROW)};
static __constant__ OzPair c_limb14[OZ_MAX_MODULI][8] = {OZ_MOD_LIST(OZ_LIMB14_ROW)};
static __constant__ OzPair c_negm[OZ_MAX_MODULI] = {OZ_MOD_LIST(OZ_NEGM)};
static __constant__ OzPair c_inv[OZ_MAX_MODULI] = {OZ_MOD_LIST(OZ_INVF)};
__device__ __forceinline__ unsigned long long oz_pair(const OzPair& p) {
  return *reinterpret_cast<const unsigned long long*>(&p);
}

// bf16 bit pattern of an integer digit |d| <= 256 (exact: the float has at
// most 9 significant bits, so its low 16 bits are zero).  The float is made
// on the FP32 pipe -- 1.5 2^23 + d by adding d to the bit pattern, minus
// 1.5 2^23 (exact for |d| < 2^22) -- instead of an integer conversion, which
// GB300 issues on its narrow FP64 / conversion pipe.
__device__ __forceinline__ uint32_t bf16_bits(int d) {
  return __float_as_uint(__fadd_rn(__int_as_float(0x4B400000 + d), -12582912.0f)) >> 16;
}

// bf16 patterns of two integer digits in one word, the first in the low half.
__device__ __forceinline__ uint32_t bf16_pair(int d0, int d1) {
  const unsigned long long f =
      add_x2(f32x2(__int_as_float(0x4B400000 + d0), __int_as_float(0x4B400000 + d1)),
             f32x2(-12582912.0f, -12582912.0f));
  return __byte_perm((uint32_t)f, (uint32_t)(f >> 32), 0x7632);
}

// Limbs of two signed integers a0, a1 (|a| <= 2^(w-1)) as pairs of exact
// floats: b-bit limbs of the two's complement (b = oz_limb_bits(NL)), the
// last one signed, so that a = sum_t h_t 2^(b t).
template <int NL, typename INT>
__device__ __forceinline__ void limbs_pair(INT a0, INT a1, unsigned long long (&h)[NL]) {
  constexpr int B = oz_limb_bits(NL);
  constexpr unsigned mask = (1u << B) - 1;
#pragma unroll
  for (int t = 0; t < NL - 1; ++t) {
    const unsigned v0 = (unsigned)(a0 >> (B * t)) & mask, v1 = (unsigned)(a1 >> (B * t)) & mask;
    h[t] = add_x2(f32x2(__uint_as_float(0x4B000000u | v0), __uint_as_float(0x4B000000u | v1)),
                  f32x2(-8388608.0f, -8388608.0f));
  }
  const int s0 = (int)(a0 >> (B * (NL - 1))), s1 = (int)(a1 >> (B * (NL - 1)));
  h[NL - 1] = add_x2(f32x2(__int_as_float(0x4B400000 + s0), __int_as_float(0x4B400000 + s1)),
                     f32x2(-12582912.0f, -12582912.0f));
}

// The residues r, |r| <= 128 (see above), of two integers given by their limb
// pairs, modulo modulus l, as one word of two bf16 patterns (the first in the
// low half): x = h_0 + sum_t h_t c_t by an FMA chain, q = rint(x RN(1/m)) by
// the FMA onto 1.5 2^23 (one rounding, to nearest for |v| < 2^22) and its
// subtraction, and r = RN(q (-m) + x), exact.
template <int NL>
__device__ __forceinline__ uint32_t res_pair(const unsigned long long (&h)[NL], int l) {
  const unsigned long long magic = f32x2(12582912.0f, 12582912.0f);
  unsigned long long x = h[0];
#pragma unroll
  for (int t = 1; t < NL; ++t)
    x = fma_x2(h[t], oz_pair(oz_limb_bits(NL) == 14 ? c_limb14[l][t] : c_limb[l][t]), x);
  const unsigned long long q = sub_x2(fma_x2(x, oz_pair(c_inv[l]), magic), magic);
  const unsigned long long r = fma_x2(q, oz_pair(c_negm[l]), x);
  return __byte_perm((uint32_t)r, (uint32_t)(r >> 32), 0x7632);
}

}  // namespace vcpcu
