// ozaki_crt.cuh -- Chinese remaindering of the interval CRT form: the basis
// of a plan's moduli (host) and the exact value of one entry from its
// residues (host- and device-callable, so that the CPU tests run the very
// code of the reassembly kernels).
//
// The moduli m_0 .. m_{L-1} (at most 16, each <= 256) are taken in groups of
// three.  With P_g the product of group g (< 2^24) and a_l = P_g / m_l
// (< 2^16), one group value
//     V_g = sum_{l in g} c_l a_l          (< 3 * 2^24: 32-bit arithmetic)
// stands for the three residues c_l: V_g = c_l a_l mod m_l.  The basis value
// Q_g = (M / P_g) t_g, t_g = (a_l M / P_g)^-1 mod m_l for every l in g,
// undoes the factor, so S = sum_g V_g Q_g = X mod M: six multi-limb products
// instead of sixteen.  Basis and modulus are shifted left by z bits so that
// M' = M 2^z lies in [2^127, 2^128): the limbs sit at fixed places whatever
// L is, and the value found is X 2^z (the caller subtracts z from its
// exponent).
//
// Quotient.  S' / M' < 2^28.2, and |X| < M / 4 (the plan's moduli), so
// S' / M' lies within 1/4 of the integer q with S' = q M' + X 2^z.  With
// T = floor of the top of S' in units 2^96 and R = 2^159 / M' rounded (2^-32
// relative), T R 2^-63 is within 2^-3.8 + 2^-30 of S' / M': its nearest
// integer is q, with no correction step.  S' - q M' is formed modulo 2^128 by
// adding q (2^128 - M'); it is X 2^z in two's complement.
#pragma once
#include "ozaki_common.cuh"

namespace vcpcu {

constexpr int OZ_CRT_GROUPS = 6;

struct CrtBasis {
  uint32_t Q[OZ_CRT_GROUPS][4];  // Q_g 2^z, 32-bit limbs (0 past the last group)
  uint32_t N[4];                 // 2^128 - M 2^z
  uint32_t a[OZ_CRT_GROUPS][3];  // a_l of the group's moduli (0 past the last)
  uint32_t R;                    // round(2^159 / (M 2^z))
  int z, groups;
};

// ---- host: the basis of the first L moduli --------------------------------
inline unsigned oz_inv_mod(unsigned r, unsigned m) {  // r^-1 mod m, r and m coprime
  int t0 = 0, t1 = 1, r0 = (int)m, r1 = (int)(r % m);
  while (r1) {
    const int q = r0 / r1, t = t0 - q * t1, s = r0 - q * r1;
    t0 = t1;
    t1 = t;
    r0 = r1;
    r1 = s;
  }
  return (unsigned)(t0 < 0 ? t0 + (int)m : t0) % m;
}

inline void crt_basis(int L, CrtBasis* b) {
  memset(b, 0, sizeof(*b));
  unsigned __int128 M = 1;
  for (int l = 0; l < L; ++l) M *= (unsigned __int128)OZ_MODULI[l];
  int z = 0;
  while (!((M << z) >> 127)) ++z;
  b->z = z;
  b->groups = (L + 2) / 3;
  for (int g = 0; g < b->groups; ++g) {
    const int l0 = 3 * g, l1 = l0 + 3 < L ? l0 + 3 : L;
    uint64_t P = 1;
    for (int l = l0; l < l1; ++l) P *= (uint64_t)OZ_MODULI[l];
    const unsigned __int128 MP = M / P;
    uint64_t t = 0;
    for (int l = l0; l < l1; ++l) {
      const unsigned m = (unsigned)OZ_MODULI[l];
      const uint64_t a = P / m;
      const unsigned am = (unsigned)(a % m);
      // t mod m_l = a * (a^2 M/P)^-1 = (a M/P)^-1
      const unsigned inv = oz_inv_mod(am * am % m * (unsigned)(MP % m) % m, m);
      t += a * inv;
      b->a[g][l - l0] = (uint32_t)a;
    }
    const unsigned __int128 Q = (MP * (t % P)) << z;
    for (int i = 0; i < 4; ++i) b->Q[g][i] = (uint32_t)(Q >> (32 * i));
  }
  const unsigned __int128 Mz = M << z, N = -Mz;
  for (int i = 0; i < 4; ++i) b->N[i] = (uint32_t)(N >> (32 * i));
  // 2^159 / M' by long division: q0 = floor(2^128 / M') = 1 (M' > 2^127),
  // then 31 more bits and the rounding bit
  unsigned __int128 rem = N;  // 2^128 - M'
  uint64_t R = 1;
  for (int i = 0; i < 31; ++i) {
    const int top = (int)(rem >> 127);
    rem <<= 1;
    R <<= 1;
    if (top || rem >= Mz) {
      rem -= Mz;
      R |= 1;
    }
  }
  const int top = (int)(rem >> 127);
  if (top || (rem << 1) >= Mz) ++R;
  b->R = R > 0xffffffffULL ? 0xffffffffu : (uint32_t)R;
}

// ---- one entry -----------------------------------------------------------
OZ_HD uint32_t crt_mulhi(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
  return __umulhi(a, b);
#else
  return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}

// X 2^z (two's complement, four limbs) from the group values V_g.
OZ_HD void crt_reduce(const uint32_t (&V)[OZ_CRT_GROUPS], const CrtBasis& b, uint32_t (&r)[4]) {
  uint64_t s[4] = {0, 0, 0, 0};
#pragma unroll
  for (int g = 0; g < OZ_CRT_GROUPS; ++g) {
#pragma unroll
    for (int t = 0; t < 4; ++t) s[t] += (uint64_t)V[g] * b.Q[g][t];
  }
  const uint64_t T = s[3] + (s[2] >> 32);
  const uint64_t u = (T >> 32) * (uint64_t)b.R + crt_mulhi((uint32_t)T, b.R) + (1u << 30);
  const uint32_t q = (uint32_t)(u >> 31);
#pragma unroll
  for (int t = 0; t < 4; ++t) s[t] += (uint64_t)q * b.N[t];
  r[0] = (uint32_t)s[0];
  s[1] += s[0] >> 32;
  r[1] = (uint32_t)s[1];
  s[2] += s[1] >> 32;
  r[2] = (uint32_t)s[2];
  r[3] = (uint32_t)s[3] + (uint32_t)(s[2] >> 32);
}

// Magnitude and sign of a two's complement value of four limbs.
OZ_HD int crt_abs(uint32_t (&r)[4]) {
  const uint32_t neg = r[3] >> 31, mask = 0u - neg;
  uint64_t c = neg;
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    c += r[t] ^ mask;
    r[t] = (uint32_t)c;
    c >>= 32;
  }
  return (int)neg;
}

// RD and RU of mag 2^e for a magnitude of four limbs (+0 for zero); ehi =
// (e + 1149) << 20 and every nonzero result is a normal double.  The top 53
// bits are the truncated significand, any bit below makes RU one unit larger
// (a carry into the exponent field is the correct rounding).  No branch: the
// leading word is brought to the top by two selections -- products far below
// their row and column maxima (R [A] beside its diagonal) are as common as
// full-length ones.  Results as the (high, low) words of doubles.
OZ_HD void crt_to_dir(const uint32_t (&mag)[4], int ehi, uint32_t (&dn)[2], uint32_t (&up)[2]) {
  const bool s2 = (mag[3] | mag[2]) == 0;
  const uint32_t v3 = s2 ? mag[1] : mag[3], v2 = s2 ? mag[0] : mag[2], v1 = s2 ? 0u : mag[1],
                 v0 = s2 ? 0u : mag[0];
  const bool s1 = v3 == 0;
  const uint32_t w3 = s1 ? v2 : v3, w2 = s1 ? v1 : v2, w1 = s1 ? v0 : v1, w0 = s1 ? 0u : v0;
#ifdef __CUDA_ARCH__
  const int lz = __clz((int)w3);  // 32 for zero: shifts of 32 give 0 or the word itself
  const uint32_t t3 = __funnelshift_l(w2, w3, lz), t2 = __funnelshift_l(w1, w2, lz);
  const uint32_t lo = __funnelshift_r(t2, t3, 11), v = w1 << (lz & 31);
#else
  const int lz = w3 ? __builtin_clz(w3) : 0;
  const uint32_t t3 = lz ? (w3 << lz) | (w2 >> (32 - lz)) : w3;
  const uint32_t t2 = lz ? (w2 << lz) | (w1 >> (32 - lz)) : w2;
  const uint32_t lo = (t2 >> 11) | (t3 << 21), v = w1 << lz;
#endif
  const uint32_t below = (t2 & 0x7ffu) | v | w0;
  // the leading significand bit adds 1 to the exponent field
  const uint32_t shift = (uint32_t)(lz + (s2 ? 64 : 0) + (s1 ? 32 : 0));
  const uint32_t hi = (t3 >> 11) + (uint32_t)ehi - (shift << 20);
  const uint64_t u = (((uint64_t)hi << 32) | lo) + (below ? 1u : 0u);
  const uint32_t keep = w3 ? 0xffffffffu : 0u;
  dn[0] = hi & keep;
  dn[1] = lo & keep;
  up[0] = (uint32_t)(u >> 32) & keep;
  up[1] = (uint32_t)u & keep;
}

}  // namespace vcpcu
