// ozaki_dd.cuh -- per-entry integer arithmetic of the dd product (host- and
// device-callable, so that the CPU tests run the very code of the kernels):
// the w-bit integer of a dd entry, the Chinese remaindering of up to 32
// residues in 256 bits, and the dd value of the result.
#pragma once
#include "ozaki_common.cuh"
#include "ozaki_crt.cuh"
#include "ozaki_prep.cuh"

namespace vcpcu {

// The exponent of a line from the encoded one of its largest |a1|: one bit of
// headroom, so that |a1 + a2| <= 2^(E-1).
OZ_HD int dd_line_exp(uint32_t c) {
  const int E = exp_dec(c);
  return E == OZ_ZERO_EXP ? E : E + 1;
}

// RN(x 2^(w - E)) of a finite double as a signed 128-bit integer in four
// words added to (a), |x| <= 2^(E-1), w <= 127: the significand shifted left,
// or right with ties to even.
OZ_HD void dd_add_int(double x, int E, int w, __int128& a) {
  const uint64_t b = oz_bits(x);
  const int f = (int)((b >> 52) & 0x7ff);
  const uint64_t m = b & ((1ULL << 52) - 1);
  const uint64_t M = f ? m | (1ULL << 52) : m;
  const int s = (f ? f : 1) - 1075 + w - E;
  unsigned __int128 N;
  if (s >= 0) {
    N = (unsigned __int128)M << s;
  } else {
    const int r = -s < 60 ? -s : 60;  // (M < 2^53: from 55 on the result is 0)
    N = (M + ((1ULL << (r - 1)) - 1) + ((M >> r) & 1)) >> r;
  }
  a += (b >> 63) ? -(__int128)N : (__int128)N;
}

// ---- Chinese remaindering of L <= 32 residues ------------------------------
// As ozaki_crt.cuh with eleven groups of three and eight limbs.  The plan's
// moduli give |X| < M / 2 only, so the quotient may be off by one where X is
// near +-M / 2: M is shifted to M' in [2^253, 2^254), the two spare bits keep
// S' - q M' a 256-bit two's complement value, and it is brought back into
// (-M' / 2, M' / 2] by one exact comparison where its top word says that this
// can be needed.
constexpr int DDL = 8, DD_GROUPS = 11;

struct DdBasis {
  uint32_t Q[DD_GROUPS][DDL];  // Q_g 2^z
  uint32_t N[DDL];             // 2^256 - M 2^z
  uint32_t M[DDL];             // M 2^z
  uint32_t H[DDL];             // M 2^(z-1)
  uint32_t a[DD_GROUPS][3];
  uint32_t R;                  // round(2^285 / (M 2^z)), in [2^31, 2^32]
  int z, groups;
};

// Host: the basis of the first L moduli.
inline void dd_basis(int L, DdBasis* b) {
  memset(b, 0, sizeof(*b));
  auto mul = [](uint32_t* x, uint32_t f) {
    uint64_t c = 0;
    for (int t = 0; t < DDL; ++t) {
      c += (uint64_t)x[t] * f;
      x[t] = (uint32_t)c;
      c >>= 32;
    }
  };
  auto div = [](const uint32_t* x, uint32_t d, uint32_t* q) {
    uint64_t r = 0;
    for (int t = DDL - 1; t >= 0; --t) {
      r = (r << 32) | x[t];
      q[t] = (uint32_t)(r / d);
      r %= d;
    }
    return (uint32_t)r;
  };
  uint32_t M[DDL] = {1};
  for (int l = 0; l < L; ++l) mul(M, (uint32_t)OZ_MODULI[l]);
  auto shifted = [&](const uint32_t* x, int z, uint32_t* out) {
    memset(out, 0, sizeof(uint32_t) * DDL);
    for (int t = 0; t < DDL; ++t) {
      const int o = t + (z >> 5);
      const uint64_t v = (uint64_t)x[t] << (z & 31);
      if (o < DDL) out[o] |= (uint32_t)v;
      if (o + 1 < DDL) out[o + 1] |= (uint32_t)(v >> 32);
    }
  };
  int top = 32 * DDL - 1;
  while (!((M[top >> 5] >> (top & 31)) & 1)) --top;
  b->z = 253 - top;
  b->groups = (L + 2) / 3;
  for (int g = 0; g < b->groups; ++g) {
    const int l0 = 3 * g, l1 = l0 + 3 < L ? l0 + 3 : L;
    uint32_t P = 1, MP[DDL], q[DDL];
    memcpy(MP, M, sizeof(MP));
    for (int l = l0; l < l1; ++l) {
      P *= (uint32_t)OZ_MODULI[l];
      div(MP, (uint32_t)OZ_MODULI[l], q);
      memcpy(MP, q, sizeof(MP));
    }
    uint64_t t = 0;
    for (int l = l0; l < l1; ++l) {
      const uint32_t m = (uint32_t)OZ_MODULI[l];
      const uint64_t a = P / m;
      const uint32_t am = (uint32_t)(a % m), mp = div(MP, m, q);
      t += a * oz_inv_mod(am * am % m * mp % m, m);
      b->a[g][l - l0] = (uint32_t)a;
    }
    mul(MP, (uint32_t)(t % P));
    shifted(MP, b->z, b->Q[g]);
  }
  shifted(M, b->z, b->M);
  if (b->z > 0)
    shifted(M, b->z - 1, b->H);
  else
    for (int t = 0; t < DDL; ++t)
      b->H[t] = (b->M[t] >> 1) | (t + 1 < DDL ? b->M[t + 1] << 31 : 0u);
  uint64_t c = 1;
  for (int t = 0; t < DDL; ++t) {
    c += (uint32_t)~b->M[t];
    b->N[t] = (uint32_t)c;
    c >>= 32;
  }
  // 2^285 / M' = 2^93 / (M' / 2^192), M' / 2^192 in [2^61, 2^62): its top 64 bits
  // determine the quotient to better than a unit
  const uint64_t Mt = ((uint64_t)b->M[7] << 32) | b->M[6];
  const unsigned __int128 num = (unsigned __int128)1 << 93;
  const uint64_t R = (uint64_t)((num + Mt / 2) / Mt);
  b->R = R > 0xffffffffULL ? 0xffffffffu : (uint32_t)R;
}

// X 2^z (two's complement) from the group values.  S' / M' < 2^29; T = the top
// of S' in units 2^224 (below 2^59), q = round(T R 2^-61).
OZ_HD void dd_reduce(const uint32_t (&V)[DD_GROUPS], const DdBasis& b, uint32_t (&r)[DDL]) {
  uint64_t s[DDL];
#pragma unroll
  for (int t = 0; t < DDL; ++t) s[t] = 0;
#pragma unroll
  for (int g = 0; g < DD_GROUPS; ++g) {
    if (g >= b.groups) break;
#pragma unroll
    for (int t = 0; t < DDL; ++t) s[t] += (uint64_t)V[g] * b.Q[g][t];
  }
  const uint64_t T = s[7] + (s[6] >> 32);
  const uint64_t u = (T >> 32) * (uint64_t)b.R + crt_mulhi((uint32_t)T, b.R) + (1u << 28);
  const uint32_t q = (uint32_t)(u >> 29);
  uint64_t c = 0;
#pragma unroll
  for (int t = 0; t < DDL; ++t) {
    s[t] += (uint64_t)q * b.N[t] + c;
    r[t] = (uint32_t)s[t];
    c = s[t] >> 32;
  }
}

// Magnitude and sign of X 2^z from dd_reduce's value: r or, past M' / 2, the
// other representative.
OZ_HD bool dd_abs(uint32_t (&r)[DDL], const DdBasis& b) {
  bool neg = (r[7] >> 31) != 0;
  {
    const uint32_t mask = neg ? 0xffffffffu : 0u;
    uint64_t c = neg ? 1 : 0;
#pragma unroll
    for (int t = 0; t < DDL; ++t) {
      c += r[t] ^ mask;
      r[t] = (uint32_t)c;
      c >>= 32;
    }
  }
  if (r[7] >= b.H[7]) {
    uint64_t borrow = 0;
#pragma unroll
    for (int t = 0; t < DDL; ++t) borrow = ((uint64_t)b.H[t] - r[t] - borrow) >> 63;
    if (borrow) {  // r > H: M' - r, the other sign
      uint64_t c = 0;
#pragma unroll
      for (int t = 0; t < DDL; ++t) {
        const uint64_t v = (uint64_t)b.M[t] - r[t] - c;
        r[t] = (uint32_t)v;
        c = v >> 63;
      }
      neg = !neg;
    }
  }
  return neg;
}

// The dd value of mag 2^ex: hi = RN(mag), lo = RN(mag - hi) as significands and
// exponents: value Mh 2^(eh) with Mh in [2^52, 2^53] (0 for zero), lo the
// same, negative with lneg.  bl: bit length of mag, lbl: of |mag - hi| (0:
// zero).  False: the remainder's leading bit is too far down for the words at
// hand (the caller takes the general path).
struct DdWords {
  uint64_t Mh, Ml;
  int eh, el, bl, lbl;
  bool lneg;
};

OZ_HD uint32_t dd_shl(uint32_t lo, uint32_t hi, int n) {  // high word of (hi : lo) << n, n < 32
#ifdef __CUDA_ARCH__
  return __funnelshift_l(lo, hi, n);
#else
  return n ? (hi << n) | (lo >> (32 - n)) : hi;
#endif
}

// RN of a 64-bit value (top bit set) and a sticky flag for what lies below, to
// 53 bits; the rounded-up bit in *up.
OZ_HD uint64_t dd_rn53(uint64_t t, bool below, bool* up) {
  const uint32_t rem = (uint32_t)t & 0x7ffu;
  uint64_t M = t >> 11;
  *up = rem > 0x400u || (rem == 0x400u && (below || (M & 1)));
  return M + (*up ? 1 : 0);
}

OZ_HD bool dd_words(const uint32_t (&r)[DDL], DdWords* w) {
  // the leading word to the top by selections
  uint32_t v[DDL];
  int off = 0;
  {
    const bool z = (r[7] | r[6] | r[5] | r[4]) == 0;
    off += z ? 128 : 0;
#pragma unroll
    for (int t = 0; t < DDL; ++t) v[t] = z ? (t >= 4 ? r[t >= 4 ? t - 4 : 0] : 0u) : r[t];
  }
  {
    const bool z = (v[7] | v[6]) == 0;
    off += z ? 64 : 0;
#pragma unroll
    for (int t = DDL - 1; t >= 0; --t) v[t] = z ? (t >= 2 ? v[t >= 2 ? t - 2 : 0] : 0u) : v[t];
  }
  {
    const bool z = v[7] == 0;
    off += z ? 32 : 0;
#pragma unroll
    for (int t = DDL - 1; t >= 0; --t) v[t] = z ? (t >= 1 ? v[t >= 1 ? t - 1 : 0] : 0u) : v[t];
  }
  w->Mh = w->Ml = 0;
  w->eh = w->el = 0;
  w->bl = w->lbl = 0;
  w->lneg = false;
  if (v[7] == 0) return true;  // zero
  const int lz = iv_clz(v[7]);
  off += lz;
  w->bl = 256 - off;
  const uint32_t W7 = dd_shl(v[6], v[7], lz), W6 = dd_shl(v[5], v[6], lz),
                 W5 = dd_shl(v[4], v[5], lz), W4 = dd_shl(v[3], v[4], lz),
                 W3 = dd_shl(v[2], v[3], lz);
  const bool rest = ((v[2] << lz) | v[1] | v[0]) != 0;  // below the 160 bits
  const uint64_t t = ((uint64_t)W7 << 32) | W6;
  bool up;
  w->Mh = dd_rn53(t, (W5 | W4 | W3) != 0 || rest, &up);
  w->eh = 203 - off;  // W7's top bit weighs 2^(255 - off)
  // the remainder in units of W3's last bit, 107 bits: rem : W5 : W4 : W3, or
  // its complement below the next significand
  const uint32_t m = up ? 0xffffffffu : 0u;
  uint32_t y[4] = {W3 ^ m, W4 ^ m, W5 ^ m, (W6 ^ m) & 0x7ffu};
  if (up && !rest) {
    uint64_t c = 1;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      c += y[q];
      y[q] = (uint32_t)c;
      c >>= 32;
    }
  }
  w->lneg = up;
  int yoff = 0;
  if (y[3] == 0) {
    yoff = 32;
    y[3] = y[2];
    y[2] = y[1];
    y[1] = y[0];
    y[0] = 0;
  }
  if (y[3] == 0) return !(y[2] | y[1] | (rest ? 1u : 0u));  // zero, or too far down
  const int yz = iv_clz(y[3]);
  const uint64_t yt = ((uint64_t)dd_shl(y[2], y[3], yz) << 32) | dd_shl(y[1], y[2], yz);
  bool up2;
  w->Ml = dd_rn53(yt, ((y[1] << yz) | y[0]) != 0 || rest, &up2);
  // y[3]'s bit 31 weighs 2^127 of W3's last bit 2^(96 - off)
  const int last = 96 - off;
  w->lbl = last + 128 - yoff - yz;
  w->el = w->lbl - 53;
  return true;
}

}  // namespace vcpcu
