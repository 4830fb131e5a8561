// FP64 multiply and divide on the integer pipe, rounded to nearest even.
//
// GB300 issues FP64 slowly: measured 0.5 T FMA/s, about 1.7 FP64 lane
// operations per clock and SM, while an SM issues up to four warp
// instructions per clock to its integer units.  IEEE binary64 operations on
// normal numbers can be computed exactly with 64-bit integer operations on the
// significands; a product of unpacked operands (below) takes about 20 integer
// instructions and 4 multiply-adds, which occupy the integer pipes for less
// time than the FP64 pipe needs for one operation.  The reference-rounding
// element kernels, whose every product and sum is a separately rounded FP64
// operation, run their products here and their sums on the FP64 pipe so that
// both pipes work at once.  The results are the IEEE round-to-nearest-even
// results bit for bit (checked against the host's FP64 on random and
// edge-case operands, and through the bit-exact element matrices).
//
// The algorithms follow the IEEE 754 definition of the operations: exact
// integer products / aligned sums of the 53-bit significands with guard and
// sticky bits, normalisation, round to nearest with ties to even.
//
// What the kernels use are the products and quotients of unpacked operands and
// mulhi.  The multiply and add of packed operands before them, for any operands
// (zeros, subnormals, infinities, NaN and results that would overflow or
// underflow return false), have no caller but their host check.
#pragma once

#include <cstdint>

#if defined(__CUDACC__)
#define AFEM_HD __host__ __device__ __forceinline__
#else
#define AFEM_HD inline
#endif

namespace afem {
namespace i64fp {

constexpr uint64_t kSign = 1ull << 63;
constexpr uint64_t kMant = (1ull << 52) - 1;
constexpr uint64_t kHidden = 1ull << 52;

AFEM_HD uint64_t mulhi(uint64_t a, uint64_t b) {
#if defined(__CUDA_ARCH__)
  return __umul64hi(a, b);
#else
  return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}

AFEM_HD int clz(uint64_t x) {
#if defined(__CUDA_ARCH__)
  return __clzll((long long)x);
#else
  return x ? __builtin_clzll(x) : 64;
#endif
}

// biased exponent in [1, 2046] (a normal number)
AFEM_HD bool normal(int e) { return (unsigned)(e - 1) < 0x7feu; }

// a * b.  The 53 x 53-bit significand product has 105 or 106 bits: with the
// first operand shifted left by 11, its high 64 bits are the top 53 or 54 bits
// and the low 64 bits hold the rest, left-aligned, for the rounding.
AFEM_HD bool mul(uint64_t ua, uint64_t ub, uint64_t* out) {
  const int ea = (int)((ua >> 52) & 0x7ff), eb = (int)((ub >> 52) & 0x7ff);
  if (!normal(ea) || !normal(eb)) return false;
  const uint64_t A = ((ua & kMant) | kHidden) << 11;
  const uint64_t B = (ub & kMant) | kHidden;
  const uint64_t hi = mulhi(A, B), lo = A * B;
  int e = ea + eb - 1023;
  uint64_t m, r;   // 53-bit significand and the bits below it, left-aligned
  if (hi >> 52) {
    m = hi;
    r = lo;
    e += 1;
  } else {
    m = (hi << 1) | (lo >> 63);
    r = lo << 1;
  }
  m += (r > kSign) | ((r == kSign) & (m & 1));   // nearest, ties to even
  if (m >> 53) {
    m >>= 1;
    e += 1;
  }
  if (!normal(e)) return false;
  *out = ((ua ^ ub) & kSign) | ((uint64_t)e << 52) | (m & kMant);
  return true;
}

// a + b.  Significands with their leading bit at bit 62 and 10 guard bits;
// the smaller is shifted right by the exponent difference with the bits it
// loses folded into a sticky bit.  A difference that cancels more than one
// bit only arises for exponent differences of 0 or 1, when no bit was lost,
// so the left normalisation is exact.
AFEM_HD bool add(uint64_t ua, uint64_t ub, uint64_t* out) {
  if ((ua & ~kSign) < (ub & ~kSign)) {
    const uint64_t t = ua;
    ua = ub;
    ub = t;
  }
  const int ea = (int)((ua >> 52) & 0x7ff), eb = (int)((ub >> 52) & 0x7ff);
  if (!normal(ea) || !normal(eb)) return false;
  const int d = ea - eb;
  const uint64_t ma = ((ua & kMant) | kHidden) << 10;
  uint64_t mb = ((ub & kMant) | kHidden) << 10;
  uint64_t sticky = 0;
  if (d >= 64) {
    sticky = 1;
    mb = 0;
  } else if (d > 0) {
    sticky = (mb << (64 - d)) != 0;
    mb >>= d;
  }
  uint64_t s;
  int e = ea;
  if (((ua ^ ub) & kSign) == 0) {
    s = ma + mb;
    if (s >> 63) {
      sticky |= s & 1;
      s >>= 1;
      e += 1;
    }
  } else {
    s = ma - mb - sticky;   // the exact difference lies in (s, s + 1) when sticky
    if (s == 0) {           // exact cancellation: +0 in round-to-nearest
      *out = 0;
      return true;
    }
    const int z = clz(s) - 1;
    s <<= z;
    e -= z;
  }
  uint64_t m = s >> 10;
  const uint64_t r = s & 0x3ff, half = 0x200;
  m += (r > half) | ((r == half) & ((sticky != 0) | (m & 1)));
  if (m >> 53) {
    m >>= 1;
    e += 1;
  }
  if (!normal(e)) return false;
  *out = (ua & kSign) | ((uint64_t)e << 52) | (m & kMant);
  return true;
}

// ---------------------------------------------------------------------------
// Products of operands that take part in several: each operand is unpacked
// once (Operand), and a product is then about 20 integer instructions and four
// 32 x 32 -> 64 multiply-adds, without a branch or a range test.  The caller
// sees to the range: zeros and normal numbers, and products that are an exact
// zero or normal.  in_window<W> tests for zero or an exponent within +-W; the
// products of three numbers within +-kWindow stay normal (3 kWindow < 1022).

constexpr int kWindow = 250;

// The significand with its hidden bit at bit 62 - 32 of hi (52 + 10 = 62 of
// the pair), 0 for a zero; sign and exponent in place in se.
struct Operand {
  uint32_t lo, hi, se;
};

AFEM_HD Operand operand(uint32_t h, uint32_t l) {
  const uint32_t m = (h & 0xfffffu) | ((h & 0x7ff00000u) ? 0x100000u : 0u);
  return {l << 10, (m << 10) | (l >> 22), h & 0xfff00000u};
}

// zero, or an exponent within 1023 +- W
template <int W = kWindow>
AFEM_HD bool in_window(uint32_t h, uint32_t l) {
  const uint32_t e = (h & 0x7fffffffu) - ((1023u - W) << 20);
  return e < ((2u * W + 1u) << 20) || ((h << 1) | l) == 0;
}

AFEM_HD Operand operand(uint64_t u) { return operand((uint32_t)(u >> 32), (uint32_t)u); }
AFEM_HD bool in_window(uint64_t u) { return in_window((uint32_t)(u >> 32), (uint32_t)u); }

// a * b rounded to nearest even.  The product of the two 62-bit-aligned
// significands has its leading bit at 125 or 124: its high 64 bits hold the
// 53 of the result at 61..9 (one place lower for a small product) and the
// rounding bits below, the low 64 bits only their sticky part.  Adding 0xff,
// and one more if the result is odd or the sticky part is not zero, carries
// into bit 9 exactly when the result rounds up.  The exponents' fields add in
// place, and so do the signs (bit 31 wraps).
AFEM_HD uint64_t mul(const Operand& a, const Operand& b) {
  const uint64_t p00 = (uint64_t)a.lo * b.lo;
  uint64_t mid = (uint64_t)a.lo * b.hi + (p00 >> 32);   // hi < 2^31: the sums stay below 2^64
  mid += (uint64_t)a.hi * b.lo;
  const uint64_t top = (uint64_t)a.hi * b.hi + (mid >> 32);
  uint32_t hi = (uint32_t)(top >> 32), lo = (uint32_t)top;
  const uint32_t rest = (uint32_t)p00 | (uint32_t)mid;
  const uint32_t sticky = rest < 1u ? rest : 1u;
  const bool small = hi < 0x20000000u;
  uint32_t se = a.se + b.se - (small ? 1024u << 20 : 1023u << 20);   // one less: the hidden bit below adds it
  if (hi == 0) se = (a.se ^ b.se) & 0x80000000u;                     // a zero operand
  if (small) {
    hi = (hi << 1) | (lo >> 31);
    lo <<= 1;
  }
  const uint64_t r = (((uint64_t)hi << 32) | lo) + (0xffu + (((lo >> 9) & 1u) | sticky));
  return ((uint64_t)(se + (uint32_t)(r >> 41)) << 32) | (uint32_t)(r >> 9);
}

// ---------------------------------------------------------------------------
// Quotients by a divisor that several dividends share.  recip is 2^127 / (d
// 2^11) from below (d the 53-bit significand), so that the high word of its
// product with a dividend's significand is the quotient to about 60 bits, from
// below; one exact remainder then settles the 54-bit floor, and its last bit
// the rounding (a quotient of two 53-bit significands is never a tie).

struct Divisor {
  uint64_t d, recip;
  uint32_t se;
};

// u: a normal number.  The reciprocal starts from an FP32 one, lowered by more
// than its error, and takes two Newton steps; from below they stay below.
AFEM_HD Divisor divisor(uint64_t u) {
  Divisor r;
  r.d = (u & kMant) | kHidden;
  r.se = (uint32_t)(u >> 32) & 0xfff00000u;
  const uint64_t dn = r.d << 11;
#if defined(__CUDA_ARCH__)
  const float f = __frcp_rn((float)(uint32_t)(dn >> 40)) * 0x1.ffffep54f;   // 2^55 (1 - 2^-20)
#else
  const float f = (1.0f / (float)(uint32_t)(dn >> 40)) * 0x1.ffffep54f;
#endif
  uint64_t v = (uint64_t)(uint32_t)f << 32;
  v += mulhi(v, (1ull << 63) - mulhi(v, dn) - 1) << 1;
  v += mulhi(v, (1ull << 63) - mulhi(v, dn) - 1) << 1;
  r.recip = v;
  return r;
}

// n / d rounded to nearest, for n in the range of in_window (0 / d is the
// signed zero).
AFEM_HD uint64_t div(const Operand& n, const Divisor& d) {
  const uint32_t rl = (uint32_t)d.recip, rh = (uint32_t)(d.recip >> 32);
  // n / d 2^62, a few units low: the cross products' low words and n.lo rl are left out
  uint64_t t = (uint64_t)n.hi * rh + (((uint64_t)n.lo * rh) >> 32);
  t += ((uint64_t)n.hi * rl) >> 32;
  const bool big = (t >> 62) != 0;   // n >= d
  const uint64_t q = (t >> (big ? 9 : 8)) + 1;   // the floor of n 2^53 / d (n 2^54 / d), or one more
  const uint64_t rem = ((uint64_t)(n.lo << (big ? 11 : 12)) << 32) - q * d.d;
  const uint64_t m = (q + ((int64_t)rem >= 0 ? 1 : 0)) >> 1;
  uint32_t se = n.se - d.se + (big ? 1022u << 20 : 1021u << 20);   // one less: the hidden bit adds it
  if (n.hi == 0) se = (n.se ^ d.se) & 0x80000000u;
  const uint32_t mh = n.hi == 0 ? 0u : (uint32_t)(m >> 32), ml = n.hi == 0 ? 0u : (uint32_t)m;
  return ((uint64_t)(se + mh) << 32) | ml;
}

}  // namespace i64fp
}  // namespace afem
