// ecp_fixed.h -- 64-bit integer-mantissa arithmetic of the batched path.
//
// GB300's FP64 pipe takes one warp instruction per 16 to 19 cycles and SM,
// whatever the number of active lanes, and holds a warp for 64 cycles per
// dependent operation; the integer pipes take one warp instruction per cycle
// and SM quarter at 4 to 6 cycles of latency.  The tabulations of the batched
// kernels (Bessel rows, exponentials, powers, prefactors) therefore run on
// the integer pipes with 64-bit mantissas -- eleven bits more than FP64 -- and
// round once, to double, where a table entry is written.
//
// Two forms:
//   xf        an unsigned 64-bit mantissa and a binary exponent, value m * 2^e.
//             Products keep the high 64 bits (mul_hi, below 3 units short) and
//             are not renormalised, so a product loses at most one leading
//             bit; norm1() wins one back.
//   fixed     a signed 64-bit integer at a scale the context knows (Horner
//             passes, exponents in Q53).
// Everything here is integer arithmetic (one float reciprocal seeds fx_recip
// on either side), so host and device agree bit for bit; tests/test_fixed.py
// measures the errors on the host against 200-bit arithmetic.
#pragma once
#include <cstdint>
#include <cstring>

#include "ecp_fastmath.h"

namespace ecpgb {

#ifdef __CUDA_ARCH__
#define ECPGB_NOUNROLL _Pragma("unroll 1")
#else
#define ECPGB_NOUNROLL
#endif

using u64 = unsigned long long;
using i64 = long long;

struct xf {
  u64 m;
  int e;
};

ECPGB_HD int clz64(u64 v) {
#ifdef __CUDA_ARCH__
  return __clzll((i64)v);
#else
  return v ? __builtin_clzll(v) : 64;
#endif
}

// High 64 bits of a * b, up to 2 units below the exact value: three 32-bit
// products instead of four.
ECPGB_HD u64 mul_hi(u64 a, u64 b) {
  const uint32_t a0 = (uint32_t)a, a1 = (uint32_t)(a >> 32), b0 = (uint32_t)b, b1 = (uint32_t)(b >> 32);
  return (u64)a1 * b1 + (((u64)a1 * b0) >> 32) + (((u64)a0 * b1) >> 32);
}

// A multiplier 0 <= x < 2^63 split for mul_hi_s: high word, signed low word.
struct fxmul {
  int hi, lo;
};
ECPGB_HD fxmul fx_split(u64 x) {
  const int lo = (int)(uint32_t)x;
  return {(int)(uint32_t)(x >> 32) - (lo >> 31), lo};
}
// v * x / 2^64 for signed v and a split x, within 2 units: the low word of x
// is taken signed so that every 32-bit product has one kind of operands.
ECPGB_HD i64 mul_hi_s(i64 v, fxmul x) {
  const int v1 = (int)(v >> 32);
  const uint32_t v0 = (uint32_t)v;
  return (i64)v1 * x.hi + (i64)(((u64)v0 * (uint32_t)x.hi) >> 32) + (((i64)v1 * x.lo) >> 32);
}

// A finite non-negative double (a subnormal counts as 0); the sign is ignored.
ECPGB_HD xf xf_from(double x) {
  const u64 b = (u64)dbits(x);
  const int be = (int)(b >> 52) & 0x7ff;
  return {be ? (b << 11) | (1ull << 63) : 0ull, be - (1023 + 63)};
}
// The sign bit of a double, in the high word's position.
ECPGB_HD uint32_t sign_of(double x) { return (uint32_t)((u64)dbits(x) >> 32) & 0x80000000u; }

ECPGB_HD xf xf_mul(xf a, xf b) { return {mul_hi(a.m, b.m), a.e + b.e + 64}; }
// Wins back the leading bit a product of normalised mantissas may have lost.
ECPGB_HD xf norm1(xf a) {
  if ((i64)a.m >= 0) {
    a.m += a.m;
    a.e -= 1;
  }
  return a;
}

// Leading bit to the top (a zero stays zero).
ECPGB_HD xf xf_norm(xf a) {
  const int lz = clz64(a.m | 1u);
  return {a.m << lz, a.e - lz};
}

// m * 2^e rounded to the nearest double, with a sign; 0 below the normal range,
// infinity above it.
ECPGB_HD double xf_to_double(u64 m, int e, uint32_t sign) {
  const int lz = clz64(m);
  int be = e + 63 + 1023 - lz;  // biased exponent
  m <<= (lz & 63);
  if (be >= 0x7ff) {
    be = 0x7ff;
    m = 0;
  }
  const u64 b = ((u64)(uint32_t)be << 52) + ((m << 1) >> 12) + ((m >> 10) & 1u);
  return lz < 64 && be > 0 ? bits_d((i64)(b | (u64)sign << 32)) : 0.0;
}

// v >> s for s >= 0 (0 from 64 on).
ECPGB_HD u64 shr64(u64 v, int s) { return s > 63 ? 0ull : v >> s; }

#ifdef __CUDACC__
static __device__ const u64 kExp2Fixed[ECPGB_EXP2_N] = ECPGB_EXP2_TABLE62;
#endif
static const u64 kExp2FixedHost[ECPGB_EXP2_N] = ECPGB_EXP2_TABLE62;

// exp(E / 2^53) for |E| < 2^63 (arguments within +-1023): Tang's table method
// as in fast_exp, in fixed point.  n = floor of E * 512/ln2 (up to 1/64 below
// the exact quotient: r then ends slightly above ln2/512), r = E - n ln2/512
// in Q62 from a 94-bit ln2/512, exp(r) to degree 5 with each term in as many
// bits as its weight needs, times 2^(j/512) with 62 bits.  Error below 2^-58
// of the result.
ECPGB_HD xf fx_exp(i64 E) {
  const int Eh = (int)(E >> 32);  // Q21
  // 512/ln2 in Q20; the bias (1/128 of a step) covers its error and Eh's
  const i64 prod = (i64)Eh * 774541002 - (1ll << 34);
  const int n = (int)(prod >> 41);
  const i64 nl = n;
  u64 r = ((u64)E << 9) - (u64)nl * ECPGB_LN2_512_Q62 - (u64)((nl * (i64)ECPGB_LN2_512_Q94LO) >> 32);
  const u64 X = r << 11;  // r * 2^9 in Q64, r < 2^-9.5
  const uint32_t X32 = (uint32_t)(X >> 32);
  const uint32_t u4 = 178956971u + (uint32_t)(((u64)X32 * 69905u) >> 32);          // 1/24 + r/120, Q32
  const uint32_t u3 = 715827883u + ((uint32_t)(((u64)X32 * u4) >> 32) >> 9);       // 1/6 + r u4, Q32
  const u64 u2 = (1ull << 63) + (((u64)X32 * u3) >> 9);                            // 1/2 + r u3, Q64
  const u64 u1 = (1ull << 63) + (mul_hi(X, u2) >> 10);                             // 1 + r u2, Q63
  const u64 p = mul_hi(X, u1) >> 8;                                                // exp(r) - 1, Q64
#ifdef __CUDA_ARCH__
  const u64 s = __ldg(&kExp2Fixed[n & (ECPGB_EXP2_N - 1)]);
#else
  const u64 s = kExp2FixedHost[n & (ECPGB_EXP2_N - 1)];
#endif
  return {s + mul_hi(s, p), (n >> ECPGB_EXP2_LOG2N) - 62};
}

// 1/x for a mantissa x in [2^63, 2^64): 2^126 / x within 2^-60 of it, by two
// Newton steps from a float reciprocal.
ECPGB_HD u64 fx_recip(u64 x) {
  const float f = (float)(uint32_t)(x >> 40) * 0x1p-23f;
#ifdef __CUDA_ARCH__
  const float g = __frcp_rn(f);
#else
  const float g = 1.0f / f;
#endif
  const u64 y0 = (u64)(uint32_t)(g * 0x1p31f);  // Q31, 23 bits
  // t = x y0 in Q62, d = 1 - t
  const u64 t0 = (x >> 32) * y0 + (((x & 0xffffffffull) * y0) >> 32);
  const i64 d0 = (i64)((1ull << 62) - t0);  // Q62, about 40 bits
  u64 y = (y0 << 32) + (u64)(((i64)y0 * (d0 >> 8)) >> 22);
  const i64 d1 = (i64)((1ull << 62) - mul_hi(x, y));  // Q62, about 18 bits
  y += (u64)(((i64)(y >> 32) * d1) >> 30);
  return y;  // Q63
}

// Table reads: 16 bytes (the rows are 16-byte aligned) and 8 bytes.
struct fxpair {
  i64 x, y;
};
ECPGB_HD fxpair ld_pair(const i64 *p) {
#ifdef __CUDA_ARCH__
  const longlong2 v = __ldg((const longlong2 *)p);
  return {v.x, v.y};
#else
  return {p[0], p[1]};
#endif
}
ECPGB_HD i64 ld_one(const i64 *p) {
#ifdef __CUDA_ARCH__
  return __ldg(p);
#else
  return *p;
#endif
}

// Octaves of z tabulated below 1/200, down to 1e-60; what is smaller counts as 0.
constexpr int kBesselOctaves = 192;

// 100 z for z = f * r, f already times 100 (xf_times100): the argument of fx_bessel_rows.
ECPGB_HD xf xf_times100(xf f) { return {mul_hi(f.m, 100ull << 57), f.e + 7}; }

// K_0..K_lmax(z) in fixed point: row(l, v, scale) gets K_l / c = v 2^-scale,
// 0 <= v < 2^62, and the call returns c (1, or 1/(2z) for large z).  z100 =
// 100 z (the reference's table step is 1/100).  The branches of
// src/bessel.c:102-199: the 5-term Taylor polynomial about the nearest table
// point (z < 16) and the large-argument polynomial are both one Horner pass
// per row over 64-bit coefficients (besX, besXA), so lanes on either branch
// run the same instructions.  The first table point's polynomial, z < 1/200, is
// tabulated once per octave of z, each row at the octave's scale: K_l falls as z^l,
// and at one scale l = 3 had 10 bits left at z = 1e-6.  (The reference's branch for
// z < 1e-7 is that polynomial's first two terms.)  z = 0 gives exactly 1, 0, 0, ...
// kLate: a row is handed out while the next one's coefficients are on their way
// (the small grid, whose warps wait for them; in the large grid the second copy of
// `row` costs more in instruction fetch than it hides).
template <bool kLate = false, class Row>
ECPGB_HD xf fx_bessel(const i64 *besX, const i64 *besXA, int HL1, int lmax, xf z100, Row row) {
  z100 = xf_norm(z100);
  const int sh = -(z100.e + 52);  // 100 z in Q52 = z100.m >> sh; sh < 0 only above 1600
  const u64 W = sh < 0 ? ~0ull : shr64(z100.m, sh);
  const bool asy = W >= 1600ull << 52;
  const i64 *q = besX;
  int rowStride = 8, scaleAt = 6;
  u64 X;
  xf c = {1ull << 63, -63};
  if (asy) {
    c.m = mul_hi(fx_recip(z100.m), 50ull << 58);  // 1/(2z) = 50 / z100
    c.e = -120 - z100.e;
    const int s = c.e + 68;  // 16 / (2z) in Q64
    X = s > 0 ? c.m << 1 : shr64(c.m, -s);
    X = X < (1ull << 63) - 1 ? X : (1ull << 63) - 1;
    q = besXA;
    rowStride = 16;
    scaleAt = 15;
  } else {
    int i = (int)((W + (1ull << 51)) >> 52);
    if (i == 0) {
      X = z100.m & ((1ull << 63) - 1);
      i = -65 - z100.e;  // octaves below 1/2
      i = 1601 + (z100.m && i < kBesselOctaves ? i : kBesselOctaves);
    } else {
      X = sh < 11 ? z100.m << (11 - sh) : z100.m >> (sh - 11);  // 100 z / 2 in Q64
      X = (X + (1ull << 62)) & ((1ull << 63) - 1);
    }
    q += (size_t)i * HL1 * 8;
  }
  const fxmul x = fx_split(X);
  u64 vp = 0;
  int sp = 0;
ECPGB_NOUNROLL
  for (int l = 0; l <= lmax; l++, q += rowStride) {
    const fxpair c45 = ld_pair(q + 4), c23 = ld_pair(q + 2), c01 = ld_pair(q);
    const int sc = (int)ld_one(q + scaleAt);
    if (kLate && l) row(l - 1, vp, sp);
    i64 v = 0;
ECPGB_NOUNROLL
    for (int k = asy ? l : 5; k > 5; k--) v = ld_one(q + k) + mul_hi_s(v, x);
    v = c45.y + mul_hi_s(v, x);
    v = c45.x + mul_hi_s(v, x);
    v = c23.y + mul_hi_s(v, x);
    v = c23.x + mul_hi_s(v, x);
    v = c01.y + mul_hi_s(v, x);
    v = c01.x + mul_hi_s(v, x);
    vp = (u64)(v > 0 ? v : 0);
    sp = sc;
    if (!kLate) row(l, vp, sp);
  }
  if (kLate) row(lmax, vp, sp);
  return c;
}

// The rows packed one word each for the type-1 tables: a mantissa of 58 bits (2^63
// <= m < 2^64, 0 for a row that is 0) with the row's exponent in the low 6 bits, as
// K_l / c = m 2^(e0 - l t - low bits).  2^t is z's size below 1 (z 2^t in 0.3 to 2.6):
// then K_l 2^(l t) <= K_0, and no less than 2^-42 of it for l <= 8.  One exponent for
// all rows cut l = 8 to 47 bits at z = 2 and to none below 0.01.
struct RowBase {
  xf c;
  int e0, t;
};
template <bool kLate = false>
ECPGB_HD RowBase fx_bessel_packed(const i64 *besX, const i64 *besXA, int HL1, int lmax, xf z100, u64 *K) {
  RowBase b;
  b.t = z100.e < -56 ? (z100.e > -183 ? -56 - z100.e : 127) : 0;  // (a byte of the entry)
  int e0 = 0, lt = 0;
  b.c = fx_bessel<kLate>(besX, besXA, HL1, lmax, z100, [&](int l, u64 v, int scale) {
    const int n = clz64(v | 1u), e = -scale - n;
    if (l == 0) e0 = e;
    const int d = e0 - lt - e;  // (above 63: 0, and a row's cut series near its root)
    K[l] = (unsigned)d > 63u ? 63ull : ((v << n) & ~63ull) | (u64)(unsigned)d;
    lt += b.t;
  });
  b.e0 = e0;
  return b;
}
// Mantissa and exponent (over c and e0 - l t) of a packed row.
ECPGB_HD xf row_packed(u64 k) { return {k & ~63ull, -(int)(k & 63u)}; }

// The rows as doubles, each times mul (mul.m = 0: times 1) with the sign bit `sign`.
ECPGB_HD void fx_bessel_rows(const i64 *besX, const i64 *besXA, int HL1, int lmax, xf z100, xf mul, uint32_t sign,
                             double *K) {
  xf k[16];
  xf c = fx_bessel(besX, besXA, HL1, lmax, z100, [&](int l, u64 v, int scale) { k[l] = xf_norm({v, -scale}); });
  if (mul.m) c = xf_norm(xf_mul(c, mul));
  const bool one = c.m == 1ull << 63;  // a power of two: exact
ECPGB_NOUNROLL
  for (int l = 0; l <= lmax; l++) {
    const xf v = one ? xf{k[l].m, k[l].e + c.e + 63} : xf_mul(k[l], c);
    K[l] = xf_to_double(v.m, v.e, sign);
  }
}

// x in Q53 (fixed point) for |x| < 1023; saturates beyond.
ECPGB_HD i64 fx_q53(double x) {
  const u64 b = (u64)dbits(x);
  const int e = (int)(b >> 52) & 0x7ff;
  const u64 m = (b & ((1ull << 52) - 1)) | (1ull << 52);
  const int sh = e - 1022;  // value = m 2^(e - 1075)
  const i64 v = sh > 10 ? 0x7fe0000000000000ll : sh >= 0 ? (i64)(m << sh) : (i64)shr64(m, -sh);
  return (i64)b < 0 ? -v : v;
}

// z d^2 in Q53 (z > 0), saturating at 2^62.
ECPGB_HD u64 fx_gauss(double z, double d) {
  const xf D = xf_from(d), v = xf_mul(xf_from(z), xf_mul(D, D));
  const u64 E = shr64(v.m, -(v.e + 53));  // v.m >= 2^61 or 0
  return v.e + 53 <= 0 && E < 1ull << 62 ? E : 1ull << 62;
}

// A signed number m * 2^e, |m| < 2^62: the running values of a quadrature.
// Sums align to the larger exponent and are never renormalised upwards
// (cancelled bits stay cancelled); an empty sum has the smallest exponent.
struct xs {
  i64 m = 0;
  int e = -100000;
};
// Back below 2^62 after a sum.
ECPGB_HD xs xs_fit(xs a) {
  const int over = (int)((uint32_t)((u64)(a.m ^ (a.m << 1)) >> 63));
  return {a.m >> over, a.e + over};
}
ECPGB_HD xs xs_add(xs a, xs b) {
  const int d = a.e - b.e;
  const int sa = d < 0 ? (d < -63 ? 63 : -d) : 0, sb = d > 0 ? (d > 63 ? 63 : d) : 0;
  return xs_fit({(a.m >> sa) + (b.m >> sb), d < 0 ? b.e : a.e});
}
ECPGB_HD xs xs_neg(xs a) { return {-a.m, a.e}; }
ECPGB_HD xs xs_shl(xs a, int k) { return {a.m, a.e + k}; }  // a 2^k
ECPGB_HD xf xs_abs(xs a) { return xf_norm({a.m < 0 ? (u64)-a.m : (u64)a.m, a.e}); }
// a * c rounded to double (c positive).
ECPGB_HD double xs_times(xs a, xf c) {
  const xf v = xf_mul(xs_abs(a), c);
  return xf_to_double(v.m, v.e, a.m < 0 ? 0x80000000u : 0u);
}
// a <= b and a < b for normalised (or zero) a, b.
ECPGB_HD bool xf_le(xf a, xf b) { return a.m == 0 || (b.m != 0 && (a.e < b.e || (a.e == b.e && a.m <= b.m))); }
ECPGB_HD bool xf_lt(xf a, xf b) { return !xf_le(b, a); }

// A run of terms +-m 2^e: 57-bit mantissas, room for 63 terms before xs_fit.
struct xf_run {
  i64 m = 0;
  int e = -100000;
  // sign: any word whose top bit is the term's sign
  ECPGB_HD void add(xf t, uint32_t sign) {
    const i64 s = (i64)(int)sign >> 31;
    const i64 tm = ((i64)(t.m >> 7) ^ s) - s;
    const int te = t.e + 7, d = e - te;
    if (d < 0) {  // a larger term: the sum moves
      m >>= (d < -63 ? 63 : -d);
      e = te;
      m += tm;
    } else {
      m += tm >> (d > 63 ? 63 : d);
    }
  }
  ECPGB_HD xs sum() const { return xs_fit({m, e}); }
};

// An ECP term d r^n exp(-a r^2), laid out by the host: normalised mantissas and
// exponents of a and d, d's sign in the top bit, n (3: any other power).
struct FxTerm {
  u64 am, dm;
  int ae, de;
  uint32_t sign;
  int n;
};
inline FxTerm fx_term(double a, double d, double n) {
  const xf A = xf_from(a), D = xf_from(d);
  return {A.m, D.m, A.e, D.e, sign_of(d), n == 0 ? 0 : n == 1 ? 1 : n == 2 ? 2 : 3};
}

}  // namespace ecpgb
