// ecp_fast.cu -- the batched path's unit stages for sm_103a (FP64 and mixed).
//
// Same results as the plain path (same quadrature schedules, windows,
// convergence tests, stale-buffer semantics of the reference's fallbacks),
// organised for two properties of GB300: its FP64 pipe takes one warp instruction
// per 16 to 19 cycles and SM, however many lanes are active, and its instruction
// cache holds little more than one of these loops.
//   * stages instead of a unit a CTA: a plan (one warp a unit) lists the type-1
//     groups, type-2 batches and fallback parts; one-warp CTAs take entries
//     from the lists, so warps that run at the same time run the same code, no
//     barrier waits for a slow primitive pair, and a chunk of units bounds the
//     scratch between the stages;
//   * tables, walks and convergence tests on the integer pipes with 64-bit
//     mantissas (ecp_fixed.h), eleven bits more than FP64; FP64 where a value is
//     rounded once (quadrature results) and in the angular linking;
//   * level-granular tabulation: grid points are tabulated 32 schedule slots
//     at a time (one slot per lane) and a primitive pair stops as soon as all
//     its quadratures have converged -- the type-2 fallback's stop after ~280 of
//     the 1023 large-grid slots, where the reference tabulates all 1023;
//   * only what is read is computed: slots whose value passes the screen (a pair's
//     own points through its index interval), the rows and channels of the
//     quadratures still running, kept in a dense list and dealt to the lanes;
//   * the type-1 block accumulated per combined Cartesian index: chi[i][j]
//     depends on (i, j) only through the index of a_i + b_j
//     (src/type1.c:323-345), so one accumulator per combined index receives
//     exactly the terms the reference adds to each chi[i][j];
//   * little code in the hot loops (no unrolling, one copy of what is used
//     twice): a kilobyte more costs the large-grid stage 1 to 9 %.
// 50-centre cluster (90,976 units): 37.1 ms in these stages; one FP64 kernel
// with a unit a CTA took 116.3.
#include <algorithm>

#include "ecp_stages.cuh"

namespace ecpgb {

// --------------------------------------------------------------- helpers

// K_0..K_lmax(z) for z < 1e-7: the reference's zeroth-order branch,
// K_l = (1 - z) z^l / (2l+1)!! by its recurrence (src/bessel.c:118-133).
static __device__ void bessel_small(int lmax, double z, double *K, int stride) {
  if (z <= 0) {
    K[0] = 1.0;
    for (int l = 1; l <= lmax; l++) K[l * stride] = 0.0;
  } else {
    K[0] = 1 - z;
    for (int l = 1; l <= lmax; l++) K[l * stride] = K[(l - 1) * stride] * z / (2 * l + 1);
  }
}

static __device__ __noinline__ void bessel_fx(const DevJob &J, int lmax, xf z100, xf mul, uint32_t sign, double *K) {
  fx_bessel_rows(J.besX, J.besXA, J.besHL + 1, lmax, z100, mul, sign, K);
}

// The rows for the type-1 tables (late: 78 units' stages 0.233 -> 0.221 ms, the
// cluster's 37.4 -> 37.15; late in the large grid too: 37.3).
template <bool kLate>
static __device__ __noinline__ RowBase bessel_rows2(const DevJob &J, int lmax, xf z100, u64 *K) {
  return fx_bessel_packed<kLate>(J.besX, J.besXA, J.besHL + 1, lmax, z100, K);
}
// Powers of r other than 0, 1, 2: rare, out of line.
static __device__ __noinline__ double rpow_rare(double r, double n) { return rpow(r, n); }

// One row K_l(z), by the same branches as bessel_fx.
static __device__ __noinline__ double bessel_row(const DevJob &J, int l, double z) {
  if (__builtin_expect(z < 1.0E-7, 0)) {  // rare: laid out of line
    if (z <= 0) return l == 0 ? 1.0 : 0.0;
    double v = 1 - z;
    for (int i = 1; i <= l; i++) v = v * z / (2 * i + 1);
    return v;
  }
  if (z >= 16.0) {
    const int HL1 = J.besHL + 1;
    const double mult = 0.5 * __drcp_rn(z), x = -mult;
    const double *q = J.besA + (size_t)l * (HL1 < 6 ? 6 : HL1);
    int k = l > 5 ? l : 5;
    double v = q[k];
    while (k > 0) {
      k--;
      v = fma(v, x, q[k]);
    }
    return v * mult;
  }
  double h = J.besselN / 16;
  int index = (int)floor(z * h + 0.5);
  double dz = z - __ldg(J.besZ + index);  // index / h, tabulated
  const double *q = J.besH + ((size_t)index * (J.besHL + 1) + l) * 6;
  double v = fma(q[5], dz, q[4]);
  v = fma(v, dz, q[3]);
  v = fma(v, dz, q[2]);
  v = fma(v, dz, q[1]);
  return fma(v, dz, q[0]);
}

// U_l(r) of centre c (src/ecp.c:42-60): its terms of channel l, summed with
// 60-bit mantissas; normalised, with its sign.  A term whose exponential is below
// e^-700 is left out.
static __device__ __noinline__ xf channel(const DevJob &J, int c, int l, double r, uint32_t &sign) {
  const xf R = xf_from(r), R2 = norm1(xf_mul(R, R));
  xs acc;
  const int *ch = J.chanT0 + c * (kMaxLEcp + 2) + l, t1 = ch[1];
#pragma unroll 1
  for (int t = ch[0]; t < t1; t++) {
    const FxTerm T = J.termFx[t];
    const xf a = xf_mul({T.am, T.ae}, R2);
    const u64 E = shr64(a.m, -(a.e + 53));  // a r^2 in Q53
    if (a.e + 53 > 0 || E > (u64)(700ll << 53)) continue;
    const xf Rn = T.n == 1 ? R : R2;
    xf v = xf_mul(fx_exp(-(i64)E), {T.dm, T.de});
    if (T.n) v = xf_mul(v, T.n < 3 ? Rn : xf_from(rpow_rare(r, J.termN[t])));
    const i64 m = (i64)(v.m >> 4), s = (i64)(int)T.sign >> 31;
    acc = xs_add(acc, {(m ^ s) - s, v.e + 4});
  }
  sign = acc.m < 0 ? 0x80000000u : 0u;
  return xs_abs(acc);
}

// ------------------------------------------- double-single (mixed path)
//
// The mixed path evaluates the type-1 large-grid fallback's tables -- Bessel
// rows, ECP channels, powers of r, the Gaussian prefactor -- and its integrand
// products in double-single arithmetic (ecp_ff.h: FP32 pairs on the FMA
// pipes), sums each level of a quadrature with a compensated FP32 sum and
// adds it to the FP64 running sum at the level's end.  The fallback's test
// (PSM92, 16 e^2 <= 3 N |I - q| tol) compares level differences far above the
// double-single rounding, so it takes the FP64 path's decisions; the
// small-grid quadratures, whose absolute test (err < tol) sits at the FP64
// rounding level for large integrals, are not touched.  The type-2 fallback
// runs on the integer tables: in double-single it took 45.1 ms of unit stages on
// the cluster against 38.7, and 65.6 against 48.2 on the 150-shell sweep.

// 1 / z: the float reciprocal refined by one Newton step in ff.
static __device__ inline ff ff_recip(ff z) {
  const float y = __frcp_rn(z.hi);
  const float e = __fmaf_rn(-z.lo, y, __fmaf_rn(-z.hi, y, 1.0f));  // 1 - z y
  return ff_norm(y, __fmul_rn(y, e));
}

// K_0..K_lmax(z) in ff: the branches of fx_bessel over the tables' float
// pairs (Taylor coefficients, table abscissae, large-argument polynomial).
static __device__ __noinline__ void bessel_ff(const DevJob &J, int lmax, ff z, ff *K, int stride) {
  if (__builtin_expect(z.hi < 1.0e-7f, 0)) {  // rare: the small-argument formula in FP64
    double Kd[kMaxRows];
    bessel_small(lmax, ff_to_double(z), Kd, 1);
    for (int l = 0; l <= lmax; l++) K[l * stride] = ff_from_double(Kd[l]);
    return;
  }
  const int HL1 = J.besHL + 1;
  if (z.hi > 16.0f || (z.hi == 16.0f && z.lo >= 0.0f)) {
    const ff inv = ff_recip(z);
    const ff mult = {0.5f * inv.hi, 0.5f * inv.lo}, x = ff_neg(mult);  // 1/(2z), -1/(2z)
    const int cs = HL1 < 6 ? 6 : HL1;
    for (int l = 0; l <= lmax; l++) {
      const ff *q = J.besAf + (size_t)l * cs;
      int k = l > 5 ? l : 5;
      ff v = q[k];
      while (k > 0) {
        k--;
        v = ff_add(ff_mul(v, x), q[k]);
      }
      K[l * stride] = ff_mul(v, mult);
    }
    return;
  }
  // the nearest table point; any neighbour would do as well (the Taylor
  // series is accurate over the whole table step)
  const int index = (int)floorf(__fmaf_rn(z.hi, (float)(J.besselN / 16), 0.5f));
  const ff x = ff_add(z, ff_neg(J.besZf[index]));
  const ff *qf = J.besHf + (size_t)index * HL1 * 6;
  for (int l = 0; l <= lmax; l++) {
    const ff *q = qf + 6 * l;
    // the two top terms (below 1e-9 of the row) in FP32
    ff v = ff_add(ff_mul_f(x, __fmaf_rn(q[5].hi, x.hi, q[4].hi)), q[3]);
    v = ff_add(ff_mul(v, x), q[2]);
    v = ff_add(ff_mul(v, x), q[1]);
    K[l * stride] = ff_add(ff_mul(v, x), q[0]);
  }
}

// One ECP term d r^n exp(-a r^2) in ff (r2 = r^2); terms below 2^-125 of
// their coefficient are 0.
static __device__ inline ff ecp_term_ff(const DevJob &J, int t, ff r, ff r2) {
  const ff arg = ff_mul(J.termAf[t], r2);
  if (arg.hi > 87.0f) return {0.0f, 0.0f};
  const ff v = ff_mul(J.termDf[t], ff_exp(ff_neg(arg)));
  const double n = J.termN[t];
  if (n == 0.0) return v;
  if (n == 1.0) return ff_mul(v, r);
  if (n == 2.0) return ff_mul(v, r2);
  return ff_mul(v, ff_from_double(rpow(ff_to_double(r), n)));  // other powers: rare
}

// U_l(r) in ff.
static __device__ __noinline__ ff channel_ff(const DevJob &J, int c, int l, ff r) {
  const ff r2 = ff_mul(r, r);
  ff pot = {0.0f, 0.0f};
  const int t0 = J.ctrT0[c], t1 = t0 + J.ctrNT[c];
  for (int t = t0; t < t1; t++)
    if (J.termL[t] == l) pot = ff_add(pot, ecp_term_ff(J, t, r, r2));
  return pot;
}


// A level's constants of both rules, in shared memory: tol 3 n / 16 and 16 / (3 n).
constexpr int kMaxLevels = 16;
struct LevelTab {
  u64 cm[kMaxLevels], rm[kMaxLevels];
  int ce[kMaxLevels], re[kMaxLevels];
};
static __device__ inline void level_tab(LevelTab &T, const double *n3, int levels, double tol) {
  const int k = threadIdx.x & 31;
  if (k < levels && k < kMaxLevels) {
    const xf c = xf_norm(xf_mul(xf_from(n3[k]), xf_from(tol)));
    const xf r = xf_from(1.0 / n3[k]);  // the quotient's rounding: half an ulp
    T.cm[k] = c.m;
    T.ce[k] = c.e - 4;
    T.rm[k] = r.m;
    T.re[k] = r.e + 4;
  }
  __syncwarp();
}

static __device__ inline uint32_t ent_h(double x) { return (uint32_t)((u64)dbits(x) >> 32); }

// xs_add and xs_times out of line: the level ends use them several times, and
// one copy keeps the kernels' loops in the instruction cache.
static __device__ __noinline__ xs xs_plus(xs a, xs b) { return xs_add(a, b); }
static __device__ __noinline__ double xs_scaled(xs a, xf c) { return xs_times(a, c); }

// A quadrature's state between levels: the running sum now, and at the ends
// of the last two levels.
struct Psm92 {
  xs I, I1, I2;
};
// After slot 0: p = I, so q = 2 p = 4 (I / 2) on the first level.
static __device__ inline void psm92_head(Psm92 &S) {
  S.I1 = S.I;
  S.I2 = xs_shl(S.I, -1);
}
// A level's end of the PSM92 walk (src/gc_integrators.c:39-86), T its sum: p =
// 2 I1 and q = 4 I2 there, and the test is 16 e^2 <= 3 N |I - q| tol.
static __device__ inline bool psm92_end(Psm92 &S, const LevelTab &L, int k) {
  const xs e = xs_plus(S.I, xs_shl(xs_neg(S.I1), 1)), d = xs_plus(S.I, xs_shl(xs_neg(S.I2), 2));
  S.I2 = S.I1;
  S.I1 = S.I;
  const xf a = xs_abs(e), b = norm1(xf_mul(xs_abs(d), {L.cm[k], L.ce[k]}));
  return a.m == 0 || xf_le(norm1(xf_mul(a, a)), b);
}
static __device__ inline double psm92_result(const Psm92 &S, const LevelTab &L, int k) {
  return xs_scaled(S.I1, {L.rm[k], L.re[k]});
}

// State of the PS93 walk (src/gc_integrators.c:157-217) and its level end: true
// when the level's test 16 d / (3 n) < tol accepts (cnt points counted).
struct Ps93 {
  xs I, p, q;
};
static __device__ inline bool ps93_end(Ps93 &S, const LevelTab &L, int k, int cnt) {
  xs d;
  if (c93_lvJ[k]) {
    d = xs_plus(S.I, xs_shl(xs_neg(S.q), 1));
    S.q = S.I;
  } else {
    S.p = xs_plus(S.p, xs_plus(S.I, xs_neg(S.q)));
    const xs h = xs_plus(S.p, xs_shl(S.p, -1));  // 3 p / 2
    d = xs_plus(S.q, xs_neg(h));
  }
  return cnt > 0 && xf_lt(xs_abs(d), {L.cm[k], L.ce[k]});
}
static __device__ inline double ps93_result(const Ps93 &S, const LevelTab &L, int k) {
  return xs_scaled(S.q, {L.rm[k], L.re[k]});
}

static __device__ inline xs combine(xs a, int P) {
#pragma unroll 1
  for (int o = 1; o < P; o <<= 1) {
    xs b;
    b.m = __shfl_xor_sync(0xffffffffu, a.m, o);
    b.e = __shfl_xor_sync(0xffffffffu, a.e, o);
    a = xs_plus(a, b);
  }
  return a;
}
static __device__ inline xs from_lane(xs a, int src) {
  xs b;
  b.m = __shfl_sync(0xffffffffu, a.m, src);
  b.e = __shfl_sync(0xffffffffu, a.e, src);
  return b;
}

// The PSM92 walk of slots s0 to s1 with val(pos) in ff: each level summed with a compensated
// FP32 sum and added to the FP64 running sum I at the level's end (and at
// the end of the slots walked, so that I is complete between calls).
template <class V, class Vis>
static __device__ inline void psm92_advance_ff(int s0, int s1, double tol, V val, Vis vis, double &I, double &p,
                                               double &q, bool &done, double &res) {
  int pos = s0;
  if (pos == 0) {
    I = ff_to_double(val(0));
    p = I;
    pos = 1;
  }
  int k = level_of(pos);
  ff_acc acc;
  while (pos < s1 && !done) {
    int lvStart = k == 0 ? 1 : c92_lvEnd[k - 1];
    if (pos == lvStart) {
      q = 2 * p;
      p = 2 * I;
    }
    acc.add(val(pos));
    if (vis(pos + 1)) acc.add(val(pos + 1));
    pos += 2;
    if (pos == c92_lvEnd[k]) {
      I += acc.value();
      acc = ff_acc();
      double N = c92_lvN[k] + 1.0, e = I - p;
      if (16 * e * e <= 3 * N * fabs(I - q) * tol) {
        res = 16 * I / (3 * N);
        done = true;
      }
      k++;
    }
  }
  I += acc.value();
}

PairPlan pair_plan(int NP, int la, int lb, int nItems, bool single) {
  PairPlan p;
  if (la < 0 || lb < 0) NP = nItems = la = lb = 0;
  p.scratch = unit_scratch(NP, la + lb, nItems, single).total;
  p.lists = (long long)unit_list_bytes(NP, nItems, single);
  p.groups = NP;
  p.batches = (nItems + 31) / 32;
  p.parts = NP ? t2_parts(NP, single) : 0;
  return p;
}

size_t fast_smem_bytes(int LB, int t2Rows, int gcap) { return sizeof(double) * (size_t)small_layout(LB, t2Rows, gcap).total; }

// Mixed path: the largest quadrature value for which double-single level
// sums still decide the large-grid convergence test as FP64 does.  The
// test 16 e^2 <= 3 N |I - q| tol needs the noise of e and I - q, about
// 2^-47 of the integral in double-single, well below 3 N tol / 16; at the
// coarsest levels (N = 256) that noise reaches it for integrals near
// 2^47 tol 48, so quadratures above 1/8 of that take FP64 tables.
__device__ inline double ff_limit(double tol) { return 0x1p47 * tol * 6.0; }

// --------------------------------------------------------------- type 1

// Direction of the k-vector P as (cos theta, cos phi, sin phi), the values
// src/util.c:75-106 and src/spherical_harmonics.c:16-114 produce through
// theta = acos(z/r), phi = atan(y/x) (+pi) and their cosines and sines,
// computed here without the inverse and direct trigonometric functions (the
// same values within a few ulps; the reference's special cases -- r or x
// below 1e-14 -- are kept).
static __device__ void direction(const double *P, double &ct, double &cp, double &sp) {
  const double eps = 1.0E-14, x = P[0], y = P[1], z = P[2];
  const double r = sqrt(x * x + y * y + z * z);
  ct = r < eps ? 1.0 : fmin(1.0, fmax(-1.0, z / r));
  if (fabs(x) < eps) {
    if (fabs(y) < eps) {
      cp = 1.0;
      sp = 0.0;
    } else {
      const double ph = y < 0.0 ? 1.5 * kPi : 0.5 * kPi;
      cp = cos(ph);
      sp = sin(ph);
    }
  } else {
    const double t = y / x, h = 1.0 / sqrt(1.0 + t * t);  // cos(atan t), sin = t cos
    cp = x > 0.0 ? h : -h;
    sp = x > 0.0 ? t * h : -(t * h);
  }
}

// Column m of the real spherical harmonics S_lm, l = m..lmax, into rsh[l*l +
// l -/+ m]: the associated Legendre recurrence, normalisation and sin/cos(m
// phi) recurrence of src/spherical_harmonics.c:16-114, one column per lane;
// x = cos theta, (c1, s1) = (cos phi, sin phi).
static __device__ void rsh_column(const DevJob &J, int lmax, int m, double x, double c1, double s1,
                                  double *rsh) {
  const int W = J.tmDim + 1;
  double sm = 0.0, cm = 1.0;
  if (m > 0) {
    sm = s1;
    cm = c1;
    for (int i = 2; i <= m; i++) {
      double sn = s1 * cm + c1 * sm, cn = c1 * cm - s1 * sm;
      sm = sn;
      cm = cn;
    }
  }
  double P2 = 0.0, P1 = 0.0, P = 0.0;
  double sp = 1.0;
  if (x != 1.0 && x != -1.0) {
    double st = sqrt(1.0 - x * x);
    sp = st;
    for (int i = 2; i <= m; i++) sp = sp * st;
  }
  for (int l = m; l <= lmax; l++) {
    if (1.0 == x) P = (m == 0) ? 1.0 : 0.0;
    else if (-1.0 == x) P = (m == 0) ? (l == 0 ? 1.0 : -P1) : 0.0;
    else if (l == m) P = (m == 0) ? 1.0 : sp * J.dfac[2 * m - 1];
    else if (l == m + 1) P = x * (2 * m + 1) * P1;
    else P = (x * (2 * l - 1) * P1 - (l + m - 1) * P2) * __ldg(kRecip + (l - m));
    P2 = P1;
    P1 = P;
    double v = J.shNorm[l * W + m] * P;
    if (m == 0) rsh[l * l + l] = v * 0x1.6a09e667f3bcdp-1;  // v / sqrt(2)
    else {
      rsh[l * l + l - m] = v * sm;
      rsh[l * l + l + m] = v * cm;
    }
  }
}

// Type-1 table entries, 2 lq + 1 words: K_l (fx_bessel_packed), then normalised
// mantissas of v r^l, then the exponents: of row l1 times K_l2,
// e + l1 er - (leading bits won back up to row l1) - l2 t - (K's low bits).
struct EntInfo {
  int e;       // 2 e + sign
  int packed;  // er (8 bits, signed), t (8 bits), from bit 16 a bit per row l = 1.. whose product was shifted
};
constexpr EntInfo kNoEntry = {-2000000, 0};
// A point past the break: the entry holds doubles.
constexpr int kStaleEntry = INT_MIN;
static __device__ inline EntInfo t1_entry_rows(u64 *WR, xf v, const RowBase &b, xf R, uint32_t sign, int lmax) {
  v = xf_norm(xf_mul(v, b.c));
  u64 m = v.m;
  WR[0] = m;
  unsigned won = 0;
#pragma unroll 1
  for (int l = 1; l <= lmax; l++) {
    m = mul_hi(m, R.m);
    if ((i64)m >= 0) {
      m += m;
      won |= 1u << (15 + l);
    }
    WR[l] = m;
  }
  return {(v.e + b.e0 + 64) * 2 + (int)(sign >> 31), ((R.e + 64) & 255) | b.t << 8 | (int)won};
}
// What a quadrature (l1, l2) reads of an entry's exponents: their factors, a byte
// each, and the mask of the products up to row l1.
struct EntRow {
  int l, won;
};
static __device__ inline EntRow t1_entry_row(int l1, int l2) { return {l1 | (-l2 & 255) << 8, (1 << (16 + l1)) - (1 << 16)}; }
// The product of row l1 and K_l2 of an entry into a run (l1 er - l2 t in one instruction).
static __device__ inline void t1_entry_add(xf_run &run, u64 wr, u64 k, EntInfo f, EntRow q) {
  const xf K = row_packed(k);
  run.add({mul_hi(wr, K.m), __dp4a(f.packed, q.l, f.e >> 1) + K.e - __popc(f.packed & q.won)}, (uint32_t)f.e << 31);
}

// One live entry of the type-1 large-grid tables: K_l(s r) and w C2 U_L(r) e^ex
// r^l; kNoEntry where it is zero.
static __device__ __noinline__ EntInfo t1_large_entry(const DevJob &J, int c, int Lc, double r, double ex, double w,
                                                      double C2, double s, int kq, int rq, u64 *K, u64 *WR) {
  const xf R = xf_from(r);
  uint32_t sign;
  xf v = channel(J, c, Lc, r, sign);
  v = xf_mul(xf_mul(fx_exp(fx_q53(ex)), v), xf_mul(xf_from(C2), xf_from(w)));
  if (v.m == 0) return kNoEntry;
  sign ^= sign_of(C2) ^ sign_of(w);
  const RowBase b = bessel_rows2<false>(J, kq, xf_mul(xf_times100(xf_from(s)), R), K);
  return t1_entry_rows(WR, v, b, R, sign, rq);
}

// --------------------------------------------------- stage 2: the small grid

// A group of G primitive pairs of one kind (perm[p0 ..]) of a unit's type-1
// quadratures on the small grid (src/type1.c:95-148), by one warp; lane =
// (pair, quadrature).  G fills the lanes of the tabulation's entries as far as the
// step table's width allows.  Converged quadratures are written to the unit's Q, the
// pairs with a failed one to the fallback list.
template <bool kMixed, int kKind>
static __device__ void t1_small(const DevJob &J, const Unit &U, const SmallSmem &L, double *sm, const LevelTab &V,
                                int off, int p0, int G) {
  const int lane = threadIdx.x & 31, lab = U.lab, lq = lab + 1, O = kSmallOrder, ws = U.ws, we = U.we;
  // odd entry strides: lanes touching neighbouring entries hit distinct banks
  const int TS = 1 + 2 * lq, nq = t1_items(lab);
  const u64 thr = J.lnAcc1Q53;
  double *rec = sm + L.rec, *tab = sm + L.tab;  // the pairs' records
  const unsigned char *perm = (const unsigned char *)(U.scr + U.L.perm);
  const double *uL = J.uL + (size_t)U.c * O;
  __syncwarp();
#pragma unroll 1
  for (int e = lane; e < G * kPairWords; e += 32)
    rec[e] = ((const double *)(U.scr + U.L.pair))[perm[p0 + e / kPairWords] * kPairWords + e % kPairWords];
  __syncwarp();
  // (2) PS93: lane = (pair g, quadrature (l1, l2))
  const bool mine = lane < G * nq;
  const int g = mine ? lane / nq : 0, qi = mine ? lane % nq : 0;
  int l1 = 0, l2 = 0;
  {
    int rem = qi;
    while (l1 <= lab && rem >= l1 / 2 + 1) { rem -= l1 / 2 + 1; l1++; }
    l2 = l1 - 2 * rem;
  }
  double *Qout = (double *)(U.scr + U.L.Q) + (size_t)perm[p0 + g] * nq + qi;
  double I = 0, p = 0, q = 0, T = 0;  // band kind, T the running slot pair
  Ps93 S;                             // normal kind
  xs lev;                             // its running level
  int *quad = (int *)(sm + L.quad);   // the running quadratures, by rank
  bool done = !mine;
  int k = -2, cnt = 0, lvEnd = 1;
  if constexpr (kKind == kPairZero) {
    // converged quadratures give 0; failed ones go to the fallback
    if (mine) {
      done = t1_zero_walk(J, rec[g * kPairWords], rec[g * kPairWords + 2], ws, we);
      if (done) *Qout = 0.0;
    }
  } else
#pragma unroll 1
  for (int s0 = 0; s0 < O;) {
    const int s1 = step_end93(s0) < O ? step_end93(s0) : O;
    // slot entry: [0, lq) K_l(s r), [lq, 2lq) w * C1 U_L e^(..) r^l; zero
    // outside the window.  The step's in-window slots are the run [lo, hi)
    // of its by-point order, dealt to consecutive lanes.
    const int ns = s1 - s0;
    int lo, hi;
    {
      const int n0 = lane < ns ? __ldg(J.byN93 + s0 + lane) >> 16 : INT_MAX;
      const int n1 = lane + 32 < ns ? __ldg(J.byN93 + s0 + lane + 32) >> 16 : INT_MAX;
      lo = __popc(__ballot_sync(0xffffffffu, n0 < ws)) + __popc(__ballot_sync(0xffffffffu, n1 < ws));
      hi = __popc(__ballot_sync(0xffffffffu, n0 < we)) + __popc(__ballot_sync(0xffffffffu, n1 < we));
    }
    const int nIn = hi - lo;
    // only the pairs of the group with a quadrature still running are
    // tabulated: a converged lane reads no entry again
    unsigned live = 0;
    {
      const unsigned run = __ballot_sync(0xffffffffu, !done), qm = nq >= 32 ? ~0u : (1u << nq) - 1u;
#pragma unroll 1
      for (int gg = 0; gg < G; gg++)
        if (run >> (gg * nq) & qm) live |= 1u << gg;
    }
    const int nLive = __popc(live);
    // the live pairs' indices, 4 bits each (G <= 8), and entry e's (slot,
    // live pair) = (e / nLive, e % nLive) with the quotient by a
    // multiply-shift: ceil(2^16 / d) is exact for d <= 8 and e < 8192
    // (e < 33 * 8 here) -- no integer divide in the loops
    unsigned packed = 0;
#pragma unroll 1
    for (unsigned m = live, j = 0; m; m &= m - 1u, j++) packed |= (unsigned)(__ffs(m) - 1) << (4 * j);
    const unsigned dmag = nLive > 0 ? (65536u + (unsigned)nLive - 1u) / (unsigned)nLive : 0u;
    auto slot_of = [&](int e) { return (int)(((unsigned)e * dmag) >> 16); };
    auto live_pair = [&](int e, int i) { return (int)((packed >> (4 * (e - i * nLive))) & 15u); };
#pragma unroll 1
    for (int e = lane; e < nIn * nLive; e += 32) {
      const int i = slot_of(e);
      const int gg = live_pair(e, i), tn = __ldg(J.byN93 + s0 + lo + i), t = tn & 0xffff, n = tn >> 16;
      double *ent = tab + ((t - s0) * G + gg) * TS, *WR = ent + lq;
      const PairRec &P = *(const PairRec *)(rec + gg * kPairWords);
      const double s = P.s, C1 = P.C1;
      if constexpr (kKind == kPairBand) {
        // row l: (C1 r^l) U; the walk multiplies by K, exp(e) and w in turn
        const double r = J.xSmall[n], ex = t1_exponent(P.z, s, r);
        bessel_fx(J, lab, xf_mul(xf_times100(xf_from(s)), xf_from(r)), {0, 0}, 0, ent);
        double R = 1.0;
#pragma unroll 1
        for (int l = 0; l <= lab; l++) {
          if (l) R = __dmul_rn(r, R);
          WR[l] = __dmul_rn(__dmul_rn(C1, R), uL[n]);
        }
        ent[2 * lq] = ex >= J.lnAcc1 ? fast_exp(ex) : 0.0;
      } else {
        // the table row in integers: e = (s - Z r) r in Q53, then
        // w C1 U_L exp(e) r^l with 60-bit mantissas
        const double w = J.wSmall[n], u = uL[n];
        const xf R = xf_from(J.xSmall[n]);
        const PairFx F = P.fx;
        const u64 zr = shr64(mul_hi(F.Zm, R.m), -(F.Ze + R.e + 64 + F.q));
        const i64 tt = F.S - (i64)zr;
        u64 E = mul_hi(tt < 0 ? (u64)-tt : (u64)tt, R.m);
        const int sh = 117 - F.q + R.e;
        E = sh <= 0 ? shr64(E, -sh) : (E >> (63 - (sh > 63 ? 63 : sh)) ? ~0ull >> 1 : E << sh);
        EntInfo info = kNoEntry;  // below the screen
        if (tt >= 0 || E <= thr) {
          const xf v = xf_mul(xf_mul(fx_exp(tt < 0 ? -(i64)E : (i64)E), xf_from(C1)), xf_mul(xf_from(w), xf_from(u)));
          const RowBase b = bessel_rows2<true>(J, lab, xf_mul({F.sm, F.se}, R), (u64 *)ent);
          info = t1_entry_rows((u64 *)WR, v, b, R, sign_of(w) ^ sign_of(u) ^ sign_of(C1), lab);
        }
        *(EntInfo *)(ent + 2 * lq) = info;
      }
    }
    __syncwarp();
    if constexpr (kKind == kPairBand) {
      // w * ((((C1 r^l1) U) K_l2) exp(e)), each product rounded; slot 0 and
      // slots 1, 2 are levels of their own (-2, -1)
#pragma unroll 1
      for (int t = s0; t < s1; t++) {
        const int n = c93_slot[t];
        if (!done && n >= ws && n < we) {
          const double *e = tab + ((t - s0) * G + g) * TS;
          T = __dadd_rn(T, __dmul_rn(J.wSmall[n], __dmul_rn(__dmul_rn(e[lq + l1], e[l2]), e[2 * lq])));
        }
        cnt += (t & 1) ? n >= ws : n <= we;
        if (t > 2 && !(t & 1)) {  // the reference's order: pair by pair
          I += T;
          T = 0.0;
        }
        if (t + 1 < lvEnd) continue;
        if (!done) {
          if (k == -2) p = T;
          else if (k == -1) {
            q = T;
            I = p + q;
          } else {
            const double n3 = c93_3n[k];
            double d;
            if (c93_lvJ[k]) {
              d = fabs(I - 2 * q);
              q = I;
            } else {
              p += I - q;
              d = fabs(q - 3 * p / 2);
            }
            if (cnt > 0 && d < J.tol * 0.0625 * n3) {
              done = true;
              *Qout = 16 * q / n3;
            }
          }
        }
        T = 0.0;
        k++;
        lvEnd = k < 0 ? 3 : c93_lvEnd[k];  // k <= the level count, inside the 32-entry table
        cnt = 0;
      }
    } else {
      // the step's slots inside the window, and those that count as points
      u64 inw, counts;
      {
        const int t = s0 + lane, n = t < s1 ? __ldg(J.s93 + t) : 0, n32 = c93_slot[32];
        inw = __ballot_sync(0xffffffffu, t < s1 && n >= ws && n < we);
        counts = __ballot_sync(0xffffffffu, t < s1 && ((t & 1) ? n >= ws : n <= we));
        if (s0 == 0) {  // the first step's 33rd slot
          inw |= (u64)(n32 >= ws && n32 < we) << 32;
          counts |= (u64)(n32 <= we) << 32;
        }
      }
      // runs of slots of one level, the lanes dealt to the running quadratures
      const unsigned act = __ballot_sync(0xffffffffu, !done);
      const LaneDeal D = deal_lanes(__popc(act));
      const int mine_rank = __popc(act & ((1u << lane) - 1u));
      if (!done) quad[mine_rank] = g | l1 << 8 | l2 << 16;
      __syncwarp();
      const bool work = D.rank < __popc(act);
      const int qd = work ? quad[D.rank] : 0;
      const int q1 = (qd >> 8) & 255;
      const u64 *eT = (const u64 *)tab + (qd & 255) * TS;
      const int oW = lq + q1, oK = qd >> 16;
      const EntRow qr = t1_entry_row(q1, oK);
#pragma unroll 1
      for (int t = s0; t < s1;) {
        const int te = lvEnd < s1 ? lvEnd : s1;
        const u64 bits = ((1ull << (te - s0)) - 1ull) & ~0ull << (t - s0);
        cnt += __popcll(counts & bits);
        xf_run run;
#pragma unroll 1
        for (int x = t + D.part; x < te; x += D.P)
          // the points inside the window (the entries outside it are zero)
          if (work && (inw >> (x - s0) & 1u)) {
            const u64 *e = eT + (x - s0) * G * TS;
            t1_entry_add(run, e[oW], e[oK], *(const EntInfo *)(e + 2 * lq), qr);
          }
        xs sum = combine(run.sum(), D.P);
        sum = from_lane(sum, (mine_rank * D.P) & 31);
        lev = xs_plus(lev, sum);
        t = te;
        if (t < lvEnd) break;
        if (!done) {
          if (k == -2) S.p = lev;
          else if (k == -1) {
            S.q = lev;
            S.I = xs_plus(S.p, S.q);
          } else {
            S.I = xs_plus(S.I, lev);
            if (ps93_end(S, V, k, cnt)) {
              done = true;
              *Qout = ps93_result(S, V, k);
            }
          }
        }
        lev = xs();
        k++;
        lvEnd = k < 0 ? 3 : c93_lvEnd[k];
        cnt = 0;
      }
    }
    __syncwarp();
    s0 = s1;
    if (__all_sync(0xffffffffu, done)) break;
  }
  // (3) the pairs with a failed quadrature, to the large grid
  const unsigned fail = __ballot_sync(0xffffffffu, mine && !done);
  if (!fail) return;
  // mixed path: double-single tables only where the sums of the pair's failed
  // quadratures can take the reference's decisions (ff_limit, judged on their
  // last small-grid estimates, by the high words); larger integrals in FP64
  unsigned est = 0, lim = 0;
  if constexpr (kMixed) {
    const double last = kKind == kPairNormal ? ps93_result(S, V, c93_nLevels - 1) : 16 * q / c93_3n[c93_nLevels - 1];
    est = mine && !done ? (unsigned)((u64)__double_as_longlong(fabs(last)) >> 32) : 0u;
    lim = (unsigned)((u64)__double_as_longlong(ff_limit(J.tol)) >> 32);
  }
#pragma unroll 1
  for (int gg = 0; gg < G; gg++) {
    const unsigned m = fail >> (gg * nq) & (nq >= 32 ? ~0u : (1u << nq) - 1u);
    if (!m) continue;
    int ffp = 0;
    if constexpr (kMixed) ffp = __reduce_max_sync(0xffffffffu, g == gg ? est : 0u) < lim;
    if (lane == 0) J.listFail[atomicAdd(J.counters + kCntFail, 1u)] = {off, perm[p0 + gg] | ffp << 16, m, 0, rec[gg * kPairWords]};
  }
}

// A batch of up to 32 type-2 small-grid quadratures (src/type2.c:337-387), by
// one warp.  32 slots at a time, a slot a lane, the rows that the batch reads of
// both F tables (derivative runs max(0, shift), src/type2.c:563-564) and of the
// weighted r^k U_l table are laid out as mantissas and 16-bit exponents (4 e +
// sign: three signs fit the low bits of a sum), so a point costs a quadrature
// two products and one sum.  The lanes are dealt to the running quadratures,
// again whenever half of them have converged.
static __device__ void t2_small(const DevJob &J, const Unit &U, const LevelTab &V, u64 *tab, int *quad, int q0) {
  const int lane = threadIdx.x & 31, O = kSmallOrder, nF = J.nF, nk = J.nk, LE = J.maxLECP > 0 ? J.maxLECP : 1,
            nRuns = J.nRuns > 0 ? J.nRuns : 1, ws = U.ws, we = U.we;
  int n = U.nItems - q0 < 32 ? U.nItems - q0 : 32;
  LaneDeal D = deal_lanes(n);
  bool done = D.rank >= n;
  int q = q0 + (done ? 0 : D.rank);
  const int item = unit_item(J, U, q), il = item & 255, i1 = (item >> 8) & 255, i2 = (item >> 16) & 255, i3 = item >> 24;
  // the batch's rows: l1 in [a0, a0 + nA), l2 in [b0, b0 + nB), l3 < n3 of
  // channels [u0, u0 + nU)
  const int a0 = __reduce_min_sync(0xffffffffu, i1), nA = __reduce_max_sync(0xffffffffu, i1) - a0 + 1;
  const int b0 = __reduce_min_sync(0xffffffffu, i2), nB = __reduce_max_sync(0xffffffffu, i2) - b0 + 1;
  const int u0 = __reduce_min_sync(0xffffffffu, il), nU = __reduce_max_sync(0xffffffffu, il) - u0 + 1;
  const int n3 = __reduce_max_sync(0xffffffffu, i3) + 1;
  const int rows = nA + nB + nU * n3, TS = (rows + (rows + 3) / 4) | 1;
  int at = (i1 - a0) | (nA + i2 - b0) << 8 | (nA + nB + (il - u0) * n3 + i3) << 16;  // the quadrature's rows
  const double *Fa = J.F + (((size_t)U.c * J.nShells + U.sa) * nRuns + U.pa0) * O * nF + a0;
  const double *Fb = J.F + (((size_t)U.c * J.nShells + U.sb) * nRuns + U.pb0) * O * nF + b0;
  const double *Ut = J.utab + (size_t)U.c * O * LE * nk + u0 * nk;
  Ps93 S;
  xs lev;
  int k = -2, cnt = 0, lvEnd = 1;  // slot 0 and slots 1, 2 are levels of their own (-2, -1)
#pragma unroll 1
  for (int s0 = 0; s0 < O; s0 += 32) {
    const int s1 = s0 + 32 < O ? s0 + 32 : O;
    const int m = s0 + lane < s1 ? __ldg(J.s93 + s0 + lane) : 0;
    const bool in = s0 + lane < s1 && m >= ws && m < we;  // (the integrand is 0 outside the window)
    const unsigned inw = __ballot_sync(0xffffffffu, in);
    const unsigned counts = __ballot_sync(0xffffffffu, s0 + lane < s1 && ((lane & 1) ? m >= ws : m <= we));
    __syncwarp();
    if (in) {
      u64 *M = tab + lane * TS;
      short *E = (short *)(M + rows);
      const xf w = xf_from(J.wSmall[m]);
      int i = 0;
#pragma unroll 1
      for (int g = 0; g < 2 + nU; g++) {
        const double *src = g == 0 ? Fa + (size_t)m * nF : g == 1 ? Fb + (size_t)m * nF : Ut + ((size_t)m * LE + g - 2) * nk;
        const int cntR = g == 0 ? nA : g == 1 ? nB : n3;
#pragma unroll 1
        for (int r = 0; r < cntR; r += 4) {
          double x[4];
#pragma unroll
          for (int j = 0; j < 4; j++) x[j] = r + j < cntR ? __ldg(src + r + j) : 0.0;
#pragma unroll
          for (int j = 0; j < 4; j++) {
            if (r + j >= cntR) break;
            xf v = xf_from(x[j]);
            if (g >= 2) v = norm1(xf_mul(v, w));
            M[i] = v.m;
            E[i] = (short)(v.e * 4 + (int)(sign_of(x[j]) >> 31));
            i++;
          }
        }
      }
    }
    __syncwarp();
#pragma unroll 1
    for (int t = s0; t < s1;) {
      const int te = lvEnd < s1 ? lvEnd : s1;
      const unsigned bits = (te - s0 >= 32 ? ~0u : (1u << (te - s0)) - 1u) & ~0u << (t - s0);
      cnt += __popc(counts & bits);
      const int ra = at & 255, rb = (at >> 8) & 255, ru = at >> 16;
      xf_run run;
#pragma unroll 1
      for (int x = t + D.part; x < te; x += D.P)
        if (inw >> (x - s0) & 1u) {
          const u64 *M = tab + (x - s0) * TS;
          const short *E = (const short *)(M + rows);
          const int e = E[ra] + E[rb] + E[ru];
          run.add({mul_hi(mul_hi(M[ra], M[rb]), M[ru]), (e >> 2) + 128}, (uint32_t)e << 31);
        }
      lev = xs_plus(lev, combine(run.sum(), D.P));
      t = te;
      if (t < lvEnd) break;
      if (k == -2) S.p = lev;
      else if (k == -1) {
        S.q = lev;
        S.I = xs_plus(S.p, S.q);
      } else {
        S.I = xs_plus(S.I, lev);
        if (!done && ps93_end(S, V, k, cnt)) {
          done = true;
          if (D.part == 0) ((double *)(U.scr + U.L.T))[q] = ps93_result(S, V, k);
        }
      }
      lev = xs();
      cnt = 0;
      k++;
      lvEnd = k < 0 ? 3 : c93_lvEnd[k];  // k <= the level count, inside the 32-entry table
      const unsigned act = __ballot_sync(0xffffffffu, !done && D.part == 0);
      n = __popc(act);
      if (n == 0) return;
      const LaneDeal N = deal_lanes(n);
      if (N.P != D.P) {  // the running quadratures move to the first lanes
        if (!done && D.part == 0) quad[__popc(act & ((1u << lane) - 1u))] = lane;
        __syncwarp();
        const int src = N.rank < n ? quad[N.rank] : 0;
        __syncwarp();
        D = N;
        done = D.rank >= n;
        q = __shfl_sync(0xffffffffu, q, src);
        at = __shfl_sync(0xffffffffu, at, src);
        S.I = from_lane(S.I, src);
        S.p = from_lane(S.p, src);
        S.q = from_lane(S.q, src);
      }
    }
  }
  if (!done && D.part == 0) {
    atomicOr((unsigned *)(U.scr + U.L.mask) + (q >> 5), 1u << (q & 31));
  }
}

// One warp a CTA; each takes up to J.take entries of the type-1 groups, then
// of the type-2 batches (one kind of work at a time on the whole GPU).
// Bound by instruction latency: 56 % of the issue slots at 16 warps an SM, the
// stalls fixed latencies (1.9 warps an issue), table rows from L2 (1.4) and
// instruction fetch (0.5); the FP64 pipe is 6 % busy.  80 registers let 24 CTAs
// share an SM (at 96 the cluster's stages took 46.5 instead of 45.3 ms, at 64
// 45.8, with spills).  8 centres of the cluster: 1.55 ms (2.46 with doubles and
// per-entry set-up).
template <bool kMixed>
__global__ void __launch_bounds__(32, 24) k_unit_small(DevJob J) {
  extern __shared__ double sm[];
  __shared__ LevelTab V;
  level_tab(V, c93_3n, c93_nLevels, J.tol);
  const SmallSmem L = small_layout(J.maxLBS, J.t2Rows, J.gcap);
  const int n0 = (int)J.counters[kCntT1], n1 = n0 + (int)J.counters[kCntRest], n = n1 + (int)J.counters[kCntT2];
#pragma unroll 1
  for (int taken = 0; taken < J.take; taken++) {
    const int i = next_item(J.counters + kHeadSmall);
    if (i >= n) return;
    const int2 it = small_entry(J, i, n0, n1);
    const Unit &U = unit_get(J, it.x);
    if (i >= n1) {
      t2_small(J, U, V, (u64 *)(sm + L.tab), (int *)(sm + L.quad), it.y);
      continue;
    }
    const long long t0 = J.classCycles ? clock64() : 0;
    const int p0 = it.y & 1023, G = (it.y >> 10) & 63, kind = it.y >> 16;
    if (kind == kPairNormal) t1_small<kMixed, kPairNormal>(J, U, L, sm, V, it.x, p0, G);
    else if (kind == kPairBand) t1_small<kMixed, kPairBand>(J, U, L, sm, V, it.x, p0, G);
    else t1_small<kMixed, kPairZero>(J, U, L, sm, V, it.x, p0, G);
    if (J.classCycles && threadIdx.x == 0) atomicAdd(&J.classCycles[U.cls], (u64)(clock64() - t0));
  }
}

// --------------------------------------------------- stage 3: the large grid

// The large-grid quadratures of one primitive pair whose small-grid ones
// (mask, by t1_index) failed (src/type1.c:149-196), one per lane.
template <bool kMixed>
static __device__ void t1_large(const DevJob &J, const Unit &U, const LargeSmem &Ls, double *sm, const LevelTab &V,
                                int kk, bool ffp, unsigned mask, double s) {
  double *tab = sm + Ls.tab + (threadIdx.x >> 5) * Ls.tabT1;
  int *quad = (int *)(sm + Ls.fail) + (threadIdx.x >> 5) * 32;  // the running quadratures, by rank
  const int lane = threadIdx.x & 31, lab = U.lab, lq = lab + 1, O = kSmallOrder, OL = J.largeOrder, TSf = 3 + 2 * lq;
  const int ws = U.ws, we = U.we, c = U.c, Lc = U.Lc;
  const double *uL = J.uL + (size_t)c * O;
  const bool fail = mask >> lane & 1u;
  int l1 = 0, l2 = 0;
  {
    int rem = lane;
    while (l1 <= lab && rem >= l1 / 2 + 1) { rem -= l1 / 2 + 1; l1++; }
    l2 = l1 - 2 * rem;
  }
  const PairRec &P = ((const PairRec *)(U.scr + U.L.pair))[kk];
  const double z = P.z, zd2 = P.zd2, C2 = P.C2;
  const double2 map = ((const double2 *)(U.scr + U.L.map))[kk];
  const double i1 = map.x, i2 = map.y;
  const ff C2f = ff_from_double(C2), sf = ff_from_double(s), i1f = ff_from_double(i1);
  const int nb = ((const int4 *)(U.scr + U.L.win))[kk].w;
  const int end = nb - 1;
  double I2 = 0, p2 = 0, q2 = 0, res2 = 0;  // double-single sums (mixed path)
  Psm92 S;
  bool done2 = !fail;
  int k = -1, lvEnd = 1;
#pragma unroll 1
  for (int s0 = 0; s0 < OL;) {
    const int s1 = step_end92(s0) < OL ? step_end92(s0) : OL;
    // the rows the quadratures still running read
    const int kq = __reduce_max_sync(0xffffffffu, done2 ? 0 : l2);
    const int rq = __reduce_max_sync(0xffffffffu, done2 ? 0 : l1);
    bool any = false;  // the lane's slot has an entry that is not zero
    if (s0 + lane < s1) {
      const int t = s0 + lane;
      int n = __ldg(J.s92 + t);
      bool upper = t > 0 && ((t - 1) & 1);
      // (mixed path's double-single entries: K_l rows, then w * C2 U_L e^(..) r^l)
      double *K = tab + (t - s0) * TSf, *WR = K + lq;
      const double w = J.wLarge[n] * i1;
      if (n < nb && !(upper && n > end)) {
        double r = i1 * J.xLarge[n] + i2, ex = (z * r + s) * r + zd2;
        if (ex >= J.lnAcc1) {
          if (kMixed && ffp) {
            ff *Kf = (ff *)K, *WRf = (ff *)WR;
            const ff rf = ff_from_double(r);
            ff v = ff_mul(ff_mul(J.wLf[n], i1f),
                          ff_mul(C2f, ff_mul(channel_ff(J, c, Lc, rf), ff_exp(ff_from_double(ex)))));
            any = v.hi != 0.0f;
            bessel_ff(J, kq, ff_mul(sf, rf), Kf, 1);
            WRf[0] = v;
#pragma unroll 1
            for (int l = 1; l <= rq; l++) {
              v = ff_mul(v, rf);
              WRf[l] = v;
            }
          } else {
            const EntInfo info = t1_large_entry(J, c, Lc, r, ex, w, C2, s, kq, rq, (u64 *)K, (u64 *)WR);
            *(EntInfo *)(K + 2 * lq) = info;
            any = info.e != kNoEntry.e;
          }
        }
      } else if (__builtin_expect(n != nb && !upper && n < O && n >= ws && n < we, 0)) {
        // beyond the break the reference integrates its small-grid buffers:
        // exponent and U_L at index n, r^l and K_l at flat offset l*OL + n of
        // rows written with the small grid's stride
        double rs = J.xSmall[n], es = (z * rs + s) * rs;
        if (es >= J.lnAcc1) {
          const double v = w * (C2 * uL[n] * fast_exp(es));
          any = v != 0.0;
#pragma unroll 1
          for (int l = 0; l <= lab; l++) {
            int f = l * OL + n, lr = f / O, nr = f % O;
            bool ok = lr <= lab && nr >= ws && nr < we;
            double xr = J.xSmall[nr], pw = 1.0;
#pragma unroll 1
            for (int i = 0; i < lr && ok; i++) pw = xr * pw;
            const double wr = ok ? v * pw : 0.0, kr = ok ? bessel_row(J, lr, s * xr) : 0.0;
            if (kMixed && ffp) {
              ((ff *)WR)[l] = ff_from_double(wr);
              ((ff *)K)[l] = ff_from_double(kr);
            } else {
              WR[l] = wr;
              K[l] = kr;
            }
          }
          if (!(kMixed && ffp)) *(EntInfo *)(K + 2 * lq) = {kStaleEntry, 0};
        }
      }
      if (kMixed && ffp && !any) {  // zero bits read as 0.0 in ff
#pragma unroll 1
        for (int l = 0; l <= kq; l++) K[l] = 0.0;
#pragma unroll 1
        for (int l = 0; l <= rq; l++) WR[l] = 0.0;
      }
    }
    const unsigned live = __ballot_sync(0xffffffffu, any);
    __syncwarp();
    if (kMixed && ffp) {
      if (!done2) {
        auto vis = [&](int t) { return c92_slot[t] <= end; };
        auto val = [&](int t) {
          const ff *e = (const ff *)(tab + (t - s0) * TSf);
          return ff_mul(e[lq + l1], e[l2]);
        };
        psm92_advance_ff(s0, s1, J.tol, val, vis, I2, p2, q2, done2, res2);
      }
    } else {
      // runs of slots of one level, the lanes dealt to the running
      // quadratures (entries of points that do not count are zero)
      const unsigned act = __ballot_sync(0xffffffffu, !done2);
      const LaneDeal D = deal_lanes(__popc(act));
      const int mine_rank = __popc(act & ((1u << lane) - 1u));
      if (!done2) quad[mine_rank] = l1 | l2 << 16;
      __syncwarp();
      const bool work = D.rank < __popc(act);
      const int qd = work ? quad[D.rank] : 0;
      const int q1 = qd & 0xffff, oW = lq + q1, oK = qd >> 16;
      const EntRow qr = t1_entry_row(q1, oK);
#pragma unroll 1
      for (int t = s0; t < s1;) {
        const int te = lvEnd < s1 ? lvEnd : s1;
        xf_run run;
#pragma unroll 1
        for (int x = t + D.part; x < te; x += D.P)
          if (work && (live >> (x - s0) & 1u)) {
            const u64 *e = (const u64 *)tab + (x - s0) * TSf;
            const EntInfo f = *(const EntInfo *)(e + 2 * lq);
            if (__builtin_expect(f.e == kStaleEntry, 0)) {
              const double a = ((const double *)e)[oW], b = ((const double *)e)[oK];
              run.add(xf_mul(xf_from(a), xf_from(b)), ent_h(a) ^ ent_h(b));
            } else {
              t1_entry_add(run, e[oW], e[oK], f, qr);
            }
          }
        xs sum = combine(run.sum(), D.P);
        S.I = xs_plus(S.I, from_lane(sum, (mine_rank * D.P) & 31));
        t = te;
        if (t < lvEnd) break;
        if (k < 0) psm92_head(S);
        else if (!done2 && psm92_end(S, V, k)) {
          done2 = true;
          res2 = psm92_result(S, V, k);
        }
        k++;
        lvEnd = c92_lvEnd[k];  // k <= the level count, inside the 32-entry table
      }
    }
    __syncwarp();
    s0 = s1;
    if (__all_sync(0xffffffffu, done2)) break;
  }
  if (fail) {
    if (!done2) {
      res2 = kMixed && ffp ? 16 * I2 / c92_3N[c92_nLevels - 1] : psm92_result(S, V, c92_nLevels - 1);
      atomicOr(&((UnitHead *)U.scr)->warn, 1);
    }
    ((double *)(U.scr + U.L.Q))[(size_t)kk * t1_items(lab) + lane] = res2;
  }
  __syncwarp();
}

template <int kWarps>
static __device__ inline void cta_sync() {
  if constexpr (kWarps > 1) __syncthreads();
  else __syncwarp();
}

// Whose tables a slot past a pair's break reads: the last earlier pair whose loop
// reached the point n (-1: none, or it broke off there), and its bra primitive.
struct StalePair {
  int owner, i;
};
static __device__ __noinline__ StalePair stale_pair(const int4 *win, int k, int n, int Nb) {
#pragma unroll 1
  for (int j = k - 1; j >= 0; j--)
    if (win[j].x >= n) return {win[j].x == n ? -1 : j, j / Nb};
  return {-1, 0};
}

// -(za (dA - r)^2 + zb (dB - r)^2) in Q53, saturating.
static __device__ __noinline__ i64 t2_exponent(double za, double zb, double dA, double dB, double r) {
  u64 E = 0;
#pragma unroll 1
  for (int side = 0; side < 2; side++) E += fx_gauss(side ? zb : za, (side ? dB : dA) - r);
  return -(i64)E;
}
// A slot's rows K_l1 and K_l2 as normalised mantissas and exponents; returns their
// common factors (large arguments).
static __device__ __noinline__ xf t2_bessel(const DevJob &J, double za, double zb, double dA, double dB, double r,
                                            u64 *Ka, u64 *Kb, short *Ea, short *Eb, int la, int lb) {
  xf f = {1ull << 63, -63};
#pragma unroll 1
  for (int side = 0; side < 2; side++) {
    const xf z = xf_mul(xf_from(side ? zb : za), xf_from(side ? dB : dA));  // 2 zeta d r: exponent + 1
    u64 *K = side ? Kb : Ka;
    short *E = side ? Eb : Ea;
    const xf c = fx_bessel(J.besX, J.besXA, J.besHL + 1, side ? lb : la,
                           xf_mul(xf_times100({z.m, z.e + 1}), xf_from(r)), [&](int l, u64 v, int scale) {
                             const xf k = xf_norm({v, -scale});
                             K[l] = k.m;
                             E[l] = (short)k.e;
                           });
    f = norm1(xf_mul(f, c));
  }
  return f;
}

// One primitive pair of the type-2 large-grid fallback, by the CTA's one or two
// warps (src/type2.c:418-528): integrates the pass's failed items (decoded in
// `fail`) and adds each result to the partial sums.  mb: the latest break of
// the earlier pairs, beyond which no earlier pair's buffers are reused.  Two
// warps share the tables (one the Bessel rows, the other the potential and the
// powers) and halve the items; each keeps the queue of slots for itself.
constexpr short kNoExp = -32000;  // the exponent of a sum without terms
static __device__ inline short exp16(int e) { return (short)(e < kNoExp ? kNoExp : e); }
struct T2Pass {
  int nf;            // failed items of the pass
  unsigned mask;     // channels they read
  int l1, l2, l3;    // highest Ka, Kb and r^l rows
};
template <int kWarps>
static __device__ void t2_pair(const DevJob &J, const Unit &U, const LargeSmem &L, double *sm, const LevelTab &V,
                               const T2Pass &S0, int k, int mb, const double2 *map, const int4 *win, int &warn) {
  const int lane = threadIdx.x & 31, warp = kWarps > 1 ? threadIdx.x >> 5 : 0, nA = 2 * J.maxLBS + 1, Nb = U.Nb, c = U.c, nf = S0.nf;
  const int LE = J.maxLECP > 0 ? J.maxLECP : 1, LBE = J.maxLBS + LE, OL = J.largeOrder;
  const int TS = L.tabStride, ES = L.expStride;
  const double *pzA = U.pzA, *pzB = U.pzB;
  const double dAC = U.gA[3], dBC = U.gB[3];
  double *tab = sm + L.tab, *part = sm + L.part;
  // an item's state: three mantissas and the exponents, 16 bits each
  i64 *s0m = (i64 *)(sm + L.I), *s1m = (i64 *)(sm + L.P), *s2m = (i64 *)(sm + L.Q);
  short4 *sE = (short4 *)(sm + L.E);
  const int *fail = (const int *)(sm + L.fail);
  unsigned char *act = (unsigned char *)(sm + L.act) + warp * (kWalkCap / 2);  // the warp's running items
  int *pend = (int *)(sm + L.pend) + warp * 64;
  int *red = (int *)(sm + L.red);
  (void)red;
  // derivative blocks: the product times zeta_a^max(0, shifta), zeta_b^max(0, shiftb)
  // (src/type2.c:456-462)
  const PairRec &P = ((const PairRec *)(U.scr + U.L.pair))[k];
  const double za = P.za, zb = P.zb, Ck = P.C2;
  const double i1 = map[k].x;
  const double iCk = i1 * Ck;
  const int4 wk = win[k];
  const int nb = wk.x, nLo = wk.y, nHi = wk.z;
#pragma unroll 1
  for (int i = lane; i * kWarps + warp < nf; i += 32) {
    const int q = i * kWarps + warp;
    act[i] = (unsigned char)q;
    s0m[q] = s1m[q] = s2m[q] = 0;
    sE[q] = make_short4(kNoExp, kNoExp, kNoExp, 0);
  }
  __syncwarp();
  // Whose tables slot t reads (the reference's reused buffers): this pair's
  // below its break; beyond it, on the lower half, the last earlier pair
  // whose loop reached that point; and the point, exponent of that pair.
  auto locate = [&](int t, int &owner, double &r, double &zaj, double &zbj) {
    const int n = __ldg(J.s92 + t);
    const bool upper = t > 0 && ((t - 1) & 1);
    owner = k;
    zaj = za;
    zbj = zb;
    if (__builtin_expect(n >= nb, 0)) {
      const StalePair p = n != nb && !upper ? stale_pair(win, k, n, Nb) : StalePair{-1, 0};
      owner = p.owner;
      if (owner < 0) return;
      zaj = pzA[p.i];
      zbj = pzB[owner - p.i * Nb];
    }
    r = map[owner].x * J.xLarge[n] + map[owner].y;
  };
  auto exponent = [&](double zaj, double zbj, double r) { return t2_exponent(zaj, zbj, dAC, dBC, r); };
  const i64 thr = fx_q53(J.lnAcc2);
  // A slot needs its tables only where they are not negligible; the others
  // integrate to exactly zero.  Slots are classified step by step (cheap),
  // the needed ones queued, and each pass evaluates 32 queued slots, one per
  // lane, before the quadratures walk every slot up to the first one still
  // queued.
  int cpos = 0, wpos = 0, nPend = 0, nAct = (nf + kWarps - 1 - warp) / kWarps;
  // channels and rows the quadratures still running read (the pass's to
  // begin with, narrowed after every walk)
  unsigned pMask = S0.mask;
  int pL1 = S0.l1, pL2 = S0.l2, pL3 = S0.l3;
  const unsigned below = (1u << lane) - 1u;
  while (wpos < OL) {
    while (nPend < 32 && cpos < OL) {
      const int c1 = step_end92(cpos) < OL ? step_end92(cpos) : OL, t = cpos + lane;
      bool need = false;
      if (t < c1) {
        const int n = __ldg(J.s92 + t);
        if (n < nb) {
          // this pair's own point: the exponent passes inside its interval
          need = n >= nLo && n <= nHi;
        } else if (n <= mb && n != nb && !(t > 0 && ((t - 1) & 1))) {
          int owner;
          double r, zaj, zbj;
          locate(t, owner, r, zaj, zbj);
          need = owner >= 0 && exponent(zaj, zbj, r) >= thr;
        }
      }
      const unsigned m = __ballot_sync(0xffffffffu, need);
      if (need) pend[nPend + __popc(m & below)] = t;
      nPend += __popc(m);
      cpos = c1;
    }
    __syncwarp();
    // this pass: the first queued slots, and the walk's end
    const int nE = nPend < 32 ? nPend : 32, b = nPend > 32 ? pend[32] : cpos;
    if (lane < nE) {
      const int t = pend[lane], n = __ldg(J.s92 + t);
      int owner;
      double r, zaj, zbj;
      locate(t, owner, r, zaj, zbj);
      double *e = tab + lane * TS;
      xf f = {1ull << 63, -63};  // the Bessel rows' common factors (large arguments)
      // the Bessel rows of both centres, then the rest: a warp each, or both by one
#pragma unroll 1
      for (int role = warp; role < 2; role += kWarps) {
        // mantissas of w Ck e^ex U_l, r^l, K_l1 and K_l2, the
        // exponents in 16 bits, U's with its sign
        u64 *Um = (u64 *)e, *R = Um + LE, *Ka = R + nA, *Kb = Ka + LBE;
        short *Ue = (short *)(tab + 32 * TS) + lane * ES, *Ae = Ue + LE, *Be = Ae + LBE, *Re = Be + LBE;
        const xf Rx = xf_from(r);
        if (role == 0) {
          f = t2_bessel(J, zaj, zbj, dAC, dBC, r, Ka, Kb, Ae, Be, pL1, pL2);
          if constexpr (kWarps > 1) {  // the other warp has the potential
#pragma unroll 1
            for (int l = 0; l <= pL2; l++) {
              const xf v = norm1(xf_mul({Kb[l], Be[l]}, f));
              Kb[l] = v.m;
              Be[l] = (short)v.e;
            }
          }
          continue;
        }
        const double w = J.wLarge[n] * iCk;
        xf wB = xf_mul(fx_exp(exponent(zaj, zbj, r)), xf_from(w));
        if constexpr (kWarps == 1) wB = xf_mul(norm1(wB), f);
        wB = xf_norm(wB);
        // only the channels and rows this pass's quadratures read
#pragma unroll 1
        for (unsigned m = pMask; m; m &= m - 1u) {
          const int l = __ffs(m) - 1;
          uint32_t sign;
          const xf u = norm1(xf_mul(channel(J, c, l, r, sign), wB));
          sign ^= sign_of(w);
          Um[l] = u.m;
          Ue[l] = (short)((u.m && u.e > -16000 ? u.e * 2 : -32000) + (int)(sign >> 31));
        }
        xf p = {1ull << 63, -63};
        R[0] = p.m;
        Re[0] = (short)p.e;
#pragma unroll 1
        for (int l = 1; l <= pL3; l++) {
          p = norm1(xf_mul(p, Rx));
          R[l] = p.m;
          Re[l] = (short)p.e;
        }
      }
    }
    const int myPend = lane < nE ? pend[lane] : INT_MAX;
    cta_sync<kWarps>();
    unsigned nMask = 0u;
    int n1 = 0, n2 = 0, n3 = 0, left = 0;
    // the running items, 32 at a time, the last ones by several lanes each
#pragma unroll 1
    for (int i0 = 0; i0 < nAct;) {
      const LaneDeal D = deal_lanes(nAct - i0);
      const bool work = i0 + D.rank < nAct;
      const int q = work ? act[i0 + D.rank] : 0;
      // the pass's item, decoded once when the pass was listed
      const int v = fail[q], l = v & 255, l1 = (v >> 8) & 255, l2 = (v >> 16) & 255, l3 = v >> 24;
      bool done = !work;
      double res = 0;
      const short4 e = sE[q];
      Psm92 S;
      S.I = {s0m[q], e.x};
      S.I1 = {s1m[q], e.y};
      S.I2 = {s2m[q], e.z};
      const u64 *eU = (const u64 *)tab + l, *eR = (const u64 *)tab + LE + l3, *eA = (const u64 *)tab + LE + nA + l1,
                *eB = (const u64 *)tab + LE + nA + LBE + l2;
      const short *xT = (const short *)(tab + 32 * TS);
      const int xA = LE + l1, xB = LE + LBE + l2, xR = LE + 2 * LBE + l3;
      int i = 0, pos = wpos, k = wpos == 0 ? -1 : level_of(wpos);
#pragma unroll 1
      while (pos < b) {
        const int lvE = k < 0 ? 1 : c92_lvEnd[k];
        pos = lvE < b ? lvE : b;
        const int ie = __popc(__ballot_sync(0xffffffffu, myPend < pos));
        xf_run run;
#pragma unroll 1
        for (int x = i + D.part; x < ie; x += D.P) {
          const short *xe = xT + x * ES;
          const int ue = xe[l];
          run.add({mul_hi(mul_hi(eA[x * TS], eB[x * TS]), mul_hi(eU[x * TS], eR[x * TS])),
                   (ue >> 1) + xe[xA] + xe[xB] + xe[xR] + 3 * 64},
                  (uint32_t)ue << 31);
        }
        i = ie;
        S.I = xs_plus(S.I, combine(run.sum(), D.P));
        if (pos == lvE) {
          if (k < 0) psm92_head(S);
          else if (!done && psm92_end(S, V, k)) {
            done = true;
            res = psm92_result(S, V, k);
          }
          k++;
        }
        if (__all_sync(0xffffffffu, done)) break;
      }
      __syncwarp();
      if (work && D.part == 0) {
        s0m[q] = done ? __double_as_longlong(res) : S.I.m;
        s1m[q] = S.I1.m;
        s2m[q] = S.I2.m;
        sE[q] = make_short4(exp16(S.I.e), exp16(S.I1.e), exp16(S.I2.e), 0);
      }
      if (!done) {
        nMask |= 1u << l;
        n1 = l1 > n1 ? l1 : n1;
        n2 = l2 > n2 ? l2 : n2;
        n3 = l3 > n3 ? l3 : n3;
      }
      // keep the items still running (the list shrinks in place); a finished
      // one adds its result
      const bool keep = work && D.part == 0 && !done;
      const unsigned km = __ballot_sync(0xffffffffu, keep);
      if (work && D.part == 0 && done) part[q] += res;
      __syncwarp();
      if (keep) act[left + __popc(km & below)] = (unsigned char)q;
      left += __popc(km);
      i0 += 32 / D.P;
      __syncwarp();
    }
    nAct = left;
    pMask = __reduce_or_sync(0xffffffffu, nMask);
    pL1 = __reduce_max_sync(0xffffffffu, n1);
    pL2 = __reduce_max_sync(0xffffffffu, n2);
    pL3 = __reduce_max_sync(0xffffffffu, n3);
    // both warps' channels (the low byte) and rows, and the end of their walks
    if constexpr (kWarps > 1) {
      if (lane == 0) red[warp] = (int)(pMask | (unsigned)pL1 << 8 | (unsigned)pL2 << 16 | (unsigned)pL3 << 24);
      cta_sync<kWarps>();
      const unsigned o = (unsigned)red[warp ^ 1];
      pMask |= o & 255u;
      pL1 = pL1 > (int)(o >> 8 & 255u) ? pL1 : (int)(o >> 8 & 255u);
      pL2 = pL2 > (int)(o >> 16 & 255u) ? pL2 : (int)(o >> 16 & 255u);
      pL3 = pL3 > (int)(o >> 24) ? pL3 : (int)(o >> 24);
    }
    // drop the evaluated slots from the queue
    const int rest = nPend - nE;
    const int keep0 = lane < rest ? pend[nE + lane] : 0, keep1 = lane + 32 < rest ? pend[nE + lane + 32] : 0;
    __syncwarp();
    if (lane < rest) pend[lane] = keep0;
    if (lane + 32 < rest) pend[lane + 32] = keep1;
    nPend = rest;
    wpos = b;
    __syncwarp();
    if (pMask == 0u) break;  // no quadrature running
  }
  // out of levels: the full-grid estimate stands and the unit is flagged
#pragma unroll 1
  for (int i = lane; i < nAct; i += 32) {
    const int q = act[i];
    Psm92 S;
    S.I1 = {s1m[q], sE[q].y};
    part[q] += psm92_result(S, V, c92_nLevels - 1);
    warn = 1;
  }
  __syncwarp();
}

// The failed type-2 quadratures of a unit over the primitive pairs of one part
// (src/type2.c:418-528), in passes of up to kWalkCap of them.
template <int kWarps>
static __device__ void t2_large(const DevJob &J, const Unit &U, const LargeSmem &L, double *sm, const LevelTab &V,
                                int part) {
  const int lane = threadIdx.x & 31, nIt = U.nItems, LE = J.maxLECP > 0 ? J.maxLECP : 1;
  const unsigned *mask = (const unsigned *)(U.scr + U.L.mask);
  int *fail = (int *)(sm + L.fail);
  double *sum = sm + L.part;
  const int pp = t2_part_pairs(U.NP, J.single), k0 = part * pp, k1 = k0 + pp < U.NP ? k0 + pp : U.NP;
  const bool single = t2_parts(U.NP, J.single) == 1;
  // partial sums of the part, or the results themselves when it is the only one
  double *dst = single ? (double *)(U.scr + U.L.T)
                       : (double *)(U.scr + U.L.part) + (size_t)part * class_items(J, U.cls * LE, LE);
  const double2 *map = (const double2 *)(U.scr + U.L.map);
  const int4 *win = (const int4 *)(U.scr + U.L.win);
  // the latest break of the pairs before the part: beyond it no earlier
  // pair's buffers are reused
  int mb0 = -1;
#pragma unroll 1
  for (int j = lane; j < k0; j += 32) mb0 = win[j].x > mb0 ? win[j].x : mb0;
  mb0 = __reduce_max_sync(0xffffffffu, mb0);
  int q0 = 0;
  while (q0 < nIt) {
    // the pass's items, decoded once
    int nf = 0;
    unsigned pMask = 0;
    int m1 = 0, m2 = 0, m3 = 0;
    const int first = q0;
#pragma unroll 1
    for (; q0 < nIt; q0 += 32) {
      const unsigned m = mask[q0 >> 5];
      if (nf + __popc(m) > kWalkCap) break;
      if (m >> lane & 1u) {
        const int v = unit_item(J, U, q0 + lane);
        if (threadIdx.x < 32) fail[nf + __popc(m & ((1u << lane) - 1u))] = v;
        pMask |= 1u << (v & 255);
        m1 = m1 > ((v >> 8) & 255) ? m1 : (v >> 8) & 255;
        m2 = m2 > ((v >> 16) & 255) ? m2 : (v >> 16) & 255;
        m3 = m3 > (v >> 24) ? m3 : v >> 24;
      }
      nf += __popc(m);
    }
    if (nf == 0) continue;
    T2Pass S;
    S.nf = nf;
    S.mask = __reduce_or_sync(0xffffffffu, pMask);
    S.l1 = __reduce_max_sync(0xffffffffu, m1);
    S.l2 = __reduce_max_sync(0xffffffffu, m2);
    S.l3 = __reduce_max_sync(0xffffffffu, m3);
#pragma unroll 1
    for (int q = threadIdx.x; q < nf; q += blockDim.x) sum[q] = 0.0;
    cta_sync<kWarps>();
    int mb = mb0, warn = 0;
#pragma unroll 1
    for (int k = k0; k < k1; k++) {
      t2_pair<kWarps>(J, U, L, sm, V, S, k, mb, map, win, warn);
      mb = win[k].x > mb ? win[k].x : mb;
    }
    if (warn) atomicOr(&((UnitHead *)U.scr)->warn, 2);
    cta_sync<kWarps>();
    int at = 0;
#pragma unroll 1
    for (int w = first; w < q0; w += 32) {
      const unsigned m = mask[w >> 5];
      if (threadIdx.x < 32 && (m >> lane & 1u)) dst[w + lane] = sum[at + __popc(m & ((1u << lane) - 1u))];
      at += __popc(m);
    }
    cta_sync<kWarps>();
  }
}

// The type-2 parts first (the longer ones), one at a time by the whole CTA, then
// the failed type-1 pairs, one a warp.  Bound by instruction latency like the
// small grid: 48 % of the issue slots at 13 warps an SM, fixed latencies 2.0
// warps an issue, table rows 1.5, fetch 0.4, FP64 pipe 4 %.  128 registers and the
// tables' shared memory admit 14 to 16 warps; fewer registers spill in the walks
// (18 warps: 48.8 against 46.5 ms on the cluster), two Bessel rows or two walk
// entries at a time overflow the instruction cache (39.6 and 39.7 against 37.4).
// 8 centres of the cluster: 3.27 ms.
template <bool kMixed, int kWarps>
__global__ void __launch_bounds__(32 * kWarps, 16 / kWarps) k_unit_large(DevJob J) {
  extern __shared__ double sm[];
  __shared__ LevelTab V;
  __shared__ int drawn;
  (void)drawn;
  level_tab(V, c92_3N, c92_nLevels, J.tol);
  const LargeSmem L = large_layout(J.maxLBS, J.maxLECP, false);
  const int n2 = (int)J.counters[kCntPart], n = n2 + (int)J.counters[kCntFail];
  int i = n2, taken = 0;
#pragma unroll 1
  for (; taken < J.take; taken++) {
    if constexpr (kWarps > 1) {
      if (threadIdx.x == 0) drawn = (int)atomicAdd(J.counters + kHeadLarge, 1u);
      __syncthreads();
      i = drawn;
      __syncthreads();
    } else {
      i = next_item(J.counters + kHeadLarge);
    }
    if (i >= n2) break;
    const int2 it = J.listPart[i];
    const Unit &U = unit_get(J, it.x);
    t2_large<kWarps>(J, U, L, sm, V, it.y);
  }
#pragma unroll 1
  for (; taken < J.take; taken++, i = n) {
    // (the first warp goes on with the entry drawn above)
    if (i >= n || threadIdx.x >= 32) i = next_item(J.counters + kHeadLarge);
    if (i >= n) return;
    const T1Fail it = J.listFail[i - n2];
    const Unit &U = unit_get(J, it.off);
    t1_large<kMixed>(J, U, L, sm, V, it.k & 0xffff, it.k >> 16, it.mask, it.s);
  }
}

// -------------------------------------------------------- stage 4: the blocks

// One unit a CTA (in small jobs one of its blocks): the type-1 block from the quadratures of its primitive
// pairs (src/type1.c:323-345), the type-2 block from its radial table
// (src/type2.c:583-623), both shifted onto A and B (src/util.c:247-334).  Bound by
// the FP64 pipe (69 % busy) and the barriers between its short phases; 44 KB of
// shared memory at g shells let five CTAs share an SM (61 KB, three CTAs: the
// 150-shell sweep's stages took 50.6 instead of 47.9 ms).  8 centres of the
// cluster: 0.39 ms.
__global__ void __launch_bounds__(kLinkThreadsMax) k_unit_link(DevJob J) {
  extern __shared__ double sm[];
  int pos = J.chunk0 + blockIdx.x;
  if (J.live) {
    const int l0 = J.liveStart[J.chunk];
    if (l0 + (int)blockIdx.x >= J.liveStart[J.chunk + 1]) return;
    pos = J.live[l0 + blockIdx.x];
  }
  const Unit U = unit_load(J, pos);
  if (!U.live) return;
  const LinkSmem Lm = link_layout(J.maxLBS, J.maxLECP);
  const bool one = blockIdx.y == 0, two = blockIdx.y == gridDim.y - 1;  // the blocks this CTA makes
  const int tid = threadIdx.x, NT = blockDim.x, lab = U.lab, lq = lab + 1, Nb = U.Nb;
  double *rsh = sm + Lm.rsh, *dir = sm + Lm.dir, *W = sm + Lm.W, *H = sm + Lm.H;
  const int dd = J.tmDim + 1, tmW = (J.tmDim + 1) * (J.tmDim + 1), RQ = lq * lq, nq = t1_items(lab);
  // type 1: W[L][l][m] = sum over the primitive pairs of S_lm Q[L][l] (the
  // pairs in order), then H[p] = sum_lm poly2sph[p][lm] W[|p|][l][m]: the
  // angular coefficients once per unit instead of once per pair
  if (one) {
    const double *Q = (const double *)(U.scr + U.L.Q);
    const int nW = NCUM(lab);  // sum over L of (L+1)(L+2)/2 entries (l, m)
#pragma unroll 1
    for (int e = tid; e < nW; e += NT) W[e] = 0.0;
#pragma unroll 1
    for (int b0 = 0; b0 < U.NP; b0 += kLinkBatch) {
      const int nb = U.NP - b0 < kLinkBatch ? U.NP - b0 : kLinkBatch;
      __syncthreads();
      if (tid < nb) {
        const int k = b0 + tid;
        const double za = U.pzA[k / Nb], zb = U.pzB[k % Nb];
        double P[3];
        for (int i = 0; i < 3; i++) P[i] = 2.0 * (za * U.gA[i] + zb * U.gB[i]);
        direction(P, dir[3 * tid], dir[3 * tid + 1], dir[3 * tid + 2]);
      }
      __syncthreads();
#pragma unroll 1
      for (int e = tid; e < nb * lq; e += NT) {
        const int g = e / lq, m = e % lq;
        rsh_column(J, lab, m, dir[3 * g], dir[3 * g + 1], dir[3 * g + 2], rsh + g * RQ);
      }
      __syncthreads();
#pragma unroll 1
      for (int e = tid; e < nW; e += NT) {
        int Lm1 = 0;
        while (NCUM(Lm1) <= e) Lm1++;
        int r = e - NCUM(Lm1 - 1), l = Lm1;
        while (r >= 2 * l + 1) { r -= 2 * l + 1; l -= 2; }
        const double *q = Q + (size_t)b0 * nq + t1_index(Lm1, l), *s = rsh + l * l + r;
        double v = W[e];
#pragma unroll 4
        for (int g = 0; g < nb; g++) v += s[g * RQ] * q[(size_t)g * nq];
        W[e] = v;
      }
    }
    __syncthreads();
#pragma unroll 1
    for (int pi = tid; pi < nW; pi += NT) {
      const int *ex = J.ijk + 3 * pi;
      const int lmax = ex[0] + ex[1] + ex[2];
      const double *p2s = J.p2s + (size_t)J.ijkIdx[(ex[0] * dd + ex[1]) * dd + ex[2]] * tmW;
      const double *w = W + NCUM(lmax - 1);
      double acc = 0.0;
#pragma unroll 1
      for (int l = lmax; l >= 0; l -= 2) {
#pragma unroll 4
        for (int m = 0; m < 2 * l + 1; m++) acc += p2s[l * l + m] * w[m];
        w += 2 * l + 1;
      }
      H[pi] = acc;
    }
    __syncthreads();
  }
  link_finish<false>(J, U, Lm, sm, one, two);
}

// The screening window and F table of every (shell, centre) -- k_shell_F of
// the drop-in path (src/type2.c:223-310, src/type2.c:149-180) with the
// batched path's Bessel rows and exp; FP64 in every mode.
__global__ void __launch_bounds__(kPointThreads) k_shell_F_fast(DevJob J) {
  __shared__ int sw[3];
  const int s = blockIdx.x, c = blockIdx.y, O = kSmallOrder;
  const int C = J.ctrAtom[c], A = J.shAtom[s];
  const double *rC = J.geom + 3 * C, *rA = J.geom + 3 * A;
  double x = rC[0] - rA[0], y = rC[1] - rA[1], z = rC[2] - rA[2];
  const double dAC = sqrt(x * x + y * y + z * z);
  if (threadIdx.x == 0) shell_window(J, s, c, dAC, sw);
  __syncthreads();
  // run = derivative order of the table: rows up to L - 1 + l + run and
  // coefficients times zeta^run (src/type2.c:229, :263-290)
  const int nF = J.nF, nRuns = J.nRuns > 0 ? J.nRuns : 1;
  const double *pa = J.primA + J.shP[s], *pd = J.primD + J.shP[s];
#pragma unroll 1
  for (int run = 0; run < nRuns; run++) {
    const int lmaxA = J.maxLECP - 1 + J.shL[s] + run;
    double *F = J.F + (((size_t)c * J.nShells + s) * nRuns + run) * O * nF;
    const int n = blockIdx.z * blockDim.x + threadIdx.x;
    if (n < O) {
      double acc[kMaxRows], K[kMaxRows];
#pragma unroll 1
      for (int i = 0; i < nF; i++) acc[i] = 0.0;
      if (!sw[2] && n >= sw[0] && n < sw[1] && lmaxA >= 0) {
        double r = J.xSmall[n];
#pragma unroll 1
        for (int p = 0; p < J.shK[s]; p++) {
          double zeta = pa[p], da = pd[p];
#pragma unroll 1
          for (int k = 0; k < run; k++) da *= zeta;
          double e = dAC - r;
          e = -zeta * e * e;
          const xf v = e > -700.0 ? xf_mul(fx_exp(fx_q53(e)), xf_from(da)) : xf{0, 0};
          if (v.m == 0) continue;
          const xf f = xf_mul(xf_from(zeta), xf_from(dAC));
          bessel_fx(J, lmaxA, xf_mul(xf_times100({f.m, f.e + 1}), xf_from(r)), v, sign_of(da), K);
#pragma unroll 1
          for (int i = 0; i <= lmaxA; i++) acc[i] += K[i];
        }
      }
#pragma unroll 1
      for (int i = 0; i < nF; i++) F[(size_t)n * nF + i] = acc[i];
    }
  }
}

// ---------------------------------------------------------- screening stage

constexpr int kScreenThreads = 256;

// Live units (those that compute blocks: the screened windows of
// src/libecp.c:296-330 and the derivative skips) per CTA chunk of the queue.
__global__ void __launch_bounds__(kScreenThreads) k_screen_count(DevJob J, long long n) {
  const long long i = (long long)blockIdx.x * kScreenThreads + threadIdx.x;
  const int cnt = __syncthreads_count(i < n && unit_live(J, (int)i));
  if (threadIdx.x == 0) J.screenBlocks[blockIdx.x] = cnt;
}

// Exclusive scan of the per-CTA counts (one CTA); the total ends the last chunk.
__global__ void __launch_bounds__(1024) k_screen_scan(DevJob J, int nBlocks) {
  __shared__ int v[1024];
  __shared__ int base;
  if (threadIdx.x == 0) base = 0;
  __syncthreads();
#pragma unroll 1
  for (int b0 = 0; b0 < nBlocks; b0 += 1024) {
    const int b = b0 + threadIdx.x;
    const int x = b < nBlocks ? J.screenBlocks[b] : 0;
    v[threadIdx.x] = x;
    __syncthreads();
    for (int off = 1; off < 1024; off <<= 1) {  // inclusive Hillis-Steele scan
      const int y = threadIdx.x >= off ? v[threadIdx.x - off] : 0;
      __syncthreads();
      v[threadIdx.x] += y;
      __syncthreads();
    }
    if (b < nBlocks) J.screenBlocks[b] = base + v[threadIdx.x] - x;
    __syncthreads();
    if (threadIdx.x == 1023) base += v[1023];
    __syncthreads();
  }
  if (threadIdx.x == 0) J.liveStart[J.nChunks] = base;
}

// Stable compaction of the live units' queue positions; the others are marked
// skipped here.  A chunk's first position notes where its live units start.
__global__ void __launch_bounds__(kScreenThreads) k_screen_scatter(DevJob J, long long n) {
  __shared__ int warpCnt[kScreenThreads / 32];
  const long long i = (long long)blockIdx.x * kScreenThreads + threadIdx.x;
  const bool live = i < n && unit_live(J, (int)i);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned m = __ballot_sync(0xffffffffu, live);
  if (lane == 0) warpCnt[warp] = __popc(m);
  __syncthreads();
  if (i >= n) return;
  int at = J.screenBlocks[blockIdx.x] + __popc(m & ((1u << lane) - 1u));
#pragma unroll 1
  for (int w = 0; w < warp; w++) at += warpCnt[w];
  if (live) J.live[at] = (int)i;
  else J.status[unit_at(J, (int)i)] = kUnitSkipped;
  int k = 0;  // the chunk that starts here, if one does
#pragma unroll 1
  for (int hi = J.nChunks; hi - k > 1;) {
    const int mid = (k + hi) >> 1;
    if (J.chunkUnit[mid] <= (int)i) k = mid; else hi = mid;
  }
  if (J.chunkUnit[k] == (int)i) J.liveStart[k] = at;
}

// --------------------------------------------------------------- launchers

int upload_schedules_fast(const int *s93slot, int s93n, const int *s93lvEnd, const int *s93lvJ,
                          const int *s93lvN, int s93levels, const int *s92slot, int s92n,
                          const int *s92lvEnd, const int *s92lvN, int s92levels, void *stream) {
  if (s93levels > kMaxLevels || s92levels > kMaxLevels) return 1;
  return upload_stage_schedules(s93slot, s93n, s93lvEnd, s93lvJ, s93lvN, s93levels, s92slot, s92n, s92lvEnd, s92lvN,
                                s92levels, stream);
}

void fast_prepare() {
  // function attributes are per device; callers hold the engine lock
  static bool attr[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || attr[dev]) return;
#pragma unroll 1
  for (const void *k : {(const void *)k_unit_small<false>, (const void *)k_unit_small<true>,
                        (const void *)k_unit_large<false, 1>, (const void *)k_unit_large<true, 1>,
                        (const void *)k_unit_large<false, 2>, (const void *)k_unit_large<true, 2>,
                        (const void *)k_unit_link}) {
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    // most of the unified L1/shared array as shared memory
    cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
  }
  attr[dev] = true;
}

int fast_ctas_per_sm(size_t smemBytes) {
  fast_prepare();
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, (const void *)k_unit_small<false>, 32, smemBytes) != cudaSuccess)
    return 0;
  return n;
}

int launch_fast_pipeline(const DevJob &J, cudaStream_t st, const FastConfig &cfg, cudaEvent_t u0, cudaEvent_t u1) {
  fast_prepare();
  DevJob Jc = J;
  Jc.gcap = cfg.gcap;
  Jc.balance = cfg.balance;
#pragma unroll 1
  for (int i = 0; i < kMaxClasses; i++) Jc.classCfg[i] = cfg.cls[i];
  Jc.classCycles = cfg.classCycles;
  const JobPlan::Order &ord = use_order(Jc, cfg.sorted);
  const size_t sSmall = fast_smem_bytes(J.maxLBS, J.t2Rows, cfg.gcap);
  const size_t sLarge = sizeof(double) * (size_t)large_layout(J.maxLBS, J.maxLECP, false).total;
  const size_t sLink = sizeof(double) * (size_t)link_layout(J.maxLBS, J.maxLECP).total;
  if (sSmall > 200 * 1024 || sLarge > 200 * 1024 || sLink > 200 * 1024) return 3;
  const bool screen = cfg.queue && cfg.screen;
  if (!screen) Jc.live = nullptr;
  launch_stage1(Jc, st);
  const int nt = point_threads(J);
  k_shell_F_fast<<<dim3(J.nShells, J.nCentres, (kSmallOrder + nt - 1) / nt), nt, 0, st>>>(Jc);
  const long long nUnits = (long long)J.nCentres * J.nPairs;
  if (screen && nUnits > 0) {  // screening stage: the live units' positions
    const long long nb = (nUnits + kScreenThreads - 1) / kScreenThreads;
    k_screen_count<<<(unsigned)nb, kScreenThreads, 0, st>>>(Jc, nUnits);
    k_screen_scan<<<1, 1024, 0, st>>>(Jc, (int)nb);
    k_screen_scatter<<<(unsigned)nb, kScreenThreads, 0, st>>>(Jc, nUnits);
  }
  if (u0) record_timing(u0, st);
  launch_chunks(Jc, ord, st, [&](const DevJob &C, unsigned units, unsigned gSmall, int takeSmall, unsigned gLarge,
                                 int takeLarge) {
    DevJob K = C;
    k_unit_plan<false><<<(units + 3) / 4, kPlanThreads, 0, st>>>(K);
    K.take = takeSmall;
    if (cfg.mixed) k_unit_small<true><<<gSmall, 32, sSmall, st>>>(K);
    else k_unit_small<false><<<gSmall, 32, sSmall, st>>>(K);
    K.take = takeLarge;
    const int nw = J.twoWarps ? 2 : 1;
    (cfg.mixed ? nw > 1 ? k_unit_large<true, 2> : k_unit_large<true, 1>
               : nw > 1 ? k_unit_large<false, 2> : k_unit_large<false, 1>)<<<gLarge, 32 * nw, sLarge, st>>>(K);
    k_unit_link<<<dim3(units, link_parts(units)), link_threads(sLink), sLink, st>>>(K);
  });
  if (u1) record_timing(u1, st);
  launch_epilogue(Jc, st);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : kLaunchErrorBase + (int)e;
}

}  // namespace ecpgb
