// ecp_device.cuh -- device helpers shared by the kernel translation units.
//
// Included by ecp_fp64.cu (compiled --fmad=false, the drop-in path) and
// ecp_fast.cu (the batched path); each unit gets its own copy of the
// __constant__ level schedules and uploads them itself.
#pragma once
#include <cuda_runtime.h>

#include <climits>
#include <cmath>

#include "ecp_engine.h"
#include "ecp_tables.h"

namespace ecpgb {

#define NCART(l) (((l) + 1) * ((l) + 2) / 2)
#define NCUM(l) (((l) + 1) * ((l) + 2) * ((l) + 3) / 6)

static constexpr double kPi = 3.14159265358979323846;
static constexpr int kMaxRows = 40;   // Bessel rows incl. the 5 Taylor guard rows

static __constant__ int c93_slot[kSmallOrder];
static __constant__ int c93_lvEnd[32], c93_lvJ[32], c93_lvN[32];
static __constant__ int c93_nLevels;
static __constant__ int c92_slot[kMaxLargeOrder];
static __constant__ int c92_lvEnd[32], c92_lvN[32];
static __constant__ int c92_nLevels, c92_order;

// ------------------------------------------------------------ primitives

// K_0..K_lmax(z) = exp(-z) i_l(z) with stride; three branches of
// src/bessel.c:102-199 (small z, 5-term Taylor about the nearest table point,
// asymptotic).  The table is stored transposed: row i holds K_0..K_tabL(z_i).
static __device__ void bessel_eval(const DevJob &J, int lmax, double z, double *K, int stride) {
  if (z < 1.0E-7) {
    if (z <= 0) {
      K[0] = 1.0;
      for (int l = 1; l <= lmax; l++) K[l * stride] = 0.0;
    } else {
      K[0] = 1 - z;
      for (int l = 1; l <= lmax; l++) K[l * stride] = K[(l - 1) * stride] * z / (2 * l + 1);
    }
  } else if (z < 16.0) {
    int top = lmax + 5;
    double d[kMaxRows], prev[kMaxRows];
    double h = J.besselN / 16;  // integer division, as the reference
    int index = (int)floor(z * h + 0.5);
    double dz = z - index / h, scale = 1.0;
    const double *row = J.besT + (size_t)index * (J.tabL + 1);
    for (int l = 0; l <= top; l++) d[l] = row[l];
    for (int l = 0; l <= lmax; l++) K[l * stride] = d[l];
    for (int i = 1; i <= 5; i++) {
      int ti = top - i;
      for (int j = 0; j <= ti + 1; j++) prev[j] = d[j];
      d[0] = prev[1] - prev[0];
      for (int j = 1; j <= ti; j++)
        d[j] = J.besC[j] * (prev[j - 1] - prev[j + 1]) - prev[j] + prev[j + 1];
      scale = scale * dz / i;
      for (int j = 0; j <= lmax; j++) K[j * stride] += scale * d[j];
    }
  } else {
    double A[kMaxRows];
    A[0] = 0.5 / z;
    for (int l = 0; l <= lmax; l++) K[l * stride] = A[0];
    for (int l = 1; l <= lmax; l++) {
      double f = l * (l + 1);
      for (int i = 1; i < l; i++) {
        K[l * stride] += f * A[i];
        f *= (l + i + 1) * (l - i);
      }
      A[l] = -A[0] * A[l - 1] / l;
      K[l * stride] += f * A[l];
    }
  }
}

// x / l for an integer l, 1 <= l <= 15: the correctly rounded quotient from
// the correctly rounded reciprocal and one residual (Markstein), three
// operations instead of a divide.
static __device__ const double kInvInt[16] = {0.0,     1.0,     1.0 / 2, 1.0 / 3,  1.0 / 4,  1.0 / 5,  1.0 / 6,  1.0 / 7,
                                              1.0 / 8, 1.0 / 9, 1.0 / 10, 1.0 / 11, 1.0 / 12, 1.0 / 13, 1.0 / 14, 1.0 / 15};
static __device__ inline double div_int(double x, double l, double inv) {
  const double q = x * inv;
  return fma(fma(-l, q, x), inv, q);
}

// The products f of the large-argument sum of K_l (src/bessel.c:170-190), as
// exact doubles: [l][i] multiplies A_i.
struct AsyFactors {
  double v[16][16];
  constexpr AsyFactors() : v() {
    for (int l = 1; l < 16; l++) {
      double f = l * (l + 1.0);
      for (int i = 1; i <= l; i++) {
        v[l][i] = f;
        f *= (double)(l + i + 1) * (l - i);
      }
    }
  }
};
static __device__ const AsyFactors kAsyF;

// bessel_eval bit for bit, with the derivative rows D^k K_l(z_i) read from the
// table (J.besD) instead of recomputed by their recurrence: the rows depend on
// the table point only.  ~10 operations a row instead of ~200.
static __device__ __noinline__ void bessel_rows(const DevJob &J, int lmax, double z, double *K) {
  if (z < 1.0E-7 || !J.besD) {
    bessel_eval(J, lmax, z, K, 1);
  } else if (z < 16.0) {
    const double h = J.besselN / 16;  // integer division, as the reference
    const int index = (int)floor(z * h + 0.5);
    const double dz = z - __ldg(J.besZ + index);
    // scale = scale * dz / i; halving and quartering are exact
    const double s1 = dz, s2 = s1 * dz * 0.5, s3 = div_int(s2 * dz, 3.0, 1.0 / 3), s4 = s3 * dz * 0.25,
                 s5 = div_int(s4 * dz, 5.0, 1.0 / 5);
    const double *d = J.besD + (size_t)index * (J.besHL + 1) * 6;
#pragma unroll 1
    for (int l = 0; l <= lmax; l++, d += 6) {
      double v = __ldg(d);
      v += s1 * __ldg(d + 1);
      v += s2 * __ldg(d + 2);
      v += s3 * __ldg(d + 3);
      v += s4 * __ldg(d + 4);
      v += s5 * __ldg(d + 5);
      K[l] = v;
    }
  } else {
    double A[16];
    A[0] = 0.5 / z;
    K[0] = A[0];
#pragma unroll 1
    for (int l = 1; l <= lmax; l++) {
      A[l] = div_int(-A[0] * A[l - 1], l, __ldg(kInvInt + l));
      double v = A[0];
#pragma unroll 1
      for (int i = 1; i <= l; i++) v += __ldg(&kAsyF.v[l][i]) * A[i];
      K[l] = v;
    }
  }
}

// Screening window [start, end) of shell s on centre c's small grid and
// whether the shell is screened out entirely (src/type2.c:149-180), written
// to J.win and to w[3]; dAC = |C - A|.  One thread computes it.
static __device__ void shell_window(const DevJob &J, int s, int c, double dAC, int *w) {
  const int end = J.gridEnd[c];
  const double R = J.radius[s], rmin = dAC - R, rmax = dAC + R;
  // points 0 .. end below rmin, and up to rmax (xSmall ascends)
  int lo = 0, hi = end + 1;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (J.xSmall[mid] < rmin) lo = mid + 1;
    else hi = mid;
  }
  w[0] = lo;
  lo = 0;
  hi = end + 1;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (J.xSmall[mid] <= rmax) lo = mid + 1;
    else hi = mid;
  }
  w[1] = lo - 1;
  w[2] = !(w[1] >= w[0]) || R < 0;
  int *g = J.win + ((size_t)c * J.nShells + s) * 3;
  g[0] = w[0]; g[1] = w[1]; g[2] = w[2];
}

// Derivative shifts (src/libecp.c:240-248), indexed [order][shift].
static __constant__ int c_shiftA[3][10] = {{0}, {+1, -1, 0, 0}, {+2, -2, +1, +1, -1, -1, 0, 0, +1, 0}};
static __constant__ int c_shiftB[3][10] = {{0}, {0, 0, +1, -1}, {0, 0, +1, -1, +1, -1, +2, -2, 0, +1}};

// c times z, n times in a row: the reference's zeta^n derivative factors
// (src/type1.c:239-246, src/type2.c:459-462); n <= 0 leaves c.
static __device__ inline double zeta_times(double c, double z, int n) {
#pragma unroll 1
  for (int k = 0; k < n; k++) c *= z;
  return c;
}

// The derivative shift of pair entry pr and whether the reference computes
// that (shift, centre) combination at all (src/libecp.c:296-330):
// la, lb are the shells' l; A, B their atoms; C the centre's atom.
struct UnitShift {
  int a, b;       // shifta, shiftb
  int lpa, lpb;   // l of the blocks handed out
  bool skip;
};
static __device__ inline UnitShift unit_shift(const DevJob &J, int pr, int la, int lb, int A, int B, int C) {
  UnitShift s{0, 0, la, lb, false};
  if (!J.pairShift || J.deriv <= 0) return s;
  const int k = J.pairShift[pr], d = J.deriv;
  s.a = c_shiftA[d][k];
  s.b = c_shiftB[d][k];
  s.lpa = la + s.a;
  s.lpb = lb + s.b;
  if (d == 2) {  // src/libecp.c:356-362
    if (s.a == 1 && s.b == 0) s.lpa = la;
    else if (s.a == 0 && s.b == 1) s.lpb = lb;
  }
  s.skip = (A == C && B == C) || la + s.a < 0 || lb + s.b < 0 || (d == 1 && C == A && s.a != 0) ||
           (d == 1 && C == B && s.b != 0);
  return s;
}

// r^n for the ECP exponent n (a double in the interface; integers are the norm).
// 0, 1 and 2 are told apart by their bits: a comparison of doubles is an
// instruction of the FP64 pipe.
static __device__ inline double rpow(double r, double n) {
  const long long b = __double_as_longlong(n);
  if (b << 1 == 0) return 1.0;
  if (b == 0x3ff0000000000000ll) return r;
  if (b == 0x4000000000000000ll) return r * r;
  return pow(r, n);
}

// Whether a term D r^n exp(-x) leaves pot as it is, bit for bit: D r^n below 2^u,
// exp(-x) at most 2^-q by x's high word, and the product below a 2^-58th of pot
// (or of the smallest double).  By integers, beside the 20-odd FP64 instructions of
// the exponential that it saves.
static __device__ inline bool ecp_term_lost(double pot, double D, double x, double n, double r, double r2) {
  const unsigned hx = (unsigned)__double2hiint(x), hD = (unsigned)__double2hiint(D) & 0x7fffffffu;
  const long long nb = __double_as_longlong(n);
  if (hx >= 0x7ff00000u || hD >= 0x7ff00000u) return false;  // negative, infinite, NaN
  int u = (int)(hD >> 20) - 1022;
  if (nb == 0x3ff0000000000000ll) u += (__double2hiint(r) >> 20) - 1022;
  else if (nb == 0x4000000000000000ll) u += (__double2hiint(r2) >> 20) - 1022;
  else if (nb << 1 != 0) return false;
  if (u > 1024) return false;  // D r^n may be infinite, and the term NaN
  const int e = (int)(hx >> 20) - 1023;
  const unsigned y = ((hx & 0xfffffu) | 0x100000u) * 1477u;  // log2(e) from below, Q30 2^-e
  const int q = e < 0 ? 0 : e > 10 ? 4096 : (int)(y >> (30 - e));
  return u - q < (__double2hiint(pot) >> 20 & 0x7ff) - 1023 - 58;
}

// U_l(r) of centre c (src/ecp.c:42-60).
static __device__ double eval_ecp(const DevJob &J, int c, int l, double r) {
  double pot = 0.0, r2 = r * r;
  if (J.chanT0) {  // the channel's terms, in order
    const int *ch = J.chanT0 + c * (kMaxLEcp + 2) + l;
#pragma unroll 1
    for (int t = ch[0], t1 = ch[1]; t < t1; t++) {
      const double D = J.termD[t], n = J.termN[t], x = J.termA[t] * r2;
      if (!ecp_term_lost(pot, D, x, n, r, r2)) pot += rpow(r, n) * D * exp(-x);
    }
    return pot;
  }
  int t0 = J.ctrT0[c], t1 = t0 + J.ctrNT[c];
  for (int t = t0; t < t1; t++)
    if (J.termL[t] == l) pot += rpow(r, J.termN[t]) * J.termD[t] * exp(-J.termA[t] * r2);
  return pot;
}

// (r, theta, phi); src/util.c:75-106.
static __device__ void to_spherical(const double *v, double *out) {
  const double eps = 1.0E-14;
  double x = v[0], y = v[1], z = v[2];
  double r = sqrt(x * x + y * y + z * z), th, ph;
  th = (r < eps) ? 0.0 : acos(z / r);
  if (fabs(x) < eps) {
    if (fabs(y) < eps) ph = 0.0;
    else if (y < 0.0) ph = 1.5 * kPi;
    else ph = 0.5 * kPi;
  } else {
    ph = (x > 0.0) ? atan(y / x) : atan(y / x) + kPi;
  }
  out[0] = r; out[1] = th; out[2] = ph;
}

// Real spherical harmonics, index l*l + l + m (m = -l..l);
// src/spherical_harmonics.c:16-114.  lmax <= 12.
static __device__ void real_sph(const DevJob &J, int lmax, double theta, double phi, double *rsh) {
  double P[169], s[14], c[14];
  int n = (lmax + 1) * (lmax + 1);
  for (int i = 0; i < n; i++) P[i] = 0.0;
  for (int i = 0; i < 14; i++) { s[i] = 0.0; c[i] = 0.0; }
#define PL(l, m) P[(l) * (l) + (m) + (l)]
  double x = cos(theta);
  if (1.0 == x) {
    for (int l = 0; l <= lmax; l++) PL(l, 0) = 1.0;
  } else if (-1.0 == x) {
    PL(0, 0) = 1.0;
    for (int l = 1; l <= lmax; l++) PL(l, 0) = -PL(l - 1, 0);
  } else {
    s[1] = sqrt(1.0 - x * x);
    for (int l = 2; l <= lmax; l++) s[l] = s[l - 1] * s[1];
    for (int l = 0; l <= lmax; l++) {
      if (l == 0) { PL(0, 0) = 1.0; continue; }
      PL(l, l) = s[l] * J.dfac[2 * l - 1];
      int m = l - 1;
      PL(l, m) = x * (2 * m + 1) * PL(l - 1, m);
      if (l > 1)
        for (m = 0; m <= l - 2; m++)
          PL(l, m) = (x * (2 * l - 1) * PL(l - 1, m) - (l + m - 1) * PL(l - 2, m)) / (l - m);
    }
  }
  for (int l = 0; l <= lmax; l++) {
    double norm0 = sqrt((2.0 * l + 1.0) / (2.0 * kPi));
    PL(l, 0) = norm0 * PL(l, 0);
    for (int m = 1; m <= l; m++) {
      double norm = sqrt(J.fac[l - m] / J.fac[l + m]) * norm0;
      PL(l, m) = norm * PL(l, m);
    }
  }
  if (lmax > 0) {
    if (0.0 == phi) {
      for (int m = 0; m <= lmax; m++) { s[m] = 0.0; c[m] = 1.0; }
    } else {
      s[1] = sin(phi);
      c[1] = cos(phi);
      for (int m = 2; m <= lmax; m++) {
        s[m] = s[1] * c[m - 1] + c[1] * s[m - 1];
        c[m] = c[1] * c[m - 1] - s[1] * s[m - 1];
      }
    }
  }
  for (int l = 0; l <= lmax; l++) {
    rsh[l * l + l] = PL(l, 0) / sqrt(2.0);
    for (int m = 1; m <= l; m++) {
      rsh[l * l + l - m] = PL(l, m) * s[m];
      rsh[l * l + l + m] = PL(l, m) * c[m];
    }
  }
#undef PL
}

// Column m of real_sph (the entries l = m..lmax of +-m), operation by
// operation, with J.shNorm's normalisation (the same values, tabulated):
// x = cos(theta), and sin, cos of phi.
static __device__ void real_sph_column(const DevJob &J, int lmax, int m, double x, double phi, double sphi, double cphi,
                                       double *rsh) {
  const int W = J.tmDim + 1;
  double sm = 0.0, cm = 1.0;
  if (m > 0 && 0.0 != phi) {
    sm = sphi;
    cm = cphi;
    for (int i = 2; i <= m; i++) {
      const double sn = sphi * cm + cphi * sm, cn = cphi * cm - sphi * sm;
      sm = sn;
      cm = cn;
    }
  }
  const bool pole = 1.0 == x || -1.0 == x;
  double P1 = 0.0, P2 = 0.0;
  for (int l = m; l <= lmax; l++) {
    double P;
    if (pole) P = m > 0 ? 0.0 : l == 0 ? 1.0 : 1.0 == x ? 1.0 : -P1;
    else if (l == 0) P = 1.0;
    else if (l == m) {
      const double s1 = sqrt(1.0 - x * x);
      double s = s1;
      for (int i = 2; i <= m; i++) s = s * s1;
      P = s * J.dfac[2 * l - 1];
    } else if (l == m + 1) P = x * (2 * m + 1) * P1;
    else P = (x * (2 * l - 1) * P1 - (l + m - 1) * P2) / (l - m);
    P2 = P1;
    P1 = P;
    const double v = J.shNorm[l * W + m] * P;
    if (m == 0) rsh[l * l + l] = v / sqrt(2.0);
    else {
      rsh[l * l + l - m] = v * sm;
      rsh[l * l + l + m] = v * cm;
    }
  }
}

// Squared radius where c r^l exp(-zeta r^2) = cutoff; -1 if Newton fails
// (src/util.c:134-172, where the reference asserts).
static __device__ double gto_radius(double c, double zeta, int l, double cutoff) {
  double delta, dg, guess, zr, r;
  const double t = log(fabs(c) / fabs(cutoff));
  dg = t / zeta;
  r = (dg > cutoff) ? dg : cutoff;
  if (l != 0) {
    bool ok = false;
    if (l > 0) {
      dg = sqrt(0.5 * l / fabs(c));
      guess = (dg > cutoff) ? dg : cutoff;
      if (guess > r) r = 0.5 * (r + guess);
    }
    for (int i = 0; i < 40; i++) {
      zr = zeta * r;
      guess = t + l * log(r) - zr * r;
      delta = guess / (l / r - 2 * zr);
      dg = r - delta;
      r = (dg > cutoff) ? dg : cutoff;
      if (fabs(delta) < cutoff) { r *= r; ok = true; break; }
    }
    if (!ok) return -1.0;
  }
  return r;
}

static __device__ inline double binom(const double *fac, int n, int k) {
  return (k >= 0 && k <= n) ? fac[n] / (fac[n - k] * fac[k]) : 0.0;
}

// ------------------------------------------------------------ quadratures

// Adaptive PS93 walk over the small grid (src/gc_integrators.c:157-217):
// `f(n)` is the integrand at abscissa index n; lower-half points count from
// `start`, upper-half points up to `end`; a level that touches no point skips
// the absolute error test.
// rel > 0 (the batched mixed mode only) also accepts a level of at least 63
// points whose error estimate is below rel times the estimate itself; rel = 0
// is the reference's test exactly (the error estimate is never negative).
template <class Fn>
static __device__ bool ps93_walk(const double *w, int start, int end, double tol, double rel, Fn f,
                                 double &res) {
  int mid = c93_slot[0], a = c93_slot[1], b = c93_slot[2];
  double p = w[mid] * f(mid);
  double q = w[a] * f(a) + w[b] * f(b);
  double I = p + q, err = 0.0;
  int pos = 3;
  for (int k = 0; k < c93_nLevels; k++) {
    int j = c93_lvJ[k], cnt = 0, e = c93_lvEnd[k];
    for (; pos < e; pos += 2) {
      int lo = c93_slot[pos], hi = c93_slot[pos + 1];
      double T = 0.0;
      if (lo >= start) { T += w[lo] * f(lo); cnt++; }
      if (hi <= end) { T += w[hi] * f(hi); cnt++; }
      I += T;
    }
    int n = c93_lvN[k];
    p += (1 - j) * (I - q);
    if (cnt > 0) err = 16 * fabs((1 - j) * (q - 3 * p / 2) + j * (I - 2 * q)) / (3 * n);
    q = (1 - j) * q + j * I;
    if (cnt == 0) continue;
    if (err < tol || (n >= 63 && err < rel * fabs(16 * q / (3 * n)))) {
      res = 16 * q / (3 * n);
      return true;
    }
  }
  return false;
}

// PSM92 walk state (src/gc_integrators.c:39-86) advanced chunk by chunk over
// the schedule.  st = {I, p, q, result}; done = 1 converged.
struct Walk {
  double *I, *p, *q, *res;
  int *done;
};

// Level of schedule slot pos (pos >= 1).
static __device__ inline int level_of(int pos) {
  int k = 0;
  while (c92_lvEnd[k] <= pos) k++;
  return k;
}

}  // namespace ecpgb
