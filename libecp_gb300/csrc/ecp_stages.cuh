// ecp_stages.cuh -- the unit stages' common parts: work lists, scratch and
// shared-memory layouts, the plan stage and the end of the linking stage.
//
// A unit (shell pair, ECP centre) runs in four stages, each a launch over
// work lists that the plan writes (small grid, large grid) or over the units
// (plan, blocks).  Independent warps take list entries, so no CTA barrier waits
// for the slowest primitive pair and a launch's warps run the same code.
// Included by ecp_fast.cu (batched FP64 and mixed) and ecp_exact.cu (the plain
// path, --fmad=false), each with its own __constant__ schedules.
#pragma once
#include <algorithm>

#include "ecp_device.cuh"
#include "ecp_fastmath.h"
#include "ecp_fixed.h"

namespace ecpgb {

constexpr int kWalkCap = 128;  // large-grid quadratures per pass
constexpr int kLargeWarps = 2; // most warps a CTA of the batched large-grid stage

// Small-grid prefactor of a type-1 primitive pair, C1 = ca cb exp(zd2) with
// zd2 = -za dAC^2 - zb dBC^2 (src/type1.c:235-246), rounded as the reference
// rounds it (no contraction), so that every evaluation of it agrees.
static __device__ inline double t1_prefactor(double za, double ca, double zb, double cb, double dAC, double dBC) {
  const double zd2 = __dsub_rn(__dmul_rn(__dmul_rn(-za, dAC), dAC), __dmul_rn(__dmul_rn(zb, dBC), dBC));
  return __dmul_rn(__dmul_rn(ca, cb), fast_exp(zd2));
}

// Kinds of type-1 primitive pairs.  The reference's small-grid integrand is
// C1 r^l U K exp(e), e = (z r + s) r, multiplied left to right
// (src/type1.c:79-88).
//  * normal: C1 >= 2^-900 and e <= s^2 / (4 (za + zb)) < 700: no partial
//    product of a non-negligible term underflows and exp(e) cannot overflow,
//    so the integrand can be regrouped (prefactor, weight and r^l in one
//    table row);
//  * band: C1 below 2^-900 but not 0, or exp(e) may overflow: partial
//    products underflow (or overflow) where a regrouped product would not, so
//    the integrand is evaluated in the reference's order;
//  * zero: C1 = 0 in a job whose products stay in FP64's range, so every integrand
//    value is 0 * (finite) = 0, or NaN where exp(e) overflows -- no table is needed.
constexpr int kPairNormal = 0, kPairBand = 1, kPairZero = 2;
constexpr double kLnDblMax = 0x1.62e42fefa39efp+9;  // exp overflows above it

// e = (z r + s) r as the reference rounds it.
static __device__ inline double t1_exponent(double z, double s, double r) {
  return __dmul_rn(__dadd_rn(__dmul_rn(z, r), s), r);
}

// A zero-kind pair's PS93 walk (src/gc_integrators.c:157-217) with an
// integrand that is 0 except NaN at window points whose exp(e) overflows:
// the first level that counts a point converges to 0 unless a NaN has been
// summed by then, after which no level converges.
static __device__ __noinline__ bool t1_zero_walk(const DevJob &J, double s, double z, int ws, int we) {
  auto nan_at = [&](int n) {
    if (n < ws || n >= we) return false;
    const double e = t1_exponent(z, s, J.xSmall[n]);
    return e >= J.lnAcc1 && e > kLnDblMax;
  };
  bool nan = nan_at(c93_slot[0]) || nan_at(c93_slot[1]) || nan_at(c93_slot[2]);
  int pos = 3;
  for (int k = 0; k < c93_nLevels; k++) {
    const int e = c93_lvEnd[k];
    int cnt = 0;
    for (; pos < e; pos += 2) {
      const int lo = c93_slot[pos], hi = c93_slot[pos + 1];
      if (lo >= ws) { nan = nan || nan_at(lo); cnt++; }
      if (hi <= we) { nan = nan || nan_at(hi); cnt++; }
    }
    if (cnt > 0) return !nan;
  }
  return false;
}

// The bits of a double as an integer that orders like it.
static __device__ inline long long ordered_bits(double x) {
  const long long b = __double_as_longlong(x);
  return b ^ (long long)((unsigned long long)(b >> 63) >> 1);
}

// The first large-grid point with abscissa x >= b, and the first with x > b.
static __device__ __noinline__ int first_key(const DevJob &J, long long key) {
  int lo = 0, hi = J.largeOrder;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (ordered_bits(J.xLarge[mid]) >= key) hi = mid; else lo = mid + 1;
  }
  return lo;
}
static __device__ inline int first_from(const DevJob &J, double b) { return first_key(J, ordered_bits(b)); }
static __device__ inline int first_after(const DevJob &J, double b) { return first_key(J, ordered_bits(b) + 1); }

// FM06 map parameters (src/gc_integrators.c:317-331).
static __device__ inline void fm06(double za, double zb, double dAC, double dBC, double &i1, double &i2) {
  double zp = za + zb, P = (za * dAC + zb * dBC) / zp;
  double sigma = 1.0 / sqrt(zp), t = P - 7.0 * sigma;
  double rmin = (t > 0.0) ? t : 0.0, rmax = P + 9.0 * sigma;
  i1 = 0.5 * (rmax - rmin);
  i2 = 0.5 * (rmax + rmin);
}

// Schedule steps: step 0 = the head plus 15 (lower, upper) pairs, every later
// step 16 pairs.  For the large grid step 0 ends exactly at level 3.
static __device__ inline int step_end93(int s0) { return s0 == 0 ? 33 : s0 + 32; }
static __device__ inline int step_end92(int s0) { return s0 == 0 ? 31 : s0 + 32; }

// Level constants of both rules as doubles (3 n, 3 N): no conversion per level.
static __constant__ double c93_3n[32], c92_3N[32];

// --------------------------------------------------------------- layout

// Quadratures per primitive pair in the type-1 block ((l1, l2), l2 = l1,
// l1-2, ...; src/type1.c:189-202), and primitive pairs packed per warp so
// that most lanes carry a quadrature.
__host__ __device__ inline int t1_items(int lab) {
  int n = 0;
  for (int l1 = 0; l1 <= lab; l1++) n += l1 / 2 + 1;
  return n;
}
// Index of quadrature (l1, l2) in that list.
__host__ __device__ inline int t1_index(int l1, int l2) { return (l1 + 1) * (l1 + 1) / 4 + ((l1 - l2) >> 1); }
__host__ __device__ inline int t1_group(int lab, int cap) {
  int g = 32 / t1_items(lab);
  g = g > 8 ? 8 : (g < 1 ? 1 : g);
  // the group's step table (33 slots x g entries of 2 (lab+1) + 1 doubles)
  // stays within 33 x cap doubles
  while (g > 1 && g * (2 * lab + 3) > cap) g--;
  return g;
}

// The type-2 fallback deals a unit's primitive pairs to warps in parts of
// consecutive pairs: at least 4 pairs a part (the list of failed quadratures
// is decoded once per part) and at most 16 parts (each keeps a partial sum
// per quadrature).  One pair a part (`single`) on the plain path, which keeps
// every pair's result and adds them in the reference's order, and for jobs of
// few primitive pairs, where the longest part sets the time.
__host__ __device__ inline int t2_part_pairs(int NP, bool single) {
  const int n = (NP + 15) / 16;
  return single ? 1 : n < 4 ? 4 : n;
}
__host__ __device__ inline int t2_parts(int NP, bool single) {
  const int n = t2_part_pairs(NP, single);
  return (NP + n - 1) / n;
}

// A unit as the stages see it: the pair's shells and derivative shift, the
// screened window, its scratch (byte offsets L).  The plan leaves it in the
// scratch, where the work-list entries point.
struct UnitScratch {
  int map, win, pair, Q, T, part, mask, perm, total;
};
struct Unit {
  int c, pr, sa, sb, A, B, la, lb, lab, lpa, lpb, pa0, pb0, ws, we, Nb, NP, Lc, cls, nItems;
  const double *gA, *gB, *pzA, *pcA, *pzB, *pcB;
  char *scr;
  UnitScratch L;
  bool live;
};
struct UnitHead {
  int warn;  // 1: a type-1, 2: a type-2 quadrature ran out of levels
  int pad;
  Unit unit;
};
// A normal-kind primitive pair's scalars in fixed point: s = |P| as S 2^-q,
// Z = za + zb (mantissa and exponent), 100 s.
struct PairFx {
  i64 S;
  u64 Zm, sm;
  int Ze, se, q;
};
// What the stages read of a primitive pair: s = |P|, the prefactor C1, -za - zb
// and, on the batched path, the exponents, the coefficients' product C2 and
// zd2 = -za dAC^2 - zb dBC^2.
struct PairRec {
  double s, C1, z, za, zb, C2, zd2;
  PairFx fx;
};
constexpr int kPairWords = sizeof(PairRec) / sizeof(double);

// Global scratch of one unit between the stages (byte offsets): the head, per
// primitive pair the FM06 map (i1, i2), {break index, window} and the record
// above, the type-1 quadratures [pair][t1_index], the type-2 quadratures of the
// class's items, their partial sums [part][item] when there are several parts, the
// bitmap of failed items, and the primitive pairs ordered by kind.
__host__ __device__ inline UnitScratch unit_scratch(int NP, int lab, int nItems, bool single) {
  UnitScratch s;
  int o = ((int)sizeof(UnitHead) + 15) & ~15;
  s.map = o; o += 16 * NP;
  s.win = o; o += 16 * NP;
  s.pair = o; o += (int)sizeof(PairRec) * NP;
  s.Q = o; o += 8 * NP * t1_items(lab);
  s.T = o; o += 8 * nItems;
  s.part = o; o += t2_parts(NP, single) > 1 ? 8 * t2_parts(NP, single) * nItems : 0;
  s.mask = o; o += 4 * ((nItems + 31) / 32);
  s.perm = o; o += NP;
  s.total = (o + 15) & ~15;
  return s;
}
// Work-list entries a unit can add: type-1 groups (at most one per pair),
// type-2 small-grid batches, type-2 parts, failed type-1 pairs.
struct T1Fail {
  int off, k;  // the unit's scratch, primitive pair (bit 16: double-single tables)
  unsigned mask;
  int pad;
  double s;  // |P|
};
__host__ __device__ inline size_t unit_list_bytes(int NP, int nItems, bool single) {
  return 8 * (size_t)NP + 8 * (size_t)((nItems + 31) / 32) + 8 * (size_t)t2_parts(NP, single) + sizeof(T1Fail) * (size_t)NP;
}

// Shared memory of the stages, in doubles.  Small grid (one warp a CTA): the
// group's pair scalars and step table.
struct SmallSmem {
  int rec, quad, tab, total;
};
__host__ __device__ inline SmallSmem small_layout(int LB, int rows, int cap) {
  SmallSmem s;
  // type 2 (batched path): 32 slots of the most rows a batch reads
  int tt = 32 * ((rows + (rows + 3) / 4) | 1);
  for (int lab = 0; lab <= 2 * LB; lab++) {
    const int w = 33 * t1_group(lab, cap) * (2 * lab + 3);
    if (w > tt) tt = w;
  }
  s.rec = 0;                      // up to 8 pairs
  s.quad = 8 * kPairWords;        // 32 ints
  s.tab = s.quad + 16;
  s.total = s.tab + tt;
  return s;
}
// Large grid: type 1 a 32-slot table a warp; type 2 a 32-slot table (U[nE],
// R[nA], Ka[LBE], Kb[LBE], on the plain path the exponential and the weight, on the
// batched path 16-bit exponents after it), the quadratures' state, the running
// ones, the pending slots and the failed items.
struct LargeSmem {
  int tab, tabT1, I, P, Q, E, part, act, pend, fail, red, total, tabStride, expStride;
};
__host__ __device__ inline LargeSmem large_layout(int LB, int LE, bool exact) {
  LargeSmem s{};
  const int nA = 2 * LB + 1, nE = LE > 0 ? LE : 1, LBE = LB + nE;
  s.tabStride = (nE + nA + 2 * LBE + (exact ? 2 : 0)) | 1;  // odd: conflict-free lane strides
  // 16-bit exponents of U, Ka, Kb and r^l (batched path): an odd number of words a lane
  s.expStride = 2 * (((nE + 2 * LBE + nA + 1) / 2) | 1);
  s.tabT1 = 32 * (2 * nA + 3);  // type-1 table of one warp
  int o = 32 * s.tabStride + (exact ? 0 : 8 * s.expStride), t1 = (exact ? 1 : kLargeWarps) * s.tabT1;
  s.tab = 0;
  if (t1 > o) o = t1;
  s.I = o; o += kWalkCap;
  s.P = o; o += kWalkCap;
  s.Q = o; o += kWalkCap;
  s.part = o; o += kWalkCap;
  s.pend = o; o += 32 * (exact ? 1 : kLargeWarps);
  s.act = o; o += kWalkCap / 8;
  if (!exact) {  // exponents of the running items, what two warps tell each other
    s.E = o; o += kWalkCap;
    s.red = o; o += 2 * kLargeWarps;
  }
  s.fail = o; o += kWalkCap / 2;
  s.total = o;
  return s;
}
// Linking: chi / gamma, the half-shifted block, the radial table T, S_lm of a
// batch of primitive pairs, the shift factors, the S_lm sums W and the
// combined-index block H.
constexpr int kLinkBatch = 16;
constexpr int kShiftTerms = 12;  // most (x+1)(y+1)(z+1) over x + y + z = l <= 4
struct LinkSmem {
  int chi, J, T, rsh, fac, dir, W, H, total;
};
__host__ __device__ inline LinkSmem link_layout(int LB, int LE) {
  LinkSmem s;
  const int nA = 2 * LB + 1, nE = LE > 0 ? LE : 1, LBE = LB + nE;
  const int nc = (LB + 1) * (LB + 2) * (LB + 3) / 6, nct = (LB + 1) * (LB + 2) / 2;
  const int ncAB = (2 * LB + 1) * (2 * LB + 2) * (2 * LB + 3) / 6;
  int o = 0;
  s.chi = o; o += nc * nc;
  {  // W, later the radial table
    const int t = nE * LBE * LBE * (LB + 1);
    s.T = s.W = o; o += t > ncAB ? t : ncAB;
  }
  {  // S_lm of a batch, later the half-contracted gamma of one (l, alpha) or the half-shifted block
    const int r = kLinkBatch * nA * nA, y = (2 * nE - 1) * (LB + 1) * nc, h = nct * nc;
    s.rsh = s.J = o; o += r > y ? (r > h ? r : h) : (y > h ? y : h);
  }
  s.fac = o; o += 2 * kShiftTerms * nct;
  s.dir = o; o += kLinkBatch * 4;
  s.H = o; o += ncAB;
  s.total = o;
  return s;
}

// Unit id of queue position pos (pairs in the plan's order, centres innermost).
static __device__ inline long long unit_at(const DevJob &J, int pos) {
  const int c = J.ctrOrder[pos % J.nCentres], pr = J.pairOrder[pos / J.nCentres];
  return (long long)c * J.nPairs + pr;
}

// Items of the unit's class over the channels below l.
static __device__ inline int class_items(const DevJob &J, int ncls, int l) {
  int n = 0;
  for (int k = 0; k < l; k++) n += J.itemCnt[ncls + k];
  return n;
}

// The unit a work-list entry points to.
static __device__ inline const Unit &unit_get(const DevJob &J, int off) {
  return ((const UnitHead *)(J.scr + (size_t)off * 16))->unit;
}

// The unit at queue position pos = (sorted pair, centre).
static __device__ inline Unit unit_load(const DevJob &J, int pos) {
  Unit U;
  const int ps = pos / J.nCentres, ci = pos % J.nCentres;
  U.c = J.ctrOrder[ci];
  U.pr = J.pairOrder[ps];
  U.sa = J.pairA[U.pr];
  U.sb = J.pairB[U.pr];
  U.A = J.shAtom[U.sa];
  U.B = J.shAtom[U.sb];
  const int *wa = J.win + ((size_t)U.c * J.nShells + U.sa) * 3, *wb = J.win + ((size_t)U.c * J.nShells + U.sb) * 3;
  // derivative shift: the shells' l moved by (shifta, shiftb) for the
  // computation, the blocks handed out with l (lpa, lpb)
  const UnitShift sh = unit_shift(J, U.pr, J.shL[U.sa], J.shL[U.sb], U.A, U.B, J.ctrAtom[U.c]);
  U.ws = wa[0] > wb[0] ? wa[0] : wb[0];
  U.we = wa[1] > wb[1] ? wa[1] : wb[1];
  U.live = !(wa[2] || wb[2] || sh.skip) && U.ws < U.we;
  U.la = J.shL[U.sa] + sh.a;
  U.lb = J.shL[U.sb] + sh.b;
  U.lab = U.la + U.lb;
  U.lpa = sh.lpa;
  U.lpb = sh.lpb;
  U.pa0 = sh.a > 0 ? sh.a : 0;
  U.pb0 = sh.b > 0 ? sh.b : 0;
  U.Nb = J.shK[U.sb];
  U.NP = J.shK[U.sa] * U.Nb;
  U.Lc = J.ctrL[U.c];
  if (!U.live) return U;
  const int LE = J.maxLECP > 0 ? J.maxLECP : 1;
  U.cls = U.la * (J.maxLBS + 1) + U.lb;
  U.nItems = class_items(J, U.cls * LE, U.Lc);
  U.gA = J.cgeo + ((size_t)U.c * J.nAtoms + U.A) * 4;
  U.gB = J.cgeo + ((size_t)U.c * J.nAtoms + U.B) * 4;
  U.pzA = J.primA + J.shP[U.sa];
  U.pcA = J.primD + J.shP[U.sa];
  U.pzB = J.primA + J.shP[U.sb];
  U.pcB = J.primD + J.shP[U.sb];
  U.L = unit_scratch(U.NP, U.lab, class_items(J, U.cls * LE, LE), J.single);
  U.scr = J.scr + (J.scrOff[ps] - J.scrBase) + (size_t)ci * U.L.total;
  return U;
}

// The item q of the unit's class as (l, l1, l2, l3), one byte each (all below 16).
static __device__ inline int unit_item(const DevJob &J, const Unit &U, int q) {
  const int ncls = U.cls * (J.maxLECP > 0 ? J.maxLECP : 1);
  int l = 0;
  while (q >= J.itemCnt[ncls + l]) { q -= J.itemCnt[ncls + l]; l++; }
  const int v = J.items[J.itemOff[ncls + l] + q];
  return l | (v & 255) << 8 | ((v >> 8) & 255) << 16 | (v >> 16) << 24;
}

// Work lists of a chunk and their counters (zeroed before the chunk).
enum { kCntT1, kCntRest, kCntT2, kCntFail, kCntPart, kHeadSmall, kHeadLarge, kCounters };

// Lanes of a warp dealt to n running quadratures: P = 2^b lanes each, which
// evaluate P points side by side (the batched path's integer sums then combine by
// shuffles; the plain path's values are added in order).
struct LaneDeal {
  int P;     // lanes per quadrature
  int rank;  // the quadrature this lane works for, n or more: none
  int part;  // which of its P lanes
};
static __device__ inline LaneDeal deal_lanes(int n) {
  const int b = n > 16 ? 0 : n > 8 ? 1 : n > 4 ? 2 : 3, lane = threadIdx.x & 31;
  return {1 << b, lane >> b, lane & ((1 << b) - 1)};
}

// The next entry of a list for a warp; its index to every lane.
static __device__ inline int next_item(unsigned *head) {
  int i = 0;
  if ((threadIdx.x & 31) == 0) i = (int)atomicAdd(head, 1u);
  return __shfl_sync(0xffffffffu, i, 0);
}

// 1/k, k <= 24 (the Legendre recurrence's divisor l - m)
static __device__ const double kRecip[25] = {0.0,        1.0,        1.0 / 2,  1.0 / 3,  1.0 / 4,
                                             1.0 / 5,    1.0 / 6,    1.0 / 7,  1.0 / 8,  1.0 / 9,
                                             1.0 / 10,   1.0 / 11,   1.0 / 12, 1.0 / 13, 1.0 / 14,
                                             1.0 / 15,   1.0 / 16,   1.0 / 17, 1.0 / 18, 1.0 / 19,
                                             1.0 / 20,   1.0 / 21,   1.0 / 22, 1.0 / 23, 1.0 / 24};

// Binomial coefficients C(n, k), n <= 15, as exact doubles: the values
// fac[n] / (fac[n-k] fac[k]) of src/util.c:247-334 (exact integers), looked
// up instead of divided out per term.
struct BinomTable {
  double v[16][16];
  constexpr BinomTable() : v() {
    for (int n = 0; n < 16; n++) {
      v[n][0] = 1.0;
      for (int k = 1; k <= n; k++) v[n][k] = v[n - 1][k - 1] + (k < n ? v[n - 1][k] : 0.0);
    }
  }
};
static __device__ const BinomTable kBinom;
static __device__ inline double binom_tab(int n, int k) { return __ldg(&kBinom.v[n][k]); }

// --------------------------------------------------------- stage 1: the plan

// A unit by one warp: its primitive pairs by kind (kind-major, each kind in
// pair order), the FM06 map, break index, point window and scalars of every pair,
// its work-list entries; a dead unit is marked skipped.  A lane a pair: bound by
// the FP64 pipe (81 % busy), some 200 instructions a unit, most of them square
// roots and divides.  8 centres of the cluster: 0.20 ms (0.22 on the plain path).
constexpr int kPlanThreads = 128;
template <bool kExact>
__global__ void __launch_bounds__(kPlanThreads) k_unit_plan(DevJob J) {
  const int lane = threadIdx.x & 31;
  const int idx = blockIdx.x * (kPlanThreads / 32) + (threadIdx.x >> 5);
  int pos = J.chunk0 + idx;
  if (J.live) {
    const int l0 = J.liveStart[J.chunk];
    if (l0 + idx >= J.liveStart[J.chunk + 1]) return;
    pos = J.live[l0 + idx];
  } else if (idx >= J.chunk1 - J.chunk0) {
    return;
  }
  const Unit U = unit_load(J, pos);
  if (!U.live) {
    if (lane == 0) J.status[(size_t)U.c * J.nPairs + U.pr] = kUnitSkipped;
    return;
  }
  const double dAC = U.gA[3], dBC = U.gB[3];
  const int NP = U.NP, Nb = U.Nb;
  unsigned char *perm = (unsigned char *)(U.scr + U.L.perm);
  double2 *map = (double2 *)(U.scr + U.L.map);
  int4 *win = (int4 *)(U.scr + U.L.win);
  unsigned *mask = (unsigned *)(U.scr + U.L.mask);
#pragma unroll 1
  for (int w = lane; w < (U.nItems + 31) / 32; w += 32) mask[w] = 0u;
  const int off = (int)((U.scr - J.scr) >> 4);
  if (lane == 0) *(UnitHead *)U.scr = {0, 0, U};
  int cnt[3] = {0, 0, 0};
  unsigned kinds = 0;  // the lane's pairs' kinds, 2 bits each (at most 8)
#pragma unroll 1
  for (int k0 = 0, j = 0; k0 < NP; k0 += 32, j++) {
    const int k = k0 + lane;
    int kind = 3;
    if (k < NP) {
      const double za = U.pzA[k / Nb], zb = U.pzB[k % Nb];
      const double ca = zeta_times(U.pcA[k / Nb], za, U.pa0), cb = zeta_times(U.pcB[k % Nb], zb, U.pb0);
      const double C1 = kExact ? ca * cb * exp(-za * dAC * dAC - zb * dBC * dBC) : t1_prefactor(za, ca, zb, cb, dAC, dBC);
      double P[3];
      for (int i = 0; i < 3; i++) P[i] = 2.0 * (za * U.gA[i] + zb * U.gB[i]);
      const double s2 = P[0] * P[0] + P[1] * P[1] + P[2] * P[2];
      kind = C1 == 0.0 && J.inRange ? kPairZero
                       : (kExact || fabs(C1) < 0x1p-900 || s2 > 2800.0 * (za + zb)) ? kPairBand : kPairNormal;
      PairRec rec;
      rec.s = sqrt(s2);
      rec.C1 = C1;
      rec.z = -za - zb;
      rec.za = za;
      rec.zb = zb;
      rec.C2 = ca * cb;
      rec.zd2 = -za * dAC * dAC - zb * dBC * dBC;
      if (!kExact && kind == kPairNormal) {
        // s and Z r (r inside the window) as integers times 2^q, both below 2^62
        const xf S = xf_from(rec.s), Z = xf_from(za + zb), s100 = xf_times100(S);
        const int zr = Z.e + xf_from(J.xSmall[U.we - 1]).e + 64, q = -3 - (S.e > zr ? S.e : zr);
        rec.fx = {(i64)shr64(S.m, -(S.e + q)), Z.m, s100.m, Z.e, s100.e, q};
      }
      ((PairRec *)(U.scr + U.L.pair))[k] = rec;
      double i1, i2;
      fm06(za, zb, dAC, dBC, i1, i2);
      map[k] = make_double2(i1, i2);
      int t1Break = 0;
      if constexpr (!kExact) {
        // first point past both centres whose type-1 exponent (z r + s) r + zd2 is
        // below the screen (src/type1.c:168-176): the root of the parabola
        const double zp = za + zb, q = rec.s * rec.s - 4.0 * zp * (J.lnAcc1 - rec.zd2);
        const double root = q > 0.0 ? 0.5 * (rec.s + sqrt(q)) / zp : 0.0, far = dAC > dBC ? dAC : dBC;
        t1Break = first_after(J, ((root > far ? root : far) - i2) / i1);
      }
      if (U.nItems > 0) {
        // break index, and the point-index interval in which the pair's
        // exponent passes the screen: past both centres the exponent falls with
        // the index; it is a parabola in r with its vertex at V, and r grows with
        // the index.  r within h of the vertex, -zp h^2 - mu = the threshold: bisections
        // of the abscissae, whose bits are compared as integers (five of the
        // exponent, at eight FP64 operations a step, were most of this kernel: 190
        // -> 69 us for 6048 units).  The plain path's stage tests every slot of the
        // interval itself (a margin of 1), and its break is settled by the exponent as
        // the reference rounds it.
        const double V = (za * dAC + zb * dBC) / (za + zb), zp = za + zb, mu = za * zb / zp * (dAC - dBC) * (dAC - dBC);
        const double m = 1.0 / i1, far = dAC > dBC ? dAC : dBC;
        const double q = ((kExact ? 1.0 : 0.0) - J.lnAcc2 - mu) / zp, h = sqrt(q > 0.0 ? q : 0.0);
        const int n0 = first_from(J, (V - h - i2) * m), n1 = first_after(J, (V + h - i2) * m);
        int brk = first_after(J, (far - i2) * m);
        if constexpr (!kExact) {
          if (q >= 0.0 && n1 > brk) brk = n1;
        } else {
          const double qb = (-J.lnAcc2 - mu) / zp;
          const int nb = qb >= 0.0 ? first_after(J, (V + sqrt(qb) - i2) * m) : 0;
          if (nb > brk) brk = nb;
          auto past = [&](int n) {
            const double r = i1 * J.xLarge[n] + i2, d1 = dAC - r, d2 = dBC - r;
            return r > dAC && r > dBC && -za * d1 * d1 - zb * d2 * d2 < J.lnAcc2;
          };
          while (brk < J.largeOrder && !past(brk)) brk++;
          while (brk > 0 && past(brk - 1)) brk--;
        }
        if (brk >= J.largeOrder) brk = INT_MAX;
        win[k] = q >= 0.0 ? make_int4(brk, n0, n1 - 1, t1Break) : make_int4(brk, 1, 0, t1Break);
      } else {
        win[k] = make_int4(INT_MAX, 1, 0, t1Break);
      }
    }
    kinds |= (unsigned)kind << (2 * j);
    for (int kd = 0; kd < 3; kd++) cnt[kd] += __popc(__ballot_sync(0xffffffffu, kind == kd));
  }
  int at[3] = {0, cnt[0], cnt[0] + cnt[1]};
#pragma unroll 1
  for (int k0 = 0, j = 0; k0 < NP; k0 += 32, j++) {
    const int kind = (kinds >> (2 * j)) & 3u;
    for (int kd = 0; kd < 3; kd++) {
      const unsigned m = __ballot_sync(0xffffffffu, kind == kd);
      if (kind == kd) perm[at[kd] + __popc(m & ((1u << lane) - 1u))] = (unsigned char)(k0 + lane);
      at[kd] += __popc(m);
    }
  }
  // the class's type-1 settings (the autotuner may set them per (la, lb))
  int gcap = J.gcap, bal = J.balance;
  if (J.classCfg[U.cls] & kClassSet) {
    gcap = J.classCfg[U.cls] & 0xfff;
    bal = (J.classCfg[U.cls] >> 12) & 1;
  }
  int G[3], n[3], nGroups = 0;
  for (int kd = 0; kd < 3; kd++) {
    // (one pair a group in jobs of few pairs, as the type-2 parts)
    G[kd] = J.few ? 1 : t1_group(U.lab, gcap);
    // balance: a unit with few primitive pairs gives its groups to four warps
    if (bal) {
      const int g = (cnt[kd] + 3) / 4;
      if (g < G[kd]) G[kd] = g > 0 ? g : 1;
    }
    n[kd] = (cnt[kd] + G[kd] - 1) / G[kd];
    nGroups += n[kd];
  }
  const int nBatch = (U.nItems + 31) / 32, nPart = U.nItems > 0 ? t2_parts(NP, J.single) : 0;
  // the type-1 list holds the groups of normal kind from its front and the others
  // from its end: warps that run at the same time run the same code
  int base = 0;
  if (lane < 4)
    base = (int)atomicAdd(J.counters + (lane == 0 ? kCntT1 : lane == 1 ? kCntRest : lane == 2 ? kCntT2 : kCntPart),
                          (unsigned)(lane == 0 ? n[0] : lane == 1 ? n[1] + n[2] : lane == 2 ? nBatch : nPart));
  const int b1 = __shfl_sync(0xffffffffu, base, 0), br = __shfl_sync(0xffffffffu, base, 1),
            b2 = __shfl_sync(0xffffffffu, base, 2), b3 = __shfl_sync(0xffffffffu, base, 3);
#pragma unroll 1
  for (int g = lane; g < nGroups; g += 32) {
    int kd = 0, gj = g, p0 = 0;
    while (gj >= n[kd]) { gj -= n[kd]; p0 += cnt[kd]; kd++; }
    p0 += gj * G[kd];
    const int left = cnt[kd] - gj * G[kd];
    J.listT1[kd == 0 ? b1 + g : J.capT1 - 1 - (br + g - n[0])] =
        make_int2(off, p0 | (left < G[kd] ? left : G[kd]) << 10 | kd << 16);
  }
#pragma unroll 1
  for (int q = lane; q < nBatch; q += 32) J.listT2[b2 + q] = make_int2(off, 32 * q);
#pragma unroll 1
  for (int q = lane; q < nPart; q += 32) J.listPart[b3 + q] = make_int2(off, q);
}

// Entry i of the small-grid stage: the type-1 groups of normal kind, the other
// groups, the type-2 batches.
static __device__ inline int2 small_entry(const DevJob &J, int i, int n0, int n1) {
  return i < n0 ? J.listT1[i] : i < n1 ? J.listT1[J.capT1 - 1 - (i - n0)] : J.listT2[i - n1];
}

// The blocks of a unit from its combined-index block H (type 1: `one`) and its
// radial table (type 2, src/type2.c:583-623: `two`), both shifted onto A and B
// (src/util.c:247-334), and its status (with `two`).
constexpr int kLinkThreadsMax = 256;
// CTAs a unit: in small jobs one for each block, which halves a unit's chain (78
// units: 42 instead of 55 us, plain path 47 instead of 80; unit stages of 2016 units
// 1.19 instead of 1.25 ms, of 6048 2.68 instead of 2.67, of 100,800 37.3 instead of 37.0).
static inline unsigned link_parts(unsigned units) { return units <= 4096 ? 2 : 1; }
// Threads a CTA: 256 where the shared memory (g shells) lets only a few CTAs
// share a multiprocessor (the 150-shell sweep's unit stages: 47.9 ms, at 128 threads
// 48.7; with less shared memory 128 and 256 measure the same).
static inline int link_threads(size_t smem) { return smem > 40 * 1024 ? 256 : 128; }
template <bool kExact>
static __device__ void link_finish(const DevJob &J, const Unit &U, const LinkSmem &Lm, double *sm, bool one, bool two) {
  const int tid = threadIdx.x, NT = blockDim.x, la = U.la, lb = U.lb, lpa = U.lpa, lpb = U.lpb, nca = NCUM(la),
            ncb = NCUM(lb), Lc = U.Lc;
  // (l1 + l2 + l3 is even: every other l3 in a row)
  const int nT = J.maxLBS + 1, LE = J.maxLECP > 0 ? J.maxLECP : 1, LBE = J.maxLBS + LE;
  const size_t cA = (size_t)U.c * J.nAtoms + U.A, cB = (size_t)U.c * J.nAtoms + U.B;
  double *chi = sm + Lm.chi, *Jsh = sm + Lm.J, *T = sm + Lm.T, *H = sm + Lm.H;
  double *out1 = J.out + (size_t)U.c * J.centreStride + J.pairOff[U.pr];
  double *out2 = out1 + NCART(lpa) * NCART(lpb);
  const int dd = J.tmDim + 1;
#pragma unroll 1
  for (int e = one ? tid : nca * ncb; e < nca * ncb; e += NT) {
    const int *ei = J.ijk + 3 * (e / ncb), *ej = J.ijk + 3 * (e % ncb);
    chi[e] = H[J.ijkIdx[((ei[0] + ej[0]) * dd + (ei[1] + ej[1])) * dd + ei[2] + ej[2]]];
  }
  // the radial table of type 2
  auto tidx = [&](int l, int l1, int l2, int l3) { return ((l * LBE + l1) * LBE + l2) * nT + (l3 >> 1); };
#pragma unroll 1
  for (int e = tid; e < LE * LBE * LBE * nT; e += NT) T[e] = 0.0;
  __syncthreads();
  if (two) {
    const double *Tq = (const double *)(U.scr + U.L.T), *part = (const double *)(U.scr + U.L.part);
    const unsigned *mask = (const unsigned *)(U.scr + U.L.mask);
    const int nParts = t2_parts(U.NP, J.single), nIt = class_items(J, U.cls * LE, LE);
#pragma unroll 1
    for (int q = tid; q < U.nItems; q += NT) {
      double v;
      if (nParts > 1 && (mask[q >> 5] >> (q & 31) & 1u)) {
        v = 0.0;
#pragma unroll 1
        for (int p = 0; p < nParts; p++) v += part[(size_t)p * nIt + q];
      } else {
        v = Tq[q];
      }
      const int it = unit_item(J, U, q);
      T[tidx(it & 255, (it >> 8) & 255, (it >> 16) & 255, it >> 24)] = v;
    }
  }
  __syncthreads();
  const double norm1 = 4.0 * kPi, norm2 = norm1 * norm1;
  if constexpr (kExact) {
    auto poly_shift = [&](double norm, double *dst) {  // src/util.c:247-334
      const int D = J.uspD, nta = NCART(lpa), ntb = NCART(lpb);
      const double *uA = J.usp + cA * D * D * D, *uB = J.usp + cB * D * D * D;
#pragma unroll 1
      for (int e = tid; e < nta * ncb; e += NT) {
        int c1 = e / ncb, q = e % ncb;
        const int *ex = J.ijk + 3 * (NCUM(lpa - 1) + c1);
        double v = 0.0;
#pragma unroll 1
        for (int x = 0; x <= ex[0]; x++) {
          double bx = binom_tab(ex[0], x);
#pragma unroll 1
          for (int y = 0; y <= ex[1]; y++) {
            double by = bx * binom_tab(ex[1], y);
#pragma unroll 1
            for (int zz = 0; zz <= ex[2]; zz++) {
              double bz = by * binom_tab(ex[2], zz);
              double factor = bz * uA[((ex[0] - x) * D + (ex[1] - y)) * D + (ex[2] - zz)];
              if (fabs(factor) <= J.acc) continue;
              v += factor * chi[J.ijkIdx[(x * dd + y) * dd + zz] * ncb + q];
            }
          }
        }
        Jsh[e] = v;
      }
      __syncthreads();
#pragma unroll 1
      for (int e = tid; e < nta * ntb; e += NT) {
        int c1 = e / ntb, c2 = e % ntb;
        const int *ex = J.ijk + 3 * (NCUM(lpb - 1) + c2);
        double v = 0.0;
#pragma unroll 1
        for (int x = 0; x <= ex[0]; x++) {
          double bx = binom_tab(ex[0], x);
#pragma unroll 1
          for (int y = 0; y <= ex[1]; y++) {
            double by = bx * binom_tab(ex[1], y);
#pragma unroll 1
            for (int zz = 0; zz <= ex[2]; zz++) {
              double bz = by * binom_tab(ex[2], zz);
              double factor = bz * uB[((ex[0] - x) * D + (ex[1] - y)) * D + (ex[2] - zz)];
              if (fabs(factor) <= J.acc) continue;
              factor *= norm;
              v += factor * Jsh[c1 * ncb + J.ijkIdx[(x * dd + y) * dd + zz]];
            }
          }
        }
        dst[e] = v;
      }
      __syncthreads();
    };
    if (one) poly_shift(norm1, out1);
    if (!two) return;
    // gamma (src/type2.c:583-623)
    {
      const double *angA = J.ang + cA * J.angLam * J.angLM * J.angC;
      const double *angB = J.ang + cB * J.angLam * J.angLM * J.angC;
      const int LMd = J.angLM, AC = J.angC;
#pragma unroll 1
      for (int e = tid; e < nca * ncb; e += NT) {
        int pidx = e / ncb, qidx = e % ncb, alpha = 0, beta = 0;
        while (NCUM(alpha) <= pidx) alpha++;
        while (NCUM(beta) <= qidx) beta++;
        double g = 0.0;
#pragma unroll 1
        for (int l = 0; l < Lc; l++) {
          int ll1 = l - alpha, p1 = (alpha + l) % 2;
          if (p1 > ll1) ll1 = p1;
          int ll2 = l - beta, p2 = (beta + l) % 2;
          if (p2 > ll2) ll2 = p2;
          double tmp = 0.0;
#pragma unroll 1
          for (int l1 = ll1; l1 <= la + l; l1 += 2)
#pragma unroll 1
            for (int l2 = ll2; l2 <= lb + l; l2 += 2) {
              double factor = 0.0;
#pragma unroll 1
              for (int m = 0; m < 2 * l + 1; m++)
                factor += angA[((size_t)l1 * LMd + l * l + m) * AC + pidx] * angB[((size_t)l2 * LMd + l * l + m) * AC + qidx];
              tmp += factor * T[tidx(l, l1, l2, alpha + beta)];
            }
          g += tmp;
        }
        chi[e] = g;
      }
    }
    __syncthreads();
    poly_shift(norm2, out2);
  } else {
    // the shift's factors binomial * (-R)^(e - x) once per unit, a row of up to
    // 12 per Cartesian function, l <= 4 (0 where the reference skips one); then both
    // blocks' shifts are one multiply-add a term
    double *fA = sm + Lm.fac, *fB = fA + NCART(lpa) * kShiftTerms;
    const int D = J.uspD, nta = NCART(lpa), ntb = NCART(lpb);
    const double *uA = J.usp + cA * D * D * D, *uB = J.usp + cB * D * D * D;
#pragma unroll 1
    for (int e = tid; e < (nta + ntb) * kShiftTerms; e += NT) {
      const bool b = e >= nta * kShiftTerms;
      const int f = b ? e - nta * kShiftTerms : e, c1 = f / kShiftTerms, i = f % kShiftTerms;
      const int *ex = J.ijk + 3 * (NCUM((b ? lpb : lpa) - 1) + c1);
      const int ny = ex[1] + 1, nz = ex[2] + 1;
      if (i >= (ex[0] + 1) * ny * nz) continue;
      const int x = i / (ny * nz), y = i / nz % ny, z = i % nz;
      const double v = binom_tab(ex[0], x) * binom_tab(ex[1], y) * binom_tab(ex[2], z) *
                       (b ? uB : uA)[((ex[0] - x) * D + (ex[1] - y)) * D + (ex[2] - z)];
      fA[e] = fabs(v) <= J.acc ? 0.0 : v;
    }
    auto shift = [&](double norm, double *dst) {
#pragma unroll 1
      for (int pass = 0; pass < 2; pass++) {
        // J = shift_A chi, then dst = norm J shift_B^T
        const double *fac = pass ? fB : fA;
        const int l = pass ? lpb : lpa, nOut = pass ? nta * ntb : nta * ncb, w = pass ? ntb : ncb;
#pragma unroll 1
        for (int e = tid; e < nOut; e += NT) {
          const int i = e / w, j = e % w, c1 = pass ? j : i;
          const int *ex = J.ijk + 3 * (NCUM(l - 1) + c1);
          const double *f = fac + c1 * kShiftTerms, *src = pass ? Jsh + i * ncb : chi + j;
          const int step = pass ? 1 : ncb;
          double v = 0.0;
#pragma unroll 1
          for (int x = 0; x <= ex[0]; x++)
#pragma unroll 1
            for (int y = 0; y <= ex[1]; y++)
#pragma unroll 1
              for (int z = 0; z <= ex[2]; z++, f++)
                if (*f != 0.0) v = fma(*f, src[J.ijkIdx[(x * dd + y) * dd + z] * step], v);
          if (pass) dst[e] = norm * v;
          else Jsh[e] = v;
        }
        __syncthreads();
      }
    };
    __syncthreads();
    if (one) shift(norm1, out1);
    if (!two) return;
    // gamma (src/type2.c:583-623), for every channel l and bra degree alpha in
    // two steps: Y[m][l1][q] = sum over l2 of Omega_B T, then the sum over
    // (m, l1) of Omega_A Y -- the radial table enters once per (l1, q) instead of
    // once per (p, q).  Omega_A vanishes for l1 > l + alpha.
    {
      const double *angA = J.ang + cA * J.angLam * J.angLM * J.angC;
      const double *angB = J.ang + cB * J.angLam * J.angLM * J.angC;
      const int LMd = J.angLM, AC = J.angC;
      double *Y = sm + Lm.rsh;
#pragma unroll 1
      for (int e = tid; e < nca * ncb; e += NT) chi[e] = 0.0;
#pragma unroll 1
      for (int l = 0; l < Lc; l++)
#pragma unroll 1
        for (int alpha = 0; alpha <= la; alpha++) {
          const int lo1 = l > alpha ? l - alpha : (alpha + l) & 1, n1 = (l + alpha - lo1) / 2 + 1, M = 2 * l + 1;
          __syncthreads();
#pragma unroll 1
          for (int e = tid; e < M * n1 * ncb; e += NT) {
            const int q = e % ncb, r = e / ncb, l1 = lo1 + 2 * (r / M), m = r % M;
            int beta = 0;
            while (NCUM(beta) <= q) beta++;
            const int lo2 = l > beta ? l - beta : (beta + l) & 1;
            const double *B = angB + ((size_t)lo2 * LMd + l * l + m) * AC + q;
            const double *t = T + tidx(l, l1, lo2, alpha + beta);
            double v = 0.0;
#pragma unroll 4
            for (int l2 = lo2; l2 <= l + beta; l2 += 2, B += 2 * (size_t)LMd * AC, t += 2 * nT) v = fma(*B, *t, v);
            Y[e] = v;
          }
          __syncthreads();
          const int p0 = NCUM(alpha - 1);
#pragma unroll 1
          for (int e = tid; e < NCART(alpha) * ncb; e += NT) {
            const int p = p0 + e / ncb, q = e % ncb;
            double v = 0.0;
            const double *A = angA + ((size_t)lo1 * LMd + l * l) * AC + p, *y = Y + q;
#pragma unroll 1
            for (int i = 0; i < n1; i++, A += 2 * (size_t)LMd * AC, y += M * ncb)
#pragma unroll 4
              for (int m = 0; m < M; m++) v = fma(A[(size_t)m * AC], y[m * ncb], v);
            chi[p * ncb + q] += v;
          }
        }
    }
    __syncthreads();
    shift(norm2, out2);
  }
  if (tid == 0) {
    const int warn = ((const UnitHead *)U.scr)->warn;
    const long long u = (long long)U.c * J.nPairs + U.pr;
    const int st = (warn & 1) ? kUnitWarnType1 : (warn & 2) ? kUnitWarnType2 : kUnitDone;
    J.status[u] = st;
    if (st != kUnitDone) atomicMin(&J.errWord[0], (int)u);
  }
}

// Whether a unit computes blocks (the screened windows of src/libecp.c:296-330
// and the derivative skips).
static __device__ bool unit_live(const DevJob &J, int pos) {
  const long long u = unit_at(J, pos);
  const int c = (int)(u / J.nPairs), pr = (int)(u % J.nPairs);
  const int sa = J.pairA[pr], sb = J.pairB[pr];
  const int *wa = J.win + ((size_t)c * J.nShells + sa) * 3;
  const int *wb = J.win + ((size_t)c * J.nShells + sb) * 3;
  const UnitShift sh = unit_shift(J, pr, J.shL[sa], J.shL[sb], J.shAtom[sa], J.shAtom[sb], J.ctrAtom[c]);
  if (wa[2] || wb[2] || sh.skip) return false;
  return (wa[0] > wb[0] ? wa[0] : wb[0]) < (wa[1] > wb[1] ? wa[1] : wb[1]);
}

// Sets J to the plan's order `sorted`.
static const JobPlan::Order &use_order(DevJob &J, int sorted) {
  const JobPlan::Order &ord = J.plan->order[sorted];
  J.pairOrder = J.pairOrders + (size_t)sorted * J.nPairs;
  J.scrOff = J.scrOffs + (size_t)sorted * (J.nPairs + 1);
  J.chunkUnit = J.chunkUnits + ord.chunkAt;
  J.nChunks = (int)ord.chunks.size();
  return ord;
}

// The unit stages of every chunk: sets the chunk's fields and clears its
// counters, then `stages` launches the four kernels.  A warp takes up to 8
// list entries where there are at least 64 a multiprocessor for each (fewer CTAs
// to start), one where there are few (every SM gets work).
template <class Stages>
static void launch_chunks(DevJob J, const JobPlan::Order &ord, cudaStream_t st, Stages stages) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  for (int k = 0; k < J.nChunks; k++) {
    const JobPlan::Chunk &ch = ord.chunks[k];
    J.chunk = k;
    J.chunk0 = ch.u0;
    J.chunk1 = ch.u1;
    J.scrBase = ch.base;
    char *lists = J.scr + ch.scratch;
    J.listT1 = (int2 *)lists;
    J.capT1 = (int)ch.groups;
    J.listT2 = J.listT1 + ch.groups;
    J.listPart = J.listT2 + ch.batches;
    J.listFail = (T1Fail *)(J.listPart + ch.parts);
    cudaMemsetAsync(J.counters, 0, sizeof(unsigned) * kCounters, st);
    auto take = [&](long long items) { return (int)std::min(8ll, std::max(1ll, items / (64ll * sms))); };
    auto grid = [&](long long items) { return (unsigned)std::max(1ll, (items + take(items) - 1) / take(items)); };
    const long long nSmall = ch.groups + ch.batches, nLarge = ch.parts + ch.groups;
    stages(J, (unsigned)(J.chunk1 - J.chunk0), grid(nSmall), take(nSmall), grid(nLarge), take(nLarge));
  }
}

// This translation unit's __constant__ schedules.
static int upload_stage_schedules(const int *s93slot, int s93n, const int *s93lvEnd, const int *s93lvJ,
                          const int *s93lvN, int s93levels, const int *s92slot, int s92n,
                          const int *s92lvEnd, const int *s92lvN, int s92levels, void *stream) {
  if (s93n > kSmallOrder || s92n > kMaxLargeOrder || s93levels > 32 || s92levels > 32) return 1;
  cudaStream_t st = (cudaStream_t)stream;
  cudaMemcpyToSymbolAsync(c93_slot, s93slot, sizeof(int) * s93n, 0, cudaMemcpyHostToDevice, st);
  cudaMemcpyToSymbolAsync(c93_lvEnd, s93lvEnd, sizeof(int) * s93levels, 0, cudaMemcpyHostToDevice, st);
  cudaMemcpyToSymbolAsync(c93_lvJ, s93lvJ, sizeof(int) * s93levels, 0, cudaMemcpyHostToDevice, st);
  cudaMemcpyToSymbolAsync(c93_lvN, s93lvN, sizeof(int) * s93levels, 0, cudaMemcpyHostToDevice, st);
  cudaMemcpyToSymbolAsync(c93_nLevels, &s93levels, sizeof(int), 0, cudaMemcpyHostToDevice, st);
  cudaMemcpyToSymbolAsync(c92_slot, s92slot, sizeof(int) * s92n, 0, cudaMemcpyHostToDevice, st);
  cudaMemcpyToSymbolAsync(c92_lvEnd, s92lvEnd, sizeof(int) * s92levels, 0, cudaMemcpyHostToDevice, st);
  cudaMemcpyToSymbolAsync(c92_lvN, s92lvN, sizeof(int) * s92levels, 0, cudaMemcpyHostToDevice, st);
  cudaMemcpyToSymbolAsync(c92_nLevels, &s92levels, sizeof(int), 0, cudaMemcpyHostToDevice, st);
  cudaMemcpyToSymbolAsync(c92_order, &s92n, sizeof(int), 0, cudaMemcpyHostToDevice, st);
  double n93[32] = {}, n92[32] = {};
#pragma unroll 1
  for (int k = 0; k < s93levels; k++) n93[k] = 3.0 * s93lvN[k];
#pragma unroll 1
  for (int k = 0; k < s92levels; k++) n92[k] = 3.0 * (s92lvN[k] + 1.0);
  cudaMemcpyToSymbolAsync(c93_3n, n93, sizeof n93, 0, cudaMemcpyHostToDevice, st);
  cudaMemcpyToSymbolAsync(c92_3N, n92, sizeof n92, 0, cudaMemcpyHostToDevice, st);
  cudaStreamSynchronize(st);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

}  // namespace ecpgb
