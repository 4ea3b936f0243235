// ecp_exact.cu -- unit stages of the plain FP64 path for sm_103a.
//
// Compiled with --fmad=false: every product and sum rounds as in the
// reference's C, in its order, so the adaptive quadratures see the same partial
// sums and take the same decisions as the CTA-per-unit kernel of ecp_fp64.cu
// (k_unit, kept for the entry point that allocates nothing), bit for bit.  What
// is left out changes no bit: table points that are not reached because every
// quadrature has converged, terms that are exactly zero, the Bessel table's
// derivative recurrence (its rows depend on the table point only, J.besD).
//
// The FP64 pipe bounds these stages (a warp instruction per 16-19 cycles and
// SM, whatever the active lanes; 82 to 84 % busy in all three): only fewer FP64
// instructions make them faster.  So quadratures of several primitive pairs
// share a warp, tables are computed a point a lane, the running quadratures stay
// packed and the products of the last ones are spread over the idle lanes.
// 8 centres of the cluster (14,564 units): small grid 5.4 ms, large grid 8.5, blocks
// 1.4; one kernel with a unit a CTA took 155.6.
#include "ecp_stages.cuh"

namespace ecpgb {

// --------------------------------------------------- stage 2: the small grid

// Level's end of the PS93 walk, operation by operation
// (src/gc_integrators.c:157-217).
static __device__ inline bool ps93_exact(int k, double tol, int cnt, double I, double &p, double &q, double &res) {
  const int j = c93_lvJ[k];
  const double n3 = c93_3n[k];
  double d;
  if (j == 0) {
    p += I - q;
    d = fabs(q - 3 * p / 2);
  } else {
    d = fabs(I - 2 * q);
    q = I;
  }
  if (cnt == 0 || !(16 * d / n3 < tol)) return false;
  res = 16 * q / n3;
  return true;
}

// Whether the walk adds slot t, grid point n (src/gc_integrators.c:157-217): the head
// always, then the lower halves from the window's start and the upper ones to its end.
// Outside the window the reference's tables are 0, and so is the integrand unless
// another factor is infinite or NaN.
static __device__ inline bool ps93_adds(int t, int n, int ws, int we) {
  return t < 3 || ((t & 1) ? n >= ws : n <= we);
}

// A group of G primitive pairs of one kind (perm[p0 ..]) on the small grid
// (src/type1.c:63-148), by one warp; lane = (pair, quadrature).
template <bool kInRange, bool kZero>
static __device__ void x1_small(const DevJob &J, const Unit &U, const SmallSmem &L, double *sm, int off, int p0,
                                int G) {
  const int lane = threadIdx.x & 31, lab = U.lab, lq = lab + 1, O = kSmallOrder, ws = U.ws, we = U.we;
  const int TS = 1 + 2 * lq, nq = t1_items(lab);
  double *rec = sm + L.rec, *tab = sm + L.tab;  // the pairs' records
  const unsigned char *perm = (const unsigned char *)(U.scr + U.L.perm);
  const double *uL = J.uL + (size_t)U.c * O;
  __syncwarp();
#pragma unroll 1
  for (int e = lane; e < G * kPairWords; e += 32)
    rec[e] = ((const double *)(U.scr + U.L.pair))[perm[p0 + e / kPairWords] * kPairWords + e % kPairWords];
  __syncwarp();
  const bool mine = lane < G * nq;
  const int g = mine ? lane / nq : 0, qi = mine ? lane % nq : 0;
  int l1 = 0, l2 = 0;
  {
    int rem = qi;
    while (l1 <= lab && rem >= l1 / 2 + 1) { rem -= l1 / 2 + 1; l1++; }
    l2 = l1 - 2 * rem;
  }
  double *Qout = (double *)(U.scr + U.L.Q) + (size_t)perm[p0 + g] * nq + qi;
  double I = 0, p = 0, q = 0, T = 0;
  int *quad = (int *)(sm + L.quad);  // the running quadratures, by rank
  bool done = !mine;
  int k = -2, cnt = 0, lvEnd = 1;
  if (kZero) {
    if (mine) {
      done = t1_zero_walk(J, rec[g * kPairWords], rec[g * kPairWords + 2], ws, we);
      if (done) *Qout = 0.0;
    }
  } else
#pragma unroll 1
  for (int s0 = 0; s0 < O;) {
    const int s1 = step_end93(s0) < O ? step_end93(s0) : O, ns = s1 - s0;
    // the step's in-window slots are the run [lo, hi) of its by-point order
    const int m0 = lane < ns ? __ldg(J.byN93 + s0 + lane) >> 16 : INT_MAX;
    const int m1 = lane + 32 < ns ? __ldg(J.byN93 + s0 + lane + 32) >> 16 : INT_MAX;
    const int lo = __popc(__ballot_sync(0xffffffffu, m0 < ws)) + __popc(__ballot_sync(0xffffffffu, m1 < ws));
    const int hi = __popc(__ballot_sync(0xffffffffu, m0 < we)) + __popc(__ballot_sync(0xffffffffu, m1 < we));
    const int nIn = hi - lo;
    // the pairs with a quadrature still running
    unsigned live = 0;
    const unsigned run = __ballot_sync(0xffffffffu, !done), qm = nq >= 32 ? ~0u : (1u << nq) - 1u;
#pragma unroll 1
    for (int gg = 0; gg < G; gg++)
      if (run >> (gg * nq) & qm) live |= 1u << gg;
    const int nLive = __popc(live);
#pragma unroll 1
    for (int e = lane; e < nIn * nLive; e += 32) {
      const int i = e / nLive, gg = __fns(live, 0, e - i * nLive + 1), tn = __ldg(J.byN93 + s0 + lo + i),
                t = tn & 0xffff, n = tn >> 16;
      // entry: K_l, then (C1 r^l) U, then the exponential
      double *ent = tab + ((t - s0) * G + gg) * TS, *WR = ent + lq;
      const PairRec &P = *(const PairRec *)(rec + gg * kPairWords);
      const double r = J.xSmall[n], s = P.s, C1 = P.C1, ex = (P.z * r + s) * r, u = uL[n];
      // below the screen the exponential is 0, and so is the product where it is finite
      const bool seen = ex >= J.lnAcc1;
      if (seen || !kInRange) {
        bessel_rows(J, lab, s * r, ent);
        double R = 1.0;
#pragma unroll 1
        for (int l = 0; l <= lab; l++) {
          WR[l] = C1 * R * u;
          R = r * R;
        }
        ent[2 * lq] = seen ? exp(ex) : 0.0;
      } else {
        ent[2 * lq] = 0.0;  // marks a zero point
      }
    }
    __syncwarp();
    // the lanes dealt to the running quadratures: P points' products side by side,
    // added in the reference's order by the quadrature's own lane
    const unsigned act = __ballot_sync(0xffffffffu, !done);
    const LaneDeal D = deal_lanes(__popc(act));
    const int rank = __popc(act & ((1u << lane) - 1u)), src = rank * D.P;
    if (!done) quad[rank] = g | l1 << 8 | l2 << 16;
    __syncwarp();
    const bool work = D.rank < __popc(act);
    const int qd = work ? quad[D.rank] : 0;
    const int oW = lq + ((qd >> 8) & 255), oK = qd >> 16;
#pragma unroll 1
    for (int t0 = s0; t0 < s1; t0 += D.P) {
      double v = 0.0;
      if (work && t0 + D.part < s1) {
        const int n = __ldg(J.s93 + t0 + D.part);
        if (n >= ws && n < we) {
          const double *e = tab + ((t0 + D.part - s0) * G + (qd & 255)) * TS;
          if (e[2 * lq] != 0.0 || !kInRange) v = J.wSmall[n] * (e[oW] * e[oK] * e[2 * lq]);
        } else if (!kInRange) {
          v = J.wSmall[n] * (((const PairRec *)(rec + (qd & 255) * kPairWords))->C1 * 0.0);
        }
      }
#pragma unroll 1
      for (int j = 0; j < D.P && t0 + j < s1; j++) {
        const int t = t0 + j, n = c93_slot[t];
        if ((n >= ws && n < we) || (!kInRange && ps93_adds(t, n, ws, we)))
          T += __shfl_sync(0xffffffffu, v, (src + j) & 31);
        cnt += (t & 1) ? n >= ws : n <= we;
        if (t > 2 && !(t & 1)) {  // the reference's order: pair by pair
          I += T;
          T = 0.0;
        }
        if (t + 1 < lvEnd) continue;
        if (!done) {
          double res;
          if (k == -2) p = T;
          else if (k == -1) {
            q = T;
            I = p + q;
          } else if (ps93_exact(k, J.tol, cnt, I, p, q, res)) {
            done = true;
            *Qout = res;
          }
        }
        T = 0.0;
        k++;
        lvEnd = k < 0 ? 3 : c93_lvEnd[k];  // k <= the level count, inside the 32-entry table
        cnt = 0;
      }
    }
    __syncwarp();
    s0 = s1;
    if (__all_sync(0xffffffffu, done)) break;
  }
  const unsigned fail = __ballot_sync(0xffffffffu, mine && !done);
#pragma unroll 1
  for (int gg = 0; fail && gg < G; gg++) {
    const unsigned m = fail >> (gg * nq) & (nq >= 32 ? ~0u : (1u << nq) - 1u);
    if (m && lane == 0) J.listFail[atomicAdd(J.counters + kCntFail, 1u)] = {off, perm[p0 + gg], m, 0, rec[gg * kPairWords]};
  }
}

// A batch of 32 type-2 small-grid quadratures, one per lane (src/type2.c:337-387).
template <bool kInRange>
static __device__ void x2_small(const DevJob &J, const Unit &U, int q0) {
  const int qx = q0 + (threadIdx.x & 31), O = kSmallOrder;
  if (qx >= U.nItems) return;
  const int nF = J.nF, nk = J.nk, LE = J.maxLECP > 0 ? J.maxLECP : 1, nRuns = J.nRuns > 0 ? J.nRuns : 1;
  const int v = unit_item(J, U, qx), l = v & 255, l1 = (v >> 8) & 255, l2 = (v >> 16) & 255, l3 = v >> 24;
  const double *Fa = J.F + (((size_t)U.c * J.nShells + U.sa) * nRuns + U.pa0) * O * nF + l1;
  const double *Fb = J.F + (((size_t)U.c * J.nShells + U.sb) * nRuns + U.pb0) * O * nF + l2;
  const double *Ut = J.utab + (size_t)U.c * O * LE * nk + l * nk + l3;
  double I = 0, p = 0, q = 0, T = 0, res;
  int k = -2, lvEnd = 1, cnt = 0;
#pragma unroll 1
  for (int t = 0;; t++) {
    const int n = c93_slot[t];
    // (F is zero outside the windows)
    if ((n >= U.ws && n < U.we) || (!kInRange && ps93_adds(t, n, U.ws, U.we)))
      T += J.wSmall[n] * (__ldg(Fa + n * nF) * __ldg(Fb + n * nF) * __ldg(Ut + (size_t)n * LE * nk));
    cnt += (t & 1) ? n >= U.ws : n <= U.we;
    if (t > 2 && !(t & 1)) {
      I += T;
      T = 0.0;
    }
    if (t + 1 < lvEnd) continue;
    if (k == -2) p = T;
    else if (k == -1) {
      q = T;
      I = p + q;
    } else if (ps93_exact(k, J.tol, cnt, I, p, q, res)) {
      ((double *)(U.scr + U.L.T))[qx] = res;
      return;
    }
    T = 0.0;
    if (++k >= c93_nLevels) break;
    lvEnd = k < 0 ? 3 : c93_lvEnd[k];
    cnt = 0;
  }
  atomicOr((unsigned *)(U.scr + U.L.mask) + (qx >> 5), 1u << (qx & 31));
}

// kInRange: no product leaves FP64's range, so what has a factor 0 is 0 (DevJob::inRange).
template <bool kInRange>
__global__ void __launch_bounds__(32, 16) k_exact_small(DevJob J) {
  extern __shared__ double sm[];
  const SmallSmem L = small_layout(J.maxLBS, 0, J.gcap);
  const int n0 = (int)J.counters[kCntT1], n1 = n0 + (int)J.counters[kCntRest], n = n1 + (int)J.counters[kCntT2];
#pragma unroll 1
  for (int taken = 0; taken < J.take; taken++) {
    const int i = next_item(J.counters + kHeadSmall);
    if (i >= n) return;
    const int2 it = small_entry(J, i, n0, n1);
    const Unit &U = unit_get(J, it.x);
    if (i >= n1) {
      x2_small<kInRange>(J, U, it.y);
      continue;
    }
    const int p0 = it.y & 1023, G = (it.y >> 10) & 63;
    if (it.y >> 16 == kPairZero) x1_small<kInRange, true>(J, U, L, sm, it.x, p0, G);
    else x1_small<kInRange, false>(J, U, L, sm, it.x, p0, G);
  }
}

// --------------------------------------------------- stage 3: the large grid

// PSM92 walk (src/gc_integrators.c:39-86) over the slots [s0, s1), of which
// slots[0 .. nE) have an integrand that is not zero (adding zero changes no sum), in
// the reference's operation order.  D.P lanes evaluate a quadrature's points side by
// side, val(x) of entry x for the quadrature of the lane's deal; the lane that holds
// the quadrature of rank src / D.P adds them up.
template <class V, class Vis>
static __device__ inline void psm92_exact(int s0, int s1, const int *slots, int nE, const LaneDeal &D, int src,
                                          double tol, V val, Vis vis, double &I, double &p, double &q, bool &done,
                                          double &res) {
  int pos = s0, i = 0, k = s0 == 0 ? -1 : level_of(s0);
#pragma unroll 1
  while (pos < s1) {
    const int lvStart = k <= 0 ? 1 : c92_lvEnd[k - 1], lvE = k < 0 ? 1 : c92_lvEnd[k];
    if (pos == lvStart && k >= 0) {
      q = 2 * p;
      p = 2 * I;
    }
    const int stop = lvE < s1 ? lvE : s1;
    double T = 0.0;
    int last = -1;  // the (lower, upper) pair T belongs to
#pragma unroll 1
    while (i < nE && slots[i] < stop) {
      int m = 1;
      while (m < D.P && i + m < nE && slots[i + m] < stop) m++;
      const double v = D.part < m ? val(i + D.part) : 0.0;
#pragma unroll 1
      for (int j = 0; j < m; j++, i++) {
        const int t = slots[i], pr = (t + 1) >> 1;
        if (pr != last) {
          I += T;
          T = 0.0;
          last = pr;
        }
        const double x = __shfl_sync(0xffffffffu, v, (src + j) & 31);
        if ((t & 1) || t == 0 || vis(t)) T += x;
      }
    }
    I += T;
    pos = stop;
    if (pos == lvE) {
      if (k < 0) p = I;
      else if (!done) {
        const double N3 = c92_3N[k], e = I - p;
        if (16 * e * e <= N3 * fabs(I - q) * tol) {
          res = 16 * I / N3;
          done = true;
        }
      }
      k++;
    }
    if (__all_sync(0xffffffffu, done)) break;
  }
}

// The failed large-grid quadratures of one type-1 primitive pair
// (src/type1.c:149-196), one per lane.
static __device__ void x1_large(const DevJob &J, const Unit &U, const LargeSmem &L, double *sm, int kk, unsigned mask,
                                double s) {
  const int lane = threadIdx.x & 31, lab = U.lab, lq = lab + 1, O = kSmallOrder, OL = J.largeOrder, TS = 1 + 2 * lq;
  const int Nb = U.Nb, ws = U.ws, we = U.we, c = U.c, Lc = U.Lc;
  double *tab = sm + L.tab;
  int *slots = (int *)(sm + L.pend), *quad = (int *)(sm + L.fail);  // the step's entries; the running quadratures
  const double *uL = J.uL + (size_t)c * O;
  const double dAC = U.gA[3], dBC = U.gB[3];
  const bool fail = mask >> lane & 1u;
  int l1 = 0, l2 = 0;
  {
    int rem = lane;
    while (l1 <= lab && rem >= l1 / 2 + 1) { rem -= l1 / 2 + 1; l1++; }
    l2 = l1 - 2 * rem;
  }
  const double za = U.pzA[kk / Nb], zb = U.pzB[kk % Nb];
  const double ca = zeta_times(U.pcA[kk / Nb], za, U.pa0), cb = zeta_times(U.pcB[kk % Nb], zb, U.pb0);
  const double z = -za - zb, zd2 = -za * dAC * dAC - zb * dBC * dBC, C2 = ca * cb;
  const double2 map = ((const double2 *)(U.scr + U.L.map))[kk];
  const double i1 = map.x, i2 = map.y;
  // the break: the first point past both centres whose exponent is below the
  // screen (the predicate is monotone there: a 32-way search in two rounds)
  auto brk = [&](int n) {
    const double r = i1 * J.xLarge[n] + i2, e = (z * r + s) * r + zd2;
    return r > dAC && r > dBC && e < J.lnAcc1;
  };
  const int chunk = (OL + 31) / 32;
  int nb = OL;
  {
    const int n = lane * chunk + chunk - 1 < OL ? lane * chunk + chunk - 1 : OL - 1;
    const unsigned b = __ballot_sync(0xffffffffu, brk(n));
    if (b) {
      const int n0 = (__ffs(b) - 1) * chunk;
#pragma unroll 1
      for (int c0 = n0; c0 < n0 + chunk && c0 < OL; c0 += 32) {
        const int m = c0 + lane;
        const unsigned b2 = __ballot_sync(0xffffffffu, m < n0 + chunk && m < OL && brk(m));
        if (b2) {
          nb = c0 + __ffs(b2) - 1;
          break;
        }
      }
    }
  }
  const int end = nb - 1;
  double I = 0, p = 0, q = 0, res = 0;
  bool done = !fail;
#pragma unroll 1
  for (int s0 = 0; s0 < OL;) {
    const int s1 = step_end92(s0) < OL ? step_end92(s0) : OL;
    const int kq = __reduce_max_sync(0xffffffffu, done ? 0 : l2);
    const int rq = __reduce_max_sync(0xffffffffu, done ? 0 : l1);
    const int t = s0 + lane;
    bool any = false;
    if (t < s1) {
      const int n = __ldg(J.s92 + t);
      const bool upper = t > 0 && !(t & 1);
      // entry: K_l, then (C2 r^l) U, then the exponential
      double *K = tab + lane * TS, *WR = K + lq;
      if (n < nb) {
        const double r = i1 * J.xLarge[n] + i2, ex = (z * r + s) * r + zd2;
        if (ex >= J.lnAcc1) {
          any = true;
          bessel_rows(J, kq, s * r, K);
          const double u = eval_ecp(J, c, Lc, r);
          double R = 1.0;
#pragma unroll 1
          for (int l = 0; l <= rq; l++) {
            WR[l] = C2 * R * u;
            R = r * R;
          }
          K[2 * lq] = exp(ex);
        }
      } else if (n != nb && !upper && n < O && n >= ws && n < we) {
        // beyond the break the reference integrates its small-grid buffers:
        // exponent and U_L at index n, r^l and K_l at flat offset l*OL + n of
        // rows written with the small grid's stride
        const double rs = J.xSmall[n], es = (z * rs + s) * rs;
        if (es >= J.lnAcc1) {
          any = true;
          K[2 * lq] = exp(es);
          double row[kMaxRows];
#pragma unroll 1
          for (int l = 0; l <= lab; l++) {
            const int f = l * OL + n, lr = f / O, nr = f % O;
            const bool ok = lr <= lab && nr >= ws && nr < we;
            double xr = J.xSmall[nr], pw = 1.0;
#pragma unroll 1
            for (int i = 0; i < lr && ok; i++) pw = xr * pw;
            if (ok) bessel_rows(J, lr, s * xr, row);
            WR[l] = C2 * (ok ? pw : 0.0) * uL[n];
            K[l] = ok ? row[lr] : 0.0;
          }
        }
      }
    }
    const unsigned b = __ballot_sync(0xffffffffu, any), act = __ballot_sync(0xffffffffu, !done);
    const unsigned below = (1u << lane) - 1u;
    const LaneDeal D = deal_lanes(__popc(act));
    const int rank = __popc(act & below), src = rank * D.P;
    if (any) slots[__popc(b & below)] = t;
    if (!done) quad[rank] = l1 | l2 << 16;
    __syncwarp();
    const bool work = D.rank < __popc(act);
    const int qd = work ? quad[D.rank] : 0;
    const int oW = lq + (qd & 0xffff), oK = qd >> 16;
    auto vis = [&](int t) { return c92_slot[t] <= end; };
    auto val = [&](int x) {
      const int t = slots[x];
      const double *e = tab + (t - s0) * TS;
      return work ? J.wLarge[__ldg(J.s92 + t)] * i1 * (e[oW] * e[oK] * e[2 * lq]) : 0.0;
    };
    psm92_exact(s0, s1, slots, __popc(b), D, src, J.tol, val, vis, I, p, q, done, res);
    __syncwarp();
    s0 = s1;
    if (__all_sync(0xffffffffu, done)) break;
  }
  if (fail) {
    if (!done) {
      res = 16 * I / c92_3N[c92_nLevels - 1];
      atomicOr(&((UnitHead *)U.scr)->warn, 1);
    }
    ((double *)(U.scr + U.L.Q))[(size_t)kk * t1_items(lab) + lane] = res;
  }
  __syncwarp();
}

// The failed type-2 quadratures of a unit on primitive pair k's large grid
// (src/type2.c:418-528), in passes of up to kWalkCap of them; each result is
// kept for the pair.
static __device__ void x2_large(const DevJob &J, const Unit &U, const LargeSmem &L, double *sm, int k) {
  const int lane = threadIdx.x & 31, nIt = U.nItems, nA = 2 * J.maxLBS + 1, Nb = U.Nb, c = U.c;
  const int LE = J.maxLECP > 0 ? J.maxLECP : 1, LBE = J.maxLBS + LE, OL = J.largeOrder, TS = L.tabStride;
  const unsigned *mask = (const unsigned *)(U.scr + U.L.mask);
  const double2 *map = (const double2 *)(U.scr + U.L.map);
  const int4 *win = (const int4 *)(U.scr + U.L.win);
  double *dst = U.NP == 1 ? (double *)(U.scr + U.L.T)
                          : (double *)(U.scr + U.L.part) + (size_t)k * class_items(J, U.cls * LE, LE);
  double *tab = sm + L.tab, *sI = sm + L.I, *sP = sm + L.P, *sQ = sm + L.Q;
  int *fail = (int *)(sm + L.fail), *pend = (int *)(sm + L.pend);
  unsigned char *act = (unsigned char *)(sm + L.act);  // the running items
  const double dAC = U.gA[3], dBC = U.gB[3];
  const double za = U.pzA[k / Nb], zb = U.pzB[k % Nb];
  const double Ck = zeta_times(zeta_times(U.pcA[k / Nb] * U.pcB[k % Nb], za, U.pa0), zb, U.pb0);
  const double i1 = map[k].x;
  const int4 wk = win[k];
  const int nb = wk.x, end = nb == INT_MAX ? OL - 1 : nb - 1, nLo = wk.y, nHi = wk.z;
  // the latest break of the earlier pairs: beyond it no earlier pair's
  // buffers are reused
  int mb = -1;
#pragma unroll 1
  for (int j = lane; j < k; j += 32) mb = win[j].x > mb ? win[j].x : mb;
  mb = __reduce_max_sync(0xffffffffu, mb);
  const unsigned below = (1u << lane) - 1u;
  // whose tables slot t reads (the reference's reused buffers): this pair's
  // below its break; beyond it, on the lower half, the last earlier pair
  // whose loop reached that point; the point and exponent of that pair
  auto locate = [&](int t, int &owner, double &r, double &ex) {
    const int n = __ldg(J.s92 + t);
    owner = -1;
    if (n < nb) owner = k;
    else if (n != nb && (t == 0 || (t & 1))) {
#pragma unroll 1
      for (int j = k - 1; j >= 0; j--)
        if (win[j].x >= n) { owner = j; break; }
      if (owner >= 0 && win[owner].x == n) owner = -1;
    }
    if (owner < 0) return;
    r = map[owner].x * J.xLarge[n] + map[owner].y;
    const double d1 = dAC - r, d2 = dBC - r;
    ex = -U.pzA[owner / Nb] * d1 * d1 - U.pzB[owner % Nb] * d2 * d2;
  };
  int q0 = 0;
#pragma unroll 1
  while (q0 < nIt) {
    // the pass's items, decoded once
    int nf = 0, pL1 = 0, pL2 = 0, pL3 = 0;
    unsigned pMask = 0;
    const int first = q0;
#pragma unroll 1
    for (; q0 < nIt; q0 += 32) {
      const unsigned m = mask[q0 >> 5];
      if (nf + __popc(m) > kWalkCap) break;
      if (m >> lane & 1u) {
        const int v = unit_item(J, U, q0 + lane);
        fail[nf + __popc(m & below)] = v;
        pMask |= 1u << (v & 255);
        pL1 = pL1 > ((v >> 8) & 255) ? pL1 : (v >> 8) & 255;
        pL2 = pL2 > ((v >> 16) & 255) ? pL2 : (v >> 16) & 255;
        pL3 = pL3 > (v >> 24) ? pL3 : v >> 24;
      }
      nf += __popc(m);
    }
    if (nf == 0) continue;
    pMask = __reduce_or_sync(0xffffffffu, pMask);
    pL1 = __reduce_max_sync(0xffffffffu, pL1);
    pL2 = __reduce_max_sync(0xffffffffu, pL2);
    pL3 = __reduce_max_sync(0xffffffffu, pL3);
#pragma unroll 1
    for (int q = lane; q < nf; q += 32) {
      act[q] = (unsigned char)q;
      sI[q] = sP[q] = sQ[q] = 0;
    }
    __syncwarp();
    int cpos = 0, wpos = 0, nPend = 0, nAct = nf;
#pragma unroll 1
    while (wpos < OL) {
      // classify slots step by step, queue the needed ones
#pragma unroll 1
      while (nPend < 32 && cpos < OL) {
        const int c1 = step_end92(cpos) < OL ? step_end92(cpos) : OL, t = cpos + lane;
        bool need = false;
        if (t < c1) {
          const int n = __ldg(J.s92 + t);
          if (n < nb ? n >= nLo && n <= nHi : n <= mb && n != nb && (t == 0 || (t & 1))) {
            int owner;
            double r, ex;
            locate(t, owner, r, ex);
            need = owner >= 0 && ex >= J.lnAcc2;
          }
        }
        const unsigned m = __ballot_sync(0xffffffffu, need);
        if (need) pend[nPend + __popc(m & below)] = t;
        nPend += __popc(m);
        cpos = c1;
      }
      __syncwarp();
      // this pass: the first queued slots, up to an odd slot (whole (lower,
      // upper) pairs) that no queued slot precedes
      int nE = nPend < 32 ? nPend : 32, b = cpos;
      if (nPend > 32) {
        b = pend[32];
        if (!(b & 1)) b -= 1;
        while (nE > 0 && pend[nE - 1] >= b) nE--;
      }
      if (lane < nE) {
        const int t = pend[lane], n = __ldg(J.s92 + t);
        int owner;
        double r, ex;
        locate(t, owner, r, ex);
        double *Uc = tab + lane * TS, *R = Uc + LE, *Ka = R + nA, *Kb = Ka + LBE;
        Kb[LBE] = exp(ex);
        Kb[LBE + 1] = J.wLarge[n] * i1;
#pragma unroll 1
        for (int l = 0; l < LE; l++)
          if (pMask >> l & 1u) Uc[l] = Ck * eval_ecp(J, c, l, r);
        bessel_rows(J, pL1, 2.0 * U.pzA[owner / Nb] * dAC * r, Ka);
        bessel_rows(J, pL2, 2.0 * U.pzB[owner % Nb] * dBC * r, Kb);
        R[0] = 1.0;
#pragma unroll 1
        for (int l = 1; l <= pL3; l++) R[l] = r * R[l - 1];
      }
      __syncwarp();
      unsigned nMask = 0u;
      int n1 = 0, n2 = 0, n3 = 0, left = 0;
      // the running items, 32 at a time, the last ones by several lanes each
#pragma unroll 1
      for (int i0 = 0; i0 < nAct;) {
        const LaneDeal D = deal_lanes(nAct - i0);
        const bool work = i0 + D.rank < nAct;  // the item the lane evaluates
        const int v = work ? fail[act[i0 + D.rank]] : 0;
        const double *eU = tab + (v & 255), *eR = tab + LE + (v >> 24), *eA = tab + LE + nA + ((v >> 8) & 255),
                     *eB = tab + LE + nA + LBE + ((v >> 16) & 255), *eK = tab + LE + nA + 2 * LBE;
        auto val = [&](int x) {
          const int o = x * TS;
          return work ? eK[o + 1] * (eU[o] * eR[o] * eA[o] * eB[o] * eK[o]) : 0.0;
        };
        auto vis = [&](int t) { return c92_slot[t] <= end; };
        // the item whose sums the lane holds
        const bool mine = lane < 32 / D.P && i0 + lane < nAct;
        const int q = mine ? act[i0 + lane] : 0;
        double I = sI[q], p = sP[q], qv = sQ[q], res = 0;
        bool done = !mine;
        psm92_exact(wpos, b, pend, nE, D, lane * D.P, J.tol, val, vis, I, p, qv, done, res);
        __syncwarp();
        if (mine) {
          sI[q] = done ? res : I;
          sP[q] = p;
          sQ[q] = qv;
        }
        const bool keep = mine && !done;
        if (keep) {
          const int u = fail[q], l1 = (u >> 8) & 255, l2 = (u >> 16) & 255, l3 = u >> 24;
          nMask |= 1u << (u & 255);
          n1 = l1 > n1 ? l1 : n1;
          n2 = l2 > n2 ? l2 : n2;
          n3 = l3 > n3 ? l3 : n3;
        }
        // the list shrinks in place
        const unsigned km = __ballot_sync(0xffffffffu, keep);
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
      // drop the evaluated slots from the queue
      const int rest = nPend - nE;
      const int keep0 = lane < rest ? pend[nE + lane] : 0, keep1 = lane + 32 < rest ? pend[nE + lane + 32] : 0;
      __syncwarp();
      if (lane < rest) pend[lane] = keep0;
      if (lane + 32 < rest) pend[lane + 32] = keep1;
      nPend = rest;
      wpos = b;
      __syncwarp();
      if (nAct == 0) break;
    }
    const double N3 = c92_3N[c92_nLevels - 1];
#pragma unroll 1
    for (int i = lane; i < nAct; i += 32) {
      sI[act[i]] = 16 * sI[act[i]] / N3;
      atomicOr(&((UnitHead *)U.scr)->warn, 2);
    }
    __syncwarp();
    int at = 0;
#pragma unroll 1
    for (int w = first; w < q0; w += 32) {
      const unsigned m = mask[w >> 5];
      if (m >> lane & 1u) dst[w + lane] = sI[at + __popc(m & below)];
      at += __popc(m);
    }
    __syncwarp();
  }
}

__global__ void __launch_bounds__(32, 14) k_exact_large(DevJob J) {
  extern __shared__ double sm[];
  const LargeSmem L = large_layout(J.maxLBS, J.maxLECP, true);
  const int n2 = (int)J.counters[kCntPart], n = n2 + (int)J.counters[kCntFail];
#pragma unroll 1
  for (int taken = 0; taken < J.take; taken++) {
    const int i = next_item(J.counters + kHeadLarge);
    if (i >= n) return;
    if (i < n2) {
      const int2 it = J.listPart[i];
      const Unit &U = unit_get(J, it.x);
      x2_large(J, U, L, sm, it.y);
    } else {
      const T1Fail it = J.listFail[i - n2];
      const Unit &U = unit_get(J, it.off);
      x1_large(J, U, L, sm, it.k, it.mask, it.s);
    }
  }
}

// -------------------------------------------------------- stage 4: the blocks

// Type-1 block (src/type1.c:266-295): per primitive pair in order, S_lm of its
// k-vector and the terms of every combined Cartesian index.
__global__ void __launch_bounds__(kLinkThreadsMax) k_exact_link(DevJob J) {
  extern __shared__ double sm[];
  const Unit U = unit_load(J, J.chunk0 + blockIdx.x);
  if (!U.live) return;
  const LinkSmem Lm = link_layout(J.maxLBS, J.maxLECP);
  const bool one = blockIdx.y == 0, two = blockIdx.y == gridDim.y - 1;  // the blocks this CTA makes
  const int tid = threadIdx.x, NT = blockDim.x, lab = U.lab, lq = lab + 1, Nb = U.Nb, RQ = lq * lq;
  double *rsh = sm + Lm.rsh, *dir = sm + Lm.dir, *H = sm + Lm.H;
  const int dd = J.tmDim + 1, tmW = (J.tmDim + 1) * (J.tmDim + 1), nq = t1_items(lab), nH = NCUM(lab);
  const double *Q = (const double *)(U.scr + U.L.Q);
#pragma unroll 1
  for (int e = tid; e < nH; e += NT) H[e] = 0.0;
#pragma unroll 1
  for (int b0 = one ? 0 : U.NP; b0 < U.NP; b0 += kLinkBatch) {
    const int nb = U.NP - b0 < kLinkBatch ? U.NP - b0 : kLinkBatch;
    __syncthreads();
    // cos(theta), phi and its sine and cosine, then S_lm a column a thread
    if ((tid & 31) < nb && tid < 96) {
      const int g = tid & 31, k = b0 + g;
      const double za = U.pzA[k / Nb], zb = U.pzB[k % Nb];
      double P[3], S[3];
      for (int i = 0; i < 3; i++) P[i] = 2.0 * (za * U.gA[i] + zb * U.gB[i]);
      to_spherical(P, S);
      if (tid < 32) {
        dir[4 * g] = cos(S[1]);
        dir[4 * g + 1] = S[2];
      } else if (tid < 64) dir[4 * g + 2] = sin(S[2]);
      else dir[4 * g + 3] = cos(S[2]);
    }
    __syncthreads();
#pragma unroll 1
    for (int e = tid; e < nb * lq; e += NT) {
      const double *d = dir + 4 * (e / lq);
      real_sph_column(J, lab, e % lq, d[0], d[1], d[2], d[3], rsh + (e / lq) * RQ);
    }
    __syncthreads();
#pragma unroll 1
    for (int pi = tid; pi < nH; pi += NT) {
      const int *ex = J.ijk + 3 * pi;
      const int lmax = ex[0] + ex[1] + ex[2];
      const double *p2s = J.p2s + (size_t)J.ijkIdx[(ex[0] * dd + ex[1]) * dd + ex[2]] * tmW;
      double acc = H[pi];
#pragma unroll 1
      for (int g = 0; g < nb; g++) {
        const double *rs = rsh + g * RQ, *q = Q + (size_t)(b0 + g) * nq + t1_index(lmax, lmax);
#pragma unroll 1
        for (int l = lmax; l >= 0; l -= 2, q++) {
          double factor = 0.0;
#pragma unroll 1
          for (int m = 0; m < 2 * l + 1; m++) factor += rs[l * l + m] * p2s[l * l + m];
          acc += factor * *q;
        }
      }
      H[pi] = acc;
    }
  }
  __syncthreads();
  link_finish<true>(J, U, Lm, sm, one, two);
}

// --------------------------------------------------------------- launchers

int upload_schedules_exact(const int *s93slot, int s93n, const int *s93lvEnd, const int *s93lvJ,
                           const int *s93lvN, int s93levels, const int *s92slot, int s92n,
                           const int *s92lvEnd, const int *s92lvN, int s92levels, void *stream) {
  return upload_stage_schedules(s93slot, s93n, s93lvEnd, s93lvJ, s93lvN, s93levels, s92slot, s92n, s92lvEnd, s92lvN,
                                s92levels, stream);
}

void exact_prepare() {
  // function attributes are per device; callers hold the engine lock
  static bool attr[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || attr[dev]) return;
  for (const void *k : {(const void *)k_exact_small<true>, (const void *)k_exact_small<false>,
                        (const void *)k_exact_large, (const void *)k_exact_link}) {
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
  }
  attr[dev] = true;
}

int launch_exact_pipeline(const DevJob &J, cudaStream_t st, cudaEvent_t u0, cudaEvent_t u1) {
  exact_prepare();
  DevJob Jc = J;
  Jc.gcap = FastConfig{}.gcap;
  Jc.balance = FastConfig{}.balance;
  Jc.live = nullptr;
  const JobPlan::Order &ord = use_order(Jc, FastConfig{}.sorted);
  const size_t sSmall = sizeof(double) * (size_t)small_layout(J.maxLBS, 0, Jc.gcap).total;
  const size_t sLarge = sizeof(double) * (size_t)large_layout(J.maxLBS, J.maxLECP, true).total;
  const size_t sLink = sizeof(double) * (size_t)link_layout(J.maxLBS, J.maxLECP).total;
  if (sSmall > 200 * 1024 || sLarge > 200 * 1024 || sLink > 200 * 1024) return 3;
  launch_stage1(Jc, st);
  launch_shell_F(Jc, st);
  if (u0) record_timing(u0, st);
  launch_chunks(Jc, ord, st, [&](const DevJob &C, unsigned units, unsigned gSmall, int takeSmall, unsigned gLarge,
                                 int takeLarge) {
    DevJob K = C;
    k_unit_plan<true><<<(units + 3) / 4, kPlanThreads, 0, st>>>(K);
    K.take = takeSmall;
    (J.inRange ? k_exact_small<true> : k_exact_small<false>)<<<gSmall, 32, sSmall, st>>>(K);
    K.take = takeLarge;
    k_exact_large<<<gLarge, 32, sLarge, st>>>(K);
    k_exact_link<<<dim3(units, link_parts(units)), link_threads(sLink), sLink, st>>>(K);
  });
  if (u1) record_timing(u1, st);
  launch_epilogue(Jc, st);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : kLaunchErrorBase + (int)e;
}

}  // namespace ecpgb
