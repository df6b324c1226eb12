// Point-implicit reaction substep by a group of GL = 3 lanes, NS / GL species
// a lane (ten nodes a warp).  The same model as the runtime-count path in
// chem.cu/chem.cuh (reference src/FiniteRateChem.cu:1466-1822,
// src/StrangSplitting.cu:43-224).  A node's substeps are a serial chain, so
// what counts is the instructions of a substep, its latency, and how many
// warps hide it:
//  * the lanes share the reactions (rates), the species (thermodynamics) and
//    the columns of the matrix;
//  * a forward rate takes one exponential and a backward one a second, of the
//    difference of the sides' g_k: only that difference is as small as the
//    reaction's own energy.  One exponential a species instead (activities
//    c_k exp(g_k), and exp(-sum of the reactants' g_k) in the rate constant)
//    carries the rounding of sums that reach 160 into every rate, and leaves
//    the range of a double where g_k depends on an element's reference state;
//  * the matrix is in molar units (rows and columns scaled by the molar
//    masses), in which its diagonal is mostly the largest entry of its column,
//    and is solved by Gauss-Jordan elimination with partial pivoting in
//    registers, three columns a lane, the multipliers passed on by shuffles;
//  * the mechanism tables are in shared memory, every factor a double.
// Lanes a node, measured on 2^20 H2/air reactors of 4-64 substeps each and on
// 1021 of them (ms): one, with the matrix in its registers, 31.9 and 2.72 (255
// registers, 8 warps an SM, 80 000 cycles a substep); nine, a row each, 52.6
// and 0.73 (a node takes four times the instructions); three, 26.0 and 0.71
// with an exponential a species, 27.2 and 0.73 with one a backward rate, which
// halves the time scale's error (3.5e-15 and 1.4e-15 against 64-bit values).
// One lane with the matrix in shared memory, before, took 49.7 and 4.54.
// Results match the runtime-count path to rounding.
#pragma once

#include "chem.cuh"
#include "thermo.cuh"

namespace cfk {

template <int NS>
__device__ __forceinline__ void enthalpy_cp_ns(const Thermo *th, double t, double *h, double *cp) {
#pragma unroll
  for (int i = 0; i < NS; ++i) enthalpy_cp_one(th, i, t, h[i], cp[i]);
}

// G_i / (R T), held at the end of the species' range outside it.
__device__ __forceinline__ double gibbs_one(const double *low, const double *high, double t_low, double t_mid,
                                            double t_high, double t, double lnT, double iT) {
  const double *c = t < t_mid ? low : high;
  double tt = t, ln = lnT, it = iT;
  if (t < t_low || t > t_high) {
    tt = t < t_low ? t_low : t_high;
    ln = log(tt);
    it = 1.0 / tt;
  }
  const double p = fma(tt, fma(tt, fma(tt, 0.05 * c[4], (1.0 / 12) * c[3]), (1.0 / 6) * c[2]), 0.5 * c[1]);
  return fma(c[0], 1.0 - ln, fma(c[5], it, fma(-tt, p, -c[6])));
}

// In GroupTables::mol[r].x: a side has more than kMaxMol molecules.
constexpr unsigned kLongSide = 1u << 24;
static_assert(kMaxMol <= 3, "three bytes of molecules and the flag");

// Mechanism tables of a CTA in shared memory, species by position.
template <int NS>
struct GroupTables {
  static constexpr int LD = (NS + 1) / 2 * 2;  // rows start on 16 bytes
  double net[kMaxReac][LD];                    // net stoichiometry of reaction r
  double tb[kMaxReac][LD];                     // third-body efficiencies
  double low[NS][7], high[NS][7], imw3[LD];    // imw3: 1e-3 / W (mol/cm^3 of kg/m^3)
  double A[kMaxReac], b[kMaxReac], Ea[kMaxReac], A2[kMaxReac], b2[kMaxReac], Ea2[kMaxReac];
  double troe_alpha[kMaxReac], troe_it3[kMaxReac], troe_it1[kMaxReac], troe_t2[kMaxReac];
  double ent_f[kMaxReac * kMaxInvolved], ent_b[kMaxReac * kMaxInvolved];
  int type[kMaxReac], order[kMaxReac];
  uint2 mol[kMaxReac];  // positions of the reactants and products, a byte each; NS stands for none, kLongSide below
  unsigned char deal[kMaxReac];
  unsigned char ent_r[kMaxReac * kMaxInvolved];
};

// A group's own shared memory.  Its size is 6 words past a multiple of 32, so
// that the ten groups of a warp, which read the same entry or three adjacent
// ones, hit different banks.
template <int NS>
struct GroupMem {
  double w[NS];
  double c[NS + 1], g[NS + 1];        // entry NS: no molecule (c 1, g 0)
  double q1[kMaxReac], q2[kMaxReac];  // rates of progress
  static constexpr int kUsed = 3 * NS + 2 + 2 * kMaxReac;
  double pad[((3 - kUsed) % 16 + 16) % 16];
};

template <int NS>
__device__ __forceinline__ void load_group_tables(GroupTables<NS> &tb, const Mech &m, int tid, int nt) {
  const Kinetics &kn = m.kn;
  for (int e = tid; e < NS * 7; e += nt) {
    const int sp = kn.order_sp[e / 7];
    tb.low[e / 7][e % 7] = m.th.low[sp][e % 7];
    tb.high[e / 7][e % 7] = m.th.high[sp][e % 7];
  }
  for (int i = tid; i < NS; i += nt) tb.imw3[i] = m.th.imw[kn.order_sp[i]] * 1e-3;
  for (int r = tid; r < kMaxReac; r += nt) {
    tb.A[r] = kn.A[r]; tb.b[r] = kn.b[r]; tb.Ea[r] = kn.Ea[r];
    tb.A2[r] = kn.A2[r]; tb.b2[r] = kn.b2[r]; tb.Ea2[r] = kn.Ea2[r];
    tb.troe_alpha[r] = kn.troe_alpha[r]; tb.troe_it3[r] = 1.0 / kn.troe_t3[r];
    tb.troe_it1[r] = 1.0 / kn.troe_t1[r]; tb.troe_t2[r] = kn.troe_t2[r];
    tb.type[r] = kn.type[r]; tb.order[r] = kn.order[r];
    tb.deal[r] = kn.deal[r];
    unsigned f = kn.long_side[r] ? kLongSide : 0u, b = 0;
    for (int k = 0; k < kMaxMol; ++k) {
      f |= (k < kn.n_f[r] ? (unsigned)kn.lf[r][k] : (unsigned)NS) << 8 * k;
      b |= (k < kn.n_b[r] ? (unsigned)kn.lb[r][k] : (unsigned)NS) << 8 * k;
    }
    tb.mol[r] = make_uint2(f, b);
    for (int i = 0; i < NS; ++i) {
      const int sp = kn.order_sp[i];
      tb.net[r][i] = (double)kn.stb[r][sp] - (double)kn.stf[r][sp];
      tb.tb[r][i] = kn.tb[r][sp];
    }
  }
  for (int e = tid; e < kn.n_ent; e += nt) {
    tb.ent_f[e] = kn.ent_f[e]; tb.ent_b[e] = kn.ent_b[e];
    tb.ent_r[e] = kn.ent_r[e];
  }
}

// A lane's place: lane j of its group, whose first lane is base; its slot k is
// position k GL + j.  Lanes beyond the last group own nothing (own = false):
// they read the last group's memory and write none.
template <int NS, int GL>
struct Lane {
  static constexpr int SPL = NS / GL;
  int j, base;
  bool own;
  int sp[SPL];                // species of the lane's slots
  double mw[SPL], R[SPL];
  double t_low[SPL], t_mid[SPL], t_high[SPL];
  int ent[SPL], ent_end[SPL];
  __device__ Lane(const Mech &m, int lane) {
    constexpr int per = 32 / GL;
    own = lane < per * GL;
    const int grp = own ? lane / GL : per - 1;
    base = grp * GL;
    j = (lane - base) % GL;
#pragma unroll
    for (int k = 0; k < SPL; ++k) {
      const int i = k * GL + j;
      sp[k] = m.kn.order_sp[i];
      mw[k] = m.th.mw[sp[k]]; R[k] = m.th.gas_const[sp[k]];
      t_low[k] = m.th.t_low[sp[k]]; t_mid[k] = m.th.t_mid[sp[k]]; t_high[k] = m.th.t_high[sp[k]];
      ent[k] = m.kn.ent_start[i];
      ent_end[k] = m.kn.ent_start[i + 1];
    }
  }
  // Sum over the group, in the same order in every lane.
  __device__ double sum(double v) const {
    double a = __shfl_sync(0xffffffffu, v, base);
#pragma unroll
    for (int k = 1; k < GL; ++k) a = __dadd_rn(a, __shfl_sync(0xffffffffu, v, base + k));
    return a;
  }
  __device__ double min(double v) const {
    double a = v;
#pragma unroll
    for (int k = 0; k < GL; ++k) a = fmin(a, __shfl_sync(0xffffffffu, v, base + k));
    return a;
  }
};

// State of a node across its substeps: the lane's species, the rest the same
// in all lanes of the group.
template <int SPL>
struct GroupState {
  double q[5], T, pres, iJac, ts;  // ts: reaction time scale
  double rY[SPL], Y[SPL];
  int64_t iq;  // the node in Cn
};

template <int NS, int GL>
__device__ __forceinline__ void load_group(const Zone &z, int64_t id, int64_t iq, const Lane<NS, GL> &me,
                                           GroupState<NS / GL> &s) {
  const int64_t sz = z.d.plane(z.d.ngg);
#pragma unroll
  for (int k = 0; k < 5; ++k) s.q[k] = z.cv[id + k * sz];
#pragma unroll
  for (int k = 0; k < NS / GL; ++k) {
    s.rY[k] = z.cv[id + (5 + me.sp[k]) * sz];
    s.Y[k] = z.sv[id + me.sp[k] * sz];
  }
  s.T = z.bv[id + 5 * sz];
  s.pres = z.bv[id + 4 * sz];
  s.iJac = 1.0 / z.jac[id];
  s.ts = z.reaction_timeScale[id];
  s.iq = iq;
}

template <int NS, int GL>
__device__ __forceinline__ void store_group(const Zone &z, int n_scalar, int64_t id, const Lane<NS, GL> &me,
                                            const GroupState<NS / GL> &s) {
  const int64_t sz = z.d.plane(z.d.ngg);
#pragma unroll
  for (int k = 0; k < NS / GL; ++k) {
    z.cv[id + (5 + me.sp[k]) * sz] = s.rY[k];
    z.sv[id + me.sp[k] * sz] = s.Y[k];
  }
  const double rho_inv = 1.0 / s.q[0];
  if (me.j == 0) {
#pragma unroll
    for (int k = 0; k < 5; ++k) z.cv[id + k * sz] = s.q[k];
    z.reaction_timeScale[id] = s.ts;
  } else if (me.j == 1) {
    z.bv[id] = s.q[0];
#pragma unroll
    for (int k = 1; k < 4; ++k) z.bv[id + k * sz] = s.q[k] * rho_inv;
    z.bv[id + 4 * sz] = s.pres;
    z.bv[id + 5 * sz] = s.T;
  } else if (me.j == 2) {
    for (int k = NS; k < n_scalar; ++k) z.sv[id + k * sz] = z.cv[id + (5 + k) * sz] * rho_inv;
  }
}

// Forward and backward rate of progress of reaction r at the group's state.
// LONG: the mechanism has a reaction with a long side, whose factors are taken
// species by species (a variant of its own: the branch costs other mechanisms
// 3 %).  65536 H2/air reactors, one reaction doubled to four molecules a side:
// 3.43 ms, against 22.4 on the runtime-count kernel.
template <int NS, bool LONG>
__device__ __forceinline__ void group_rate(const Kinetics &kn, const GroupTables<NS> &tb, const GroupMem<NS> &S,
                                           int r, double t, double lnT, double iT, double temp_t, double itemp_t,
                                           double &q1, double &q2) {
  const int type = tb.type[r];
  double kf = tb.A[r] * exp(fma(tb.b[r], lnT, -tb.Ea[r] * iT));
  if (type == 3) kf = fma(tb.A2[r], exp(fma(tb.b2[r], lnT, -tb.Ea2[r] * iT)), kf);
  if (type > 3) {
    double cc = 0;
#pragma unroll
    for (int l = 0; l < NS; ++l) cc = fma(S.c[l], tb.tb[r][l], cc);
    if (type == 4) {
      kf *= cc;
    } else {
      const double kf_low = tb.A2[r] * exp(fma(tb.b2[r], lnT, -tb.Ea2[r] * iT));
      const double kf_high = kf;
      if (kf_high < 1e-25 && kf_low < 1e-25) {
        kf = 0;
      } else {
        const double pr = kf_low * cc / kf_high;  // kf_high can be subnormal
        kf = kf_high * pr * rcp_nr(1.0 + pr);
        if (type > 5) {
          const double al = tb.troe_alpha[r];
          double f_cent = fma(1 - al, exp(-t * tb.troe_it3[r]), al * exp(-t * tb.troe_it1[r]));
          if (type == 7) f_cent += exp(-tb.troe_t2[r] * iT);
          // ln F = ln Fc / (1 + (x / n)^2), with one reciprocal, of n^2 + x^2: n passes zero
          constexpr double per_ln10 = 0.43429448190325182765;
          const double lnFc = log(f_cent), logFc = lnFc * per_ln10;
          const double x = fma(log(pr), per_ln10, fma(-0.67, logFc, -0.4));
          const double n = fma(-0.14, x, fma(-1.27, logFc, 0.75)), nn = n * n;
          kf *= exp(lnFc * nn * rcp_nr(fma(x, x, nn)));
        }
      }
    }
  }
  const uint2 mol = tb.mol[r];
  double dg = 0, af = 1, ab = 1;  // dg: g of the products less that of the reactants
  if (LONG && (mol.x & kLongSide)) {
    for (int q = 0; q < kn.n_inv[r]; ++q) {
      const int i = kn.inv_pos[r][q], f = kn.inv_f[r][q], b = kn.inv_b[r][q];
      dg = fma(S.g[i], (double)(b - f), dg);
      for (int k = 0; k < f; ++k) af *= S.c[i];
      for (int k = 0; k < b; ++k) ab *= S.c[i];
    }
  } else {
#pragma unroll
    for (int k = 0; k < kMaxMol; ++k) {
      const int i = mol.x >> 8 * k & 255u, j = mol.y >> 8 * k & 255u;
      dg += S.g[j] - S.g[i];
      af *= S.c[i];
      ab *= S.c[j];
    }
  }
  q1 = kf * af;
  // kb = kf / Kc, Kc = (p_atm / R_u T)^order exp(-dg)
  q2 = 0;
  if (type != 0) {
    q2 = kf * exp(dg) * ab;
    const int o = tb.order[r];
    for (int k = 0; k < (o < 0 ? -o : o); ++k) q2 *= o < 0 ? temp_t : itemp_t;
  }
}

// Solves the group's system by Gauss-Jordan elimination with partial pivoting:
// a[k][m] is row m of the lane's column k GL + j, x the right-hand side, the
// same in all lanes; y receives the lane's unknowns.  The owner of a column
// picks its pivot and passes its multipliers on.  Rows are swapped, by the whole
// warp, only if some group's pivot is off the diagonal.  Swapping only where the
// pivot is four times the diagonal is 0.6 % faster on 2^20 reactors (11 % at
// substeps of 0.1 us, 15 % at 1 us), but its error on burning H2/O2/Ar at substeps
// of 10 us and more is up to twice that of an LU factorisation with partial
// pivoting; with partial pivoting here it is below that one's.
template <int NS, int GL>
__device__ __forceinline__ void group_solve(double (&a)[NS / GL][NS], double (&x)[NS], const Lane<NS, GL> &me,
                                            double (&y)[NS / GL]) {
  constexpr int SPL = NS / GL;
  double inv[SPL];
#pragma unroll
  for (int i = 0; i < NS; ++i) {
    const int k = i / GL, src = me.base + i % GL;
    int p = i;
    double best = fabs(a[k][i]);
#pragma unroll
    for (int m = i + 1; m < NS; ++m)
      if (fabs(a[k][m]) > best) {
        best = fabs(a[k][m]);
        p = m;
      }
    p = __shfl_sync(0xffffffffu, p, src);
    if (__any_sync(0xffffffffu, p != i)) {
#pragma unroll
      for (int m = i + 1; m < NS; ++m) {
        const bool sw = p == m;
#pragma unroll
        for (int c = k; c < SPL; ++c) {
          const double u = a[c][i], v = a[c][m];
          a[c][i] = sw ? v : u;
          a[c][m] = sw ? u : v;
        }
        const double u = x[i], v = x[m];
        x[i] = sw ? v : u;
        x[m] = sw ? u : v;
      }
    }
    const double r = rcp_nr(a[k][i]);
    if (me.j == i % GL) inv[k] = r;
#pragma unroll
    for (int m = 0; m < NS; ++m) {
      if (m == i) continue;
      const double f = __shfl_sync(0xffffffffu, a[k][m] * r, src);
      // the columns up to i are done: their entries are no longer read
#pragma unroll
      for (int c = (i % GL == GL - 1 ? k + 1 : k); c < SPL; ++c) a[c][m] = fma(-f, a[c][i], a[c][m]);
      x[m] = fma(-f, x[i], x[m]);
    }
  }
#pragma unroll
  for (int k = 0; k < SPL; ++k) {
    double v = x[k * GL];
#pragma unroll
    for (int j = 1; j < GL; ++j)
      if (me.j == j) v = x[k * GL + j];
    y[k] = v * inv[k];
  }
}

// One substep of wu_zeroDReaction (methods 0 and 1) of a warp's groups, all
// lanes of the warp together; `on`: the lane's group has a node and a step to
// take (the others compute along and keep their state).
template <int NS, int GL, bool LONG>
__device__ __forceinline__ bool group_substep(const Zone &z, const Kinetics &kn, const GroupTables<NS> &tb,
                                              GroupMem<NS> &S, const Lane<NS, GL> &me, int method, double dt, bool on,
                                              GroupState<NS / GL> &s) {
  constexpr int SPL = NS / GL;
  const double t = s.T, lnT = log(t), iT = rcp_nr(t);
#pragma unroll
  for (int k = 0; k < SPL; ++k) {
    const int i = k * GL + me.j;
    const double g = gibbs_one(tb.low[i], tb.high[i], me.t_low[k], me.t_mid[k], me.t_high[k], t, lnT, iT);
    if (me.own) {
      S.c[i] = s.rY[k] * tb.imw3[i];
      S.g[i] = g;
    }
  }
  __syncwarp();
  constexpr double temp_p = 101325.0 / kRu * 1e-3;  // mol K / cm^3
  const double temp_t = temp_p * iT, itemp_t = t * (1.0 / temp_p);
  if (me.own)
    for (int k = me.j; k < kn.n_reac; k += GL) {
      const int r = tb.deal[k];
      double q1, q2;
      group_rate<NS, LONG>(kn, tb, S, r, t, lnT, iT, temp_t, itemp_t, q1, q2);
      S.q1[r] = q1;
      S.q2[r] = q2;
    }
  __syncwarp();
  // the lane's species: creation, destruction and its columns of the matrix
  double a[SPL][NS], y[SPL], tsl = 1e6;
#pragma unroll
  for (int k = 0; k < SPL; ++k) {
    // minus the column's scale: dt 1e3 W_n / rhoY_n
    const double w = 1e+3 * me.mw[k], sn = s.rY[k] > 1e-25 ? -dt * w * rcp_nr(s.rY[k]) : 0.0;
    double make = 0, use = 0;
#pragma unroll
    for (int m = 0; m < NS; ++m) a[k][m] = m == k * GL + me.j ? 1.0 : 0.0;
    for (int e = me.ent[k]; e < me.ent_end[k]; ++e) {
      const int r = tb.ent_r[e];
      const double f = tb.ent_f[e], b = tb.ent_b[e], q1 = S.q1[r], q2 = S.q2[r];
      make = fma(q2, f, fma(q1, b, make));
      use = fma(q1, f, fma(q2, b, use));
      if (method == 1) {
        const double d = sn * fma(f, q1, -b * q2);
#pragma unroll
        for (int m = 0; m < NS; ++m) a[k][m] = fma(tb.net[r][m], d, a[k][m]);
      }
    }
    y[k] = 1e+3 * (make - use);
    use *= w;
    if (s.rY[k] > 1e-25 && fabs(use) > 1e-25) tsl = fmin(tsl, fabs(s.rY[k] * rcp_nr(use)));
  }
  if (method == 1) {
    if (me.own) {
#pragma unroll
      for (int k = 0; k < SPL; ++k) S.w[k * GL + me.j] = y[k];
    }
    __syncwarp();
    double x[NS];
#pragma unroll
    for (int m = 0; m < NS; ++m) x[m] = S.w[m];
    group_solve<NS, GL>(a, x, me, y);
  }
  double q[5], cnY[SPL];
#pragma unroll
  for (int k = 0; k < SPL; ++k) cnY[k] = 0;
#pragma unroll
  for (int k = 0; k < 5; ++k) q[k] = s.q[k];
  if (z.Cn) {
    const int64_t szq = z.d.plane(0);
#pragma unroll
    for (int k = 0; k < 5; ++k) q[k] = fma(z.Cn[s.iq + k * szq], dt * s.iJac, q[k]);
#pragma unroll
    for (int k = 0; k < SPL; ++k) cnY[k] = z.Cn[s.iq + (5 + me.sp[k]) * szq] * s.iJac;
  }
  double nY[SPL], part = 0;
#pragma unroll
  for (int k = 0; k < SPL; ++k) {
    nY[k] = fma(fma(y[k], me.mw[k], cnY[k]), dt, s.rY[k]);
    if (nY[k] < 0) nY[k] = 0;
    part = __dadd_rn(part, nY[k]);
  }
  const double sum = rcp_nr(me.sum(part)), ts = me.min(tsl);
  const double rho = q[0], rho_inv = rcp_nr(rho), ratio = rho * sum;
  const double u = q[1] * rho_inv, v = q[2] * rho_inv, w = q[3] * rho_inv;
  double Y[SPL];
  part = 0;
#pragma unroll
  for (int k = 0; k < SPL; ++k) {
    Y[k] = nY[k] * sum;
    nY[k] *= ratio;
    part = fma(Y[k], me.R[k], part);
  }
  // T by Newton's iteration from the energy (temperature_newton)
  const double gas_const = me.sum(part);
  const double e = fma(-0.5, fma(u, u, fma(v, v, w * w)), q[4] * rho_inv);
  double T = t, err = 1;
  for (int iter = 0; iter < 1000; ++iter) {
    const bool go = on && err > 1e-5;
    if (!__any_sync(0xffffffffu, go)) break;
    double h = 0, cp = 0;
#pragma unroll
    for (int k = 0; k < SPL; ++k) {
      const int i = k * GL + me.j;
      const double tt = fmin(fmax(T, me.t_low[k]), me.t_high[k]);
      const double *c = T < me.t_mid[k] ? tb.low[i] : tb.high[i];
      const double p0 = fma(tt, fma(tt, fma(tt, fma(tt, c[4], c[3]), c[2]), c[1]), c[0]);
      const double p1 =
          fma(tt, fma(tt, fma(tt, fma(tt, 0.2 * c[4], 0.25 * c[3]), (1.0 / 3) * c[2]), 0.5 * c[1]), c[0]);
      const double ry = me.R[k] * Y[k];
      cp = fma(ry, p0, cp);
      h = fma(ry, fma(p0, T - tt, fma(tt, p1, c[5])), h);
    }
    h = me.sum(h);
    cp = me.sum(cp);
    if (go) {
      const double t1 = fma(e - fma(-gas_const, T, h), rcp_nr(cp - gas_const), T);
      err = fabs(fma(-t1, rcp_nr(T), 1.0));
      T = t1;
    }
  }
  if (on) {
#pragma unroll
    for (int k = 0; k < 5; ++k) s.q[k] = q[k];
#pragma unroll
    for (int k = 0; k < SPL; ++k) {
      s.rY[k] = nY[k];
      s.Y[k] = Y[k];
    }
    s.ts = ts;
    s.T = T;
    s.pres = rho * T * gas_const;
  }
  return !on || err <= 1e-5;
}

}  // namespace cfk
