// Fused characteristic WENO flux + flux difference for a reacting mixture
// (NS species, thermally perfect, NASA-7 thermo).
//
// Restates compute_convective_term_weno_{x,y,z} with the mixture branch of
// the characteristic reconstruction (reference src/WENO.cu:1096-1469) and
// compute_derivative_{x,y,z} (:1544, 2219, 2885) in the stage / faces / diff
// structure of weno_air.cu:
//   stage — Q[5], the species densities rho*Y_k, the face-normal flux
//           G = (rho U, rho u U + p k_x, ..., (rho E + p) U), U, p, J and the
//           spectral radius |U| + c|grad k| (c from the acoustic-speed array)
//           of every stencil point, in shared memory;
//   faces — Roe average of u, v, w, Y_k and T, mixture gamma and c from the
//           NASA-7 cp at the averaged temperature, the five characteristic
//           fields with the species coupling terms (beta_k = (gamma R_k T -
//           (gamma-1) h_k) / c^2), NS species fields (rho Y_k - Y~_k rho),
//           LLF split, WENO5-JS / WENO7-Z, back projection;
//   diff  — dq -= F(n+1/2) - F(n-1/2) for all 5 + NS variables.
// The mixture tables are a __grid_constant__ parameter (constant bank).
#include "cfk_common.cuh"
#include "chem_fast.cuh"
#include "thermo.cuh"
#include "weno.cuh"

namespace cfk {

namespace {

// staged values per point: J/2 times Q0..4, the face-normal flux G0..4 and
// rhoY[NS]; U, p, 2/J, lambda
template <int NS>
struct MixVals {
  static constexpr int U = 10, P = 11, IJ = 12, LAM = 13, Y0 = 14, N = 14 + NS;
};

// Tile shapes of a sweep (nodes per column TN x columns C); VAR is chosen per
// direction by the tile autotuner.  Every shape has 128 faces, one a thread,
// and at 128 registers and 40 to 58 KB four CTAs fit an SM (three of WENO7's
// y/z 7x16, which has 58 KB):
// FP64-bound.  Tiles of 256 faces in two CTAs an SM recompute less halo but put
// half as many independent barriers in flight and leave a longer last wave:
// 2048 x 512 WENO5 557 -> 510 us, 90 x 70 x 60 WENO7 478 -> 413 us, a 97 x 49 x
// 33 Wu step 1956 -> 1896 us, and bitwise the same.  With all 14 fields unrolled
// a face took 226 registers, one CTA of 256 an SM, and its code did not fit the
// instruction cache (2048 x 512: 1786 us, 90 x 70 x 60: 1561 us).
template <int DIR, int VAR>
struct MixShape {
  static constexpr int TN = DIR == 0 ? (VAR == 0 ? 31 : VAR == 1 ? 63 : 15) : (VAR == 0 ? 15 : VAR == 1 ? 7 : 31);
  static constexpr int C = DIR == 0 ? (VAR == 0 ? 4 : VAR == 1 ? 2 : 8) : (VAR == 0 ? 8 : VAR == 1 ? 16 : 4);
};

template <int DIR, int ORD, int NS, int VAR = 0>
struct MixTile {
  static constexpr int R = ORD == 7 ? 3 : 2;
  static constexpr int NPF = 2 * R + 2;
  static constexpr int TN = MixShape<DIR, VAR>::TN;
  static constexpr int C = MixShape<DIR, VAR>::C;
  static constexpr int NF = TN + 1;
  static constexpr int NPT = TN + 2 * R + 2;
  static constexpr int NT = 128;
  static constexpr int NQ = MixVals<NS>::N;
  static constexpr int NV = 5 + NS;
  __device__ static int spt(int q, int c, int t) {
    return DIR == 0 ? (q * C + c) * NPT + t : (q * NPT + t) * C + c;
  }
  __device__ static int sfl(int v, int c, int t) {
    return DIR == 0 ? (v * C + c) * NF + t : (v * NF + t) * C + c;
  }
  static constexpr size_t smem_bytes() { return sizeof(double) * (size_t)(NQ * C * NPT + NV * C * NF); }
};

// Positive-preserving limiter of the species face fluxes (reference
// src/WENO.cu:1471-1540; the characteristic scheme has it in the x sweep
// only).  For each species whose one-sided updates alpha/2 J rhoY -/+ dt f
// would go negative, the face flux is blended towards the first-order flux
// f1 = 1/2 (fp + U_L J_L rhoY_L) + 1/2 (fm - U_R J_R rhoY_R) with
// fp/m = 1/2 J (U +/- c|grad k|) rhoY, theta in [0, 1].  Out of line: the
// branch is rare and must not add registers to the face loop.  s/sf point at
// the staged values and face fluxes of this tile; the species face fluxes
// are updated in shared memory.
template <int ORD, int NS, int VAR>
__device__ __noinline__ void pp_limit_x(const double *s, double *sf, int c, int t, const Zone &z, int64_t idl,
                                        double dt, double alpha_dim, double rho_ref) {
  using T = MixTile<0, ORD, NS, VAR>;
  using V = MixVals<NS>;
  const int pc = t + T::R;
  const double il = s[T::spt(V::IJ, c, pc)], ir = s[T::spt(V::IJ, c, pc + 1)];  // 2 / J: back to rho Y
  const double jac_l = 2 / il, jac_r = 2 / ir;
  const double alphaL = 0.5 * alpha_dim * jac_l, alphaR = 0.5 * alpha_dim * jac_r;
  int start_l = -1;
  for (int l = 0; l < NS; ++l) {
    const double fl = sf[T::sfl(5 + l, c, t)];
    const double up = alphaL * (il * s[T::spt(V::Y0 + l, c, pc)]) - dt * fl;
    const double um = alphaR * (ir * s[T::spt(V::Y0 + l, c, pc + 1)]) + dt * fl;
    if (up < 0 || um < 0) { start_l = l; break; }
  }
  if (start_l < 0) return;
  // c|grad k| of the two nodes, as staged by the reference (F[5])
  const int64_t sz = z.d.plane(z.d.ngg);
  double cg[2];
  for (int n = 0; n < 2; ++n) {
    const int64_t id = idl + n;
    const double m0 = z.metric[id], m1 = z.metric[id + sz], m2 = z.metric[id + 2 * sz];
    cg[n] = sqrt(m0 * m0 + m1 * m1 + m2 * m2) * z.acoustic_speed[id];
  }
  const double UkL = s[T::spt(V::U, c, pc)], UkR = s[T::spt(V::U, c, pc + 1)];
  const double U1 = UkL * jac_l, U2 = UkR * jac_r;
  for (int l = start_l; l < NS; ++l) {
    const double fc = sf[T::sfl(5 + l, c, t)];
    double f1 = 0, theta_p = 1.0, theta_m = 1.0;
    bool f1_computed = false;
    const double rhoYL = il * s[T::spt(V::Y0 + l, c, pc)], rhoYR = ir * s[T::spt(V::Y0 + l, c, pc + 1)];
    const double fp = 0.5 * jac_l * (UkL + cg[0]) * rhoYL;
    const double fm = 0.5 * jac_r * (UkR - cg[1]) * rhoYR;
    const double up = alphaL * rhoYL - dt * fc;
    if (up < 0) {
      f1 = 0.5 * (fp + U1 * rhoYL) + 0.5 * (fm - U2 * rhoYR);
      f1_computed = true;
      const double up_lf = alphaL * rhoYL - dt * f1;
      if (abs(up - up_lf) > 1e-20 * rho_ref) theta_p = min(max((0 - up_lf) / (up - up_lf), 0.0), 1.0);
    }
    const double um = alphaR * rhoYR + dt * fc;
    if (um < 0) {
      if (!f1_computed) f1 = 0.5 * (fp + U1 * rhoYL) + 0.5 * (fm - U2 * rhoYR);
      const double um_lf = alphaR * rhoYR + dt * f1;
      if (abs(um - um_lf) > 1e-20 * rho_ref) theta_m = min(max((0 - um_lf) / (um - um_lf), 0.0), 1.0);
    }
    sf[T::sfl(5 + l, c, t)] = min(theta_p, theta_m) * (fc - f1) + f1;
  }
}

// Settings of the positive-preserving limiter: off unless `on`; the step's
// dt from the device (CFL runs) or the host (fixed dt); dt <= 0 selects the
// node's dt_local as the reference does.
struct PPArgs {
  int on;
  const double *dt_dev;
  double dt_host, alpha_dim, rho_ref;
};

}  // namespace

// HYB: hybrid UD/WENO scheme, the face switches on the shock sensor.
// VAR: tile shape (MixShape).
template <int DIR, int ORD, int NS, bool HYB, int VAR>
__global__ void __launch_bounds__(128, 4) weno_mix_flux_diff(Zone z, double eps_ref,
                                                             const __grid_constant__ Thermo thermo,
                                                             const double *sensor, double threshold, PPArgs pp) {
  using T = MixTile<DIR, ORD, NS, VAR>;
  using V = MixVals<NS>;
  constexpr int R = T::R, NPF = T::NPF, TN = T::TN, C = T::C, NF = T::NF, NPT = T::NPT;
  static_assert(NF * C % T::NT == 0, "every lane of a warp comes to the __syncwarps of the face loop in every round");
  const Thermo *th = &thermo;
  extern __shared__ double sm[];
  double *spts = sm;
  double *sflx = sm + T::NQ * C * NPT;

  const Dims d = z.d;
  const int g = d.ngg;
  const int64_t sz = d.plane(g), szq = d.plane(0);
  const int m = d.ext(DIR);
  int n0, cbase, cfix;
  if (DIR == 0) { n0 = blockIdx.x * TN; cbase = blockIdx.y * C; cfix = blockIdx.z; }
  else { n0 = blockIdx.y * TN; cbase = blockIdx.x * C; cfix = blockIdx.z; }
  const int ncol_max = DIR == 0 ? d.my : d.mx;
  auto node_idx = [&](int g_, int c, int a) -> int64_t {
    const int cc = cbase + c;
    if (DIR == 0) return d.idx(g_, a, cc, cfix);
    if (DIR == 1) return d.idx(g_, cc, a, cfix);
    return d.idx(g_, cc, cfix, a);
  };
  auto split = [&](int item, int n_t, int &c, int &t) {
    if (DIR == 0) { c = item / n_t; t = item - c * n_t; }
    else { t = item / C; c = item - t * C; }
  };
  const int mmo = 3 * DIR;
  double dt_pp = 0;
  if (DIR == 0 && pp.on) dt_pp = pp.dt_dev ? *pp.dt_dev : pp.dt_host;

  // ---- stage ------------------------------------------------------------
  for (int item = threadIdx.x; item < NPT * C; item += T::NT) {
    int c, t;
    split(item, NPT, c, t);
    const int a = n0 - 1 - R + t;
    if (cbase + c >= ncol_max || a > m + R) continue;
    const int64_t id = node_idx(g, c, a);
    const double q0 = z.cv[id], q1 = z.cv[id + sz], q2 = z.cv[id + 2 * sz], q3 = z.cv[id + 3 * sz],
                 q4 = z.cv[id + 4 * sz];
    const double m0 = z.metric[id + mmo * sz], m1 = z.metric[id + (mmo + 1) * sz], m2 = z.metric[id + (mmo + 2) * sz];
    const double Uk = dot3(q1, m0, q2, m1, q3, m2) * rcp_nr(q0);
    const double pk = z.bv[id + 4 * sz], hj = 0.5 * z.jac[id], hp = hj * pk;
    const double h0 = hj * q0, h1 = hj * q1, h2 = hj * q2, h3 = hj * q3, h4 = hj * q4;
    double *s = spts;
    s[T::spt(0, c, t)] = h0;
    s[T::spt(1, c, t)] = h1;
    s[T::spt(2, c, t)] = h2;
    s[T::spt(3, c, t)] = h3;
    s[T::spt(4, c, t)] = h4;
    s[T::spt(5, c, t)] = h0 * Uk;
    s[T::spt(6, c, t)] = fma(h1, Uk, hp * m0);
    s[T::spt(7, c, t)] = fma(h2, Uk, hp * m1);
    s[T::spt(8, c, t)] = fma(h3, Uk, hp * m2);
    s[T::spt(9, c, t)] = __dadd_rn(h4, hp) * Uk;
    s[T::spt(V::U, c, t)] = Uk;
    s[T::spt(V::P, c, t)] = pk;
    s[T::spt(V::IJ, c, t)] = rcp_nr(hj);
    s[T::spt(V::LAM, c, t)] = fma(sqrt(dot3(m0, m0, m1, m1, m2, m2)), z.acoustic_speed[id], abs(Uk));
#pragma unroll
    for (int l = 0; l < NS; ++l) s[T::spt(V::Y0 + l, c, t)] = hj * z.cv[id + (5 + l) * sz];
  }
  __syncthreads();

  // ---- face fluxes ------------------------------------------------------
  for (int item = threadIdx.x; item < NF * C; item += T::NT) {
    int c, t;
    split(item, NF, c, t);
    const int f = n0 - 1 + t;
    const bool valid = cbase + c < ncol_max && f < m;
    const double *s = spts;
    const int pc = t + R;
    auto recon = [&](const double *vp, const double *vm, bool shock) -> double {
      if constexpr (ORD == 7) return shock ? weno7_z(vp, vm, eps_ref) : weno7_linear(vp, vm);
      else return shock ? weno5_js(vp, vm, eps_ref) : weno5_linear(vp, vm);
    };
    // face normal averaged with the (i+1) node, as the reference does
    const int64_t idf = valid ? node_idx(g, c, f) : 0;
    double kx = 0.5 * (z.metric[idf + mmo * sz] + z.metric[idf + 1 + mmo * sz]);
    double ky = 0.5 * (z.metric[idf + (mmo + 1) * sz] + z.metric[idf + 1 + (mmo + 1) * sz]);
    double kz = 0.5 * (z.metric[idf + (mmo + 2) * sz] + z.metric[idf + 1 + (mmo + 2) * sz]);
    const bool shock = !HYB || (valid && face_shocked(sensor, idf, d.stride(g, DIR), g, threshold));

    const double il = s[T::spt(V::IJ, c, pc)], ir = s[T::spt(V::IJ, c, pc + 1)];
    const double rho_l = s[T::spt(0, c, pc)] * il, rho_r = s[T::spt(0, c, pc + 1)] * ir;
    const double root = sqrt(rho_l * rho_r);
    const double rlc = rcp_nr(__dadd_rn(rho_l, root)), rrc = rcp_nr(__dadd_rn(root, rho_r));
    const double sl = rlc * il, sr = rrc * ir;  // weights of the scaled conserved variables
    const double um = dot2(sl, s[T::spt(1, c, pc)], sr, s[T::spt(1, c, pc + 1)]);
    const double vm = dot2(sl, s[T::spt(2, c, pc)], sr, s[T::spt(2, c, pc + 1)]);
    const double wm = dot2(sl, s[T::spt(3, c, pc)], sr, s[T::spt(3, c, pc + 1)]);
    auto yk = [&](int l) { return dot2(sl, s[T::spt(V::Y0 + l, c, pc)], sr, s[T::spt(V::Y0 + l, c, pc + 1)]); };
    const double pr = dot2(rlc, s[T::spt(V::P, c, pc)], rrc, s[T::spt(V::P, c, pc + 1)]);
    const double H = fma(sl, s[T::spt(4, c, pc)], fma(sr, s[T::spt(4, c, pc + 1)], pr));
    double rg = 0;
#pragma unroll
    for (int l = 0; l < NS; ++l) rg = fma(yk(l), th->gas_const[l], rg);
    const double T3 = pr * rcp_nr(rg);
    // h_l, then beta_l, wait in this face's species slots of the flux buffer;
    // the loops over the species stay loops: unrolled, the face code of all
    // fields overflows the instruction cache
    double cps = 0;
#pragma unroll 3
    for (int l = 0; l < NS; ++l) {
      double h, cp;
      enthalpy_cp_one(th, l, T3, h, cp);
      cps = fma(yk(l), cp, cps);
      sflx[T::sfl(5 + l, c, t)] = h;
    }
    const double gamma = cps / (cps - rg), gm1 = gamma - 1;
    const double c2 = gamma * pr, cm = sqrt(c2), ic2 = rcp_nr(c2);
#pragma unroll 3
    for (int l = 0; l < NS; ++l)
      sflx[T::sfl(5 + l, c, t)] = dot2(gamma * T3, th->gas_const[l], -gm1, sflx[T::sfl(5 + l, c, t)]) * ic2;

    double nrm = rsqrt(dot3(kx, kx, ky, ky, kz, kz));
    kx *= nrm; ky *= nrm; kz *= nrm;
    const double Uk_bar = dot3(kx, um, ky, vm, kz, wm);
    const double alpha = 0.5 * gm1 * dot3(um, um, vm, vm, wm, wm);
    double lam = 0;
#pragma unroll
    for (int q = 0; q < NPF; ++q) lam = max(lam, s[T::spt(V::LAM, c, t + q)]);

    // the fields in pairs that share the loads of the staged points, as in
    // weno_air.cu; __syncwarp keeps the loads of a later block below the
    // arithmetic of an earlier one
    double f1, f2, f3, f4;
    {  // shear fields: n and q = k x n complete the basis; no energy or species term
      double A1 = 0, A2 = 0, A3 = 0;
      if (abs(kx) > 0.8) { A1 = -kz; A3 = kx; }
      else { A2 = kz; A3 = -ky; }
      nrm = rsqrt(dot3(A1, A1, A2, A2, A3, A3));
      A1 *= nrm; A2 *= nrm; A3 *= nrm;
      const double B1 = dot2(ky, A3, -kz, A2), B2 = dot2(kz, A1, -kx, A3), B3 = dot2(kx, A2, -ky, A1);
      const double A0 = -dot3(A1, um, A2, vm, A3, wm), B0 = -dot3(B1, um, B2, vm, B3, wm);
      __syncwarp();
      double va[NPF - 1], wa[NPF - 1], vb[NPF - 1], wb[NPF - 1];
#pragma unroll
      for (int q = 0; q < NPF; ++q) {
        const int tq = t + q;
        const double g0 = s[T::spt(5, c, tq)], g1 = s[T::spt(6, c, tq)], g2 = s[T::spt(7, c, tq)],
                     g3 = s[T::spt(8, c, tq)];
        const double q0 = s[T::spt(0, c, tq)], q1 = s[T::spt(1, c, tq)], q2 = s[T::spt(2, c, tq)],
                     q3 = s[T::spt(3, c, tq)];
        const double Fa = dot4p(A1, g1, A2, g2, A3, g3, A0, g0, 0.0), Fb = dot4p(B1, g1, B2, g2, B3, g3, B0, g0, 0.0);
        const double Qa = dot4p(A1, q1, A2, q2, A3, q3, A0, q0, 0.0), Qb = dot4p(B1, q1, B2, q2, B3, q3, B0, q0, 0.0);
        if (q < NPF - 1) { va[q] = fma(lam, Qa, Fa); vb[q] = fma(lam, Qb, Fb); }
        if (q > 0) { wa[q - 1] = fma(-lam, Qa, Fa); wb[q - 1] = fma(-lam, Qb, Fb); }
      }
      const double ca = recon(va, wa, shock), cb = recon(vb, wb, shock);
      f1 = dot2(A1, ca, B1, cb);
      f2 = dot2(A2, ca, B2, cb);
      f3 = dot2(A3, ca, B3, cb);
      f4 = -dot2(A0, ca, B0, cb);
    }
    __syncwarp();
    double sb[NPF];  // sum of beta_k rho Y_k at the stencil points; their flux is U times it
    {
      double beta[NS];
#pragma unroll
      for (int l = 0; l < NS; ++l) beta[l] = sflx[T::sfl(5 + l, c, t)];
#pragma unroll
      for (int q = 0; q < NPF; ++q) {
        sb[q] = 0;
#pragma unroll
        for (int l = 0; l < NS; ++l) sb[q] = fma(beta[l], s[T::spt(V::Y0 + l, c, t + q)], sb[q]);
      }
    }
    double f04, f034;
    {  // acoustic fields
      const double h = 0.5 * ic2, E = gm1 * h, kc = cm * h, a0 = alpha * h;
      const double A0 = fma(Uk_bar, kc, a0), B0 = fma(-Uk_bar, kc, a0);
      const double A1 = -dot2(E, um, kx, kc), A2 = -dot2(E, vm, ky, kc), A3 = -dot2(E, wm, kz, kc);
      const double B1 = dot2(kx, kc, -E, um), B2 = dot2(ky, kc, -E, vm), B3 = dot2(kz, kc, -E, wm);
      __syncwarp();
      double va[NPF - 1], wa[NPF - 1], vb[NPF - 1], wb[NPF - 1];
#pragma unroll
      for (int q = 0; q < NPF; ++q) {
        const int tq = t + q;
        const double hs = 0.5 * sb[q];
        const double g0 = s[T::spt(5, c, tq)], g1 = s[T::spt(6, c, tq)], g2 = s[T::spt(7, c, tq)],
                     g3 = s[T::spt(8, c, tq)], eg = fma(E, s[T::spt(9, c, tq)], s[T::spt(V::U, c, tq)] * hs);
        const double q0 = s[T::spt(0, c, tq)], q1 = s[T::spt(1, c, tq)], q2 = s[T::spt(2, c, tq)],
                     q3 = s[T::spt(3, c, tq)], eq = fma(E, s[T::spt(4, c, tq)], hs);
        const double Fa = dot4p(A0, g0, A1, g1, A2, g2, A3, g3, eg);
        const double Fb = dot4p(B0, g0, B1, g1, B2, g2, B3, g3, eg);
        const double Qa = dot4p(A0, q0, A1, q1, A2, q2, A3, q3, eq);
        const double Qb = dot4p(B0, q0, B1, q1, B2, q2, B3, q3, eq);
        if (q < NPF - 1) { va[q] = fma(lam, Qa, Fa); vb[q] = fma(lam, Qb, Fb); }
        if (q > 0) { wa[q - 1] = fma(-lam, Qa, Fa); wb[q - 1] = fma(-lam, Qb, Fb); }
      }
      const double ca = recon(va, wa, shock), cb = recon(vb, wb, shock);
      f04 = cm * (ca - cb);
      f034 = ca + cb;
    }
    {  // entropy field
      const double L4 = -gm1 * ic2, L0 = fma(-alpha, ic2, 1.0), L1 = -L4 * um, L2 = -L4 * vm, L3 = -L4 * wm;
      __syncwarp();
      double va[NPF - 1], wa[NPF - 1];
#pragma unroll
      for (int q = 0; q < NPF; ++q) {
        const int tq = t + q;
        const double F = dot4p(L0, s[T::spt(5, c, tq)], L1, s[T::spt(6, c, tq)], L2, s[T::spt(7, c, tq)], L3,
                               s[T::spt(8, c, tq)], dot2(L4, s[T::spt(9, c, tq)], -s[T::spt(V::U, c, tq)], sb[q]));
        const double Q = dot4p(L0, s[T::spt(0, c, tq)], L1, s[T::spt(1, c, tq)], L2, s[T::spt(2, c, tq)], L3,
                               s[T::spt(3, c, tq)], fma(L4, s[T::spt(4, c, tq)], -sb[q]));
        if (q < NPF - 1) va[q] = fma(lam, Q, F);
        if (q > 0) wa[q - 1] = fma(-lam, Q, F);
      }
      const double c3 = recon(va, wa, shock);
      f034 += c3;
      f4 = fma(-c2 / gm1, c3, f4);
    }
    if (valid) {
      sflx[T::sfl(0, c, t)] = f034;
      sflx[T::sfl(1, c, t)] = fma(um, f034, fma(-kx, f04, f1));
      sflx[T::sfl(2, c, t)] = fma(vm, f034, fma(-ky, f04, f2));
      sflx[T::sfl(3, c, t)] = fma(wm, f034, fma(-kz, f04, f3));
    }
    f4 = fma(H, f034, fma(-Uk_bar, f04, f4));
    // species fields rho Y_k - Y~_k rho: their fluxes are U times them
    __syncwarp();
    double bsum = 0;
    {
      double q0[NPF], up[NPF], dn[NPF];
#pragma unroll
      for (int q = 0; q < NPF; ++q) {
        const double U = s[T::spt(V::U, c, t + q)];
        q0[q] = s[T::spt(0, c, t + q)];
        up[q] = U + lam;
        dn[q] = U - lam;
      }
#pragma unroll 1
      for (int l = 0; l < NS; ++l) {
        const double y = yk(l);
        double va[NPF - 1], wa[NPF - 1];
#pragma unroll
        for (int q = 0; q < NPF; ++q) {
          const double w = fma(-y, q0[q], s[T::spt(V::Y0 + l, c, t + q)]);
          if (q < NPF - 1) va[q] = up[q] * w;
          if (q > 0) wa[q - 1] = dn[q] * w;
        }
        const double cs = recon(va, wa, shock);
        bsum = fma(sflx[T::sfl(5 + l, c, t)], cs, bsum);
        sflx[T::sfl(5 + l, c, t)] = fma(y, f034, cs);
      }
    }
    if (!valid) continue;
    sflx[T::sfl(4, c, t)] = fma(-bsum, c2 / gm1, f4);
    if constexpr (DIR == 0) {
      if (pp.on) {
        const double dt = dt_pp > 0 ? dt_pp : z.dt_local[node_idx(0, c, f < 0 ? 0 : f)];
        pp_limit_x<ORD, NS, VAR>(s, sflx, c, t, z, idf, dt, pp.alpha_dim, pp.rho_ref);
      }
    }
  }
  __syncthreads();

  // ---- flux difference into dq -----------------------------------------
  for (int item = threadIdx.x; item < TN * C; item += T::NT) {
    int c, t;
    split(item, TN, c, t);
    const int a = n0 + t;
    if (cbase + c >= ncol_max || a > m - 1) continue;
    const int64_t iq = node_idx(0, c, a);
#pragma unroll
    for (int v = 0; v < T::NV; ++v) red_add(z.dq + iq + v * szq, sflx[T::sfl(v, c, t)] - sflx[T::sfl(v, c, t + 1)]);
  }
}

namespace {

template <int DIR, int ORD, int VAR>
cudaError_t launch_mix_var(const Zone &z, double eps_ref, const Thermo &th, const double *sensor, double threshold,
                           const PPArgs &pp, cudaStream_t st) {
  using T = MixTile<DIR, ORD, kMaxSpec, VAR>;
  const Dims &d = z.d;
  dim3 grid;
  if (DIR == 0) grid = dim3((d.mx + T::TN - 1) / T::TN, (d.my + T::C - 1) / T::C, d.mz);
  else if (DIR == 1) grid = dim3((d.mx + T::C - 1) / T::C, (d.my + T::TN - 1) / T::TN, d.mz);
  else grid = dim3((d.mx + T::C - 1) / T::C, (d.mz + T::TN - 1) / T::TN, d.my);
  if (sensor)
    weno_mix_flux_diff<DIR, ORD, kMaxSpec, true, VAR>
        <<<grid, T::NT, T::smem_bytes(), st>>>(z, eps_ref, th, sensor, threshold, pp);
  else
    weno_mix_flux_diff<DIR, ORD, kMaxSpec, false, VAR>
        <<<grid, T::NT, T::smem_bytes(), st>>>(z, eps_ref, th, nullptr, threshold, pp);
  return cudaGetLastError();
}

template <int DIR, int ORD>
cudaError_t launch_mix_dir(const Zone &z, double eps_ref, const Thermo &th, const double *sensor, double threshold,
                           const PPArgs &pp, int var, cudaStream_t st) {
  if (var == 1) return launch_mix_var<DIR, ORD, 1>(z, eps_ref, th, sensor, threshold, pp, st);
  if (var == 2) return launch_mix_var<DIR, ORD, 2>(z, eps_ref, th, sensor, threshold, pp, st);
  return launch_mix_var<DIR, ORD, 0>(z, eps_ref, th, sensor, threshold, pp, st);
}

template <int DIR, int ORD, int VAR>
cudaError_t set_mix_attr() {
  const int b = (int)MixTile<DIR, ORD, kMaxSpec, VAR>::smem_bytes();
  cudaError_t e = cudaFuncSetAttribute(weno_mix_flux_diff<DIR, ORD, kMaxSpec, false, VAR>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, b);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(weno_mix_flux_diff<DIR, ORD, kMaxSpec, true, VAR>,
                              cudaFuncAttributeMaxDynamicSharedMemorySize, b);
}

template <int DIR, int ORD>
cudaError_t set_mix_attrs() {
  cudaError_t e;
  if ((e = set_mix_attr<DIR, ORD, 0>()) != cudaSuccess) return e;
  if ((e = set_mix_attr<DIR, ORD, 1>()) != cudaSuccess) return e;
  return set_mix_attr<DIR, ORD, 2>();
}

}  // namespace

cudaError_t weno_mix_init_attributes() {
  cudaError_t e;
  if ((e = set_mix_attrs<0, 5>()) != cudaSuccess) return e;
  if ((e = set_mix_attrs<1, 5>()) != cudaSuccess) return e;
  if ((e = set_mix_attrs<2, 5>()) != cudaSuccess) return e;
  if ((e = set_mix_attrs<0, 7>()) != cudaSuccess) return e;
  if ((e = set_mix_attrs<1, 7>()) != cudaSuccess) return e;
  return set_mix_attrs<2, 7>();
}

// One sweep (dir 0/1/2) with tile variant var; the species count is fixed at
// 9 (kMaxSpec).  dt_dev / dt_host: the step's dt for the positive-preserving
// limiter (x sweep only, as in the reference).
cudaError_t launch_weno_mix_dir(const Zone &z, const Param &p, const Thermo &th, const double *dt_dev,
                                double dt_host, int dir, int var, cudaStream_t st) {
  const double eps_ref = kEpsWeno * p.weno_eps_scale;
  const double tr = p.sensor_threshold;
  const double *sn = tr > 1e-10 ? z.shock_sensor : nullptr;  // hybrid UD + WENO
  const PPArgs pp{p.positive_preserving && dir == 0 ? 1 : 0, dt_dev, dt_host, p.dim == 3 ? 1.0 / 3.0 : 0.5,
                  p.rho_ref};
  const bool w7 = p.inviscid_scheme == 72;
  if (dir == 0)
    return w7 ? launch_mix_dir<0, 7>(z, eps_ref, th, sn, tr, pp, var, st)
              : launch_mix_dir<0, 5>(z, eps_ref, th, sn, tr, pp, var, st);
  if (dir == 1)
    return w7 ? launch_mix_dir<1, 7>(z, eps_ref, th, sn, tr, pp, var, st)
              : launch_mix_dir<1, 5>(z, eps_ref, th, sn, tr, pp, var, st);
  return w7 ? launch_mix_dir<2, 7>(z, eps_ref, th, sn, tr, pp, var, st)
            : launch_mix_dir<2, 5>(z, eps_ref, th, sn, tr, pp, var, st);
}

// x, y and (3-D) z sweeps; var[d] is the tile variant of sweep d.
cudaError_t launch_weno_mix(const Zone &z, const Param &p, const Thermo &th, const double *dt_dev, double dt_host,
                            const int *var, cudaStream_t st, int *n_launch) {
  const int nd = z.d.mz > 1 ? 3 : 2;
  for (int dir = 0; dir < nd; ++dir) {
    cudaError_t e = launch_weno_mix_dir(z, p, th, dt_dev, dt_host, dir, var[dir], st);
    if (e != cudaSuccess) return e;
    *n_launch += 1;
  }
  return cudaSuccess;
}

}  // namespace cfk
