// Mixture thermodynamics and transport on the device.
//
// NASA-7 two-range polynomials with linear extrapolation outside
// [t_low, t_high] (the Combustion2Part branch, reference
// src/Thermo.cu:385-633), the temperature Newton iteration of
// compute_temperature_and_pressure (reference src/FieldOperation.cu:4-45) and
// the mixture-averaged viscosity / conductivity / diffusivity of
// compute_transport_property (reference src/Transport.cu:43-165).  The
// tables live in one device-resident Thermo block read through the uniform
// (warp-broadcast) cache.
#pragma once

#include "cfk_common.cuh"

namespace cfk {

struct Thermo {
  int n_spec;
  double imw[kMaxSpec], gas_const[kMaxSpec], mw[kMaxSpec];
  double t_low[kMaxSpec], t_mid[kMaxSpec], t_high[kMaxSpec];
  double low[kMaxSpec][7], high[kMaxSpec][7];
  // transport
  int geometry[kMaxSpec];
  double LJ_potent_inv[kMaxSpec], vis_coeff[kMaxSpec], ZRotF298[kMaxSpec];
  double WjDivWi_to_One4th[kMaxSpec][kMaxSpec];
  double sqrt_WiDivWjPl1Mul8[kMaxSpec][kMaxSpec];
  double binary_diffusivity_coeff[kMaxSpec][kMaxSpec];
  double kb_over_eps_jk[kMaxSpec][kMaxSpec];
  // powers of the tables that the collision integrals split into a power of T
  // and a constant: LJ_potent_inv^-0.145, kb_over_eps_jk^-0.15504; and
  // 1 / binary_diffusivity_coeff
  double LJ_pow[kMaxSpec], kb_pow[kMaxSpec][kMaxSpec], inv_bdc[kMaxSpec][kMaxSpec];
};

__host__ __device__ inline double sutherland(double t) {
  // reference src/Transport.cu:6-9; (T/288.16)^1.5 as x sqrt(x) (correctly
  // rounded sqrt and one product) instead of the general power function
  const double x = t / 288.16;
  return 1.7894e-5 * (x * sqrt(x)) * (288.16 + 110) / (t + 110);
}

// h and cp (J/kg, J/kg/K) of species i, extrapolated linearly outside its
// range: the polynomials are taken at the clamped temperature, so inside the
// range the extrapolation adds zero, and no branch is left.
__device__ __forceinline__ void enthalpy_cp_one(const Thermo *th, int i, double t, double &h, double &cp) {
  const double tt = fmin(fmax(t, th->t_low[i]), th->t_high[i]);
  const double *c = t < th->t_mid[i] ? th->low[i] : th->high[i];
  cp = th->gas_const[i] * fma(tt, fma(tt, fma(tt, fma(tt, c[4], c[3]), c[2]), c[1]), c[0]);
  const double p = fma(tt, fma(tt, fma(tt, fma(tt, 0.2 * c[4], 0.25 * c[3]), (1.0 / 3) * c[2]), 0.5 * c[1]), c[0]);
  h = fma(th->gas_const[i], fma(tt, p, c[5]), cp * (t - tt));
}

__device__ __forceinline__ void compute_enthalpy_and_cp(const Thermo *th, double t, double *h, double *cp) {
  for (int i = 0; i < th->n_spec; ++i) enthalpy_cp_one(th, i, t, h[i], cp[i]);
}

__device__ __forceinline__ void compute_enthalpy(const Thermo *th, double t, double *h) {
  for (int i = 0; i < th->n_spec; ++i) {
    double cp;
    enthalpy_cp_one(th, i, t, h[i], cp);
  }
}

// cp of species i.  The powers of t are summed in this order because the sound
// speed, and with it the CFL step, follows from it: the reaction step's first
// plan, floor(dt / (0.2 dt)) substeps, depends on the step's last bit.
__device__ __forceinline__ double cp_one(const Thermo *th, int i, double t) {
  const double tt = fmin(fmax(t, th->t_low[i]), th->t_high[i]);
  const double *c = t < th->t_mid[i] ? th->low[i] : th->high[i];
  const double t2 = tt * tt, t3 = t2 * tt, t4 = t3 * tt;
  return (c[0] + c[1] * tt + c[2] * t2 + c[3] * t3 + c[4] * t4) * th->gas_const[i];
}

__device__ __forceinline__ void compute_cp(const Thermo *th, double t, double *cp) {
  for (int i = 0; i < th->n_spec; ++i) cp[i] = cp_one(th, i, t);
}

// T from the internal energy by Newton's method, eps = 1e-5, at most 1000
// iterations, starting from the previous T (reference src/FieldOperation.cu:4-45).
// Returns false if the iteration cap was reached (the reference then keeps
// the last iterate; so does this routine).
__device__ __forceinline__ bool temperature_newton(const Thermo *th, int ns, const double *yk, double total_energy,
                                                   double rho, double V2, double &t, double &p) {
  double gas_const = 0;
  for (int l = 0; l < ns; ++l) gas_const += yk[l] * th->gas_const[l];
  const double e = total_energy / rho - 0.5 * V2;
  double err = 1;
  int iter = 0;
  double h_i[kMaxSpec], cp_i[kMaxSpec];
  while (err > 1e-5 && iter++ < 1000) {
    compute_enthalpy_and_cp(th, t, h_i, cp_i);
    double cp_tot = 0, h = 0;
    for (int l = 0; l < ns; ++l) {
      cp_tot += cp_i[l] * yk[l];
      h += h_i[l] * yk[l];
    }
    const double e_t = h - gas_const * t;
    const double cv = cp_tot - gas_const;
    const double t1 = t - (e_t - e) / cv;
    err = abs(1 - t1 / t);
    t = t1;
  }
  p = rho * t * gas_const;
  return err <= 1e-5;
}

// Collision integral of the pair (l, n), 1.0548 t^-0.15504 + (t + 0.55909)^
// -2.1705 at the reduced temperature t = T kb/eps (reference
// src/Transport.cu:182-184).  The first power is T^-0.15504 (t_pow) times a
// table; the second is x^-2 exp(-0.1705 ln x), whose small exponent keeps the
// logarithm's rounding below an ulp of the result.  One logarithm and one
// exponential a pair instead of two general powers.
__device__ __forceinline__ double omega_d(const Thermo *th, int l, int n, double temperature, double t_pow) {
  const double x = fma(temperature, th->kb_over_eps_jk[l][n], 0.55909);
  return fma(1.0548 * th->kb_pow[l][n], t_pow, rcp_nr(x * x) * exp(-0.1705 * log(x)));
}

// gamma, acoustic speed, Mach, mu, kappa, rho*D_k at one node
// (reference src/FieldOperation.cuh:95-114, src/Transport.cu:43-165).
// Bound by the 45 collision integrals (FP64 and instruction issue); the pair
// loops stay loops: unrolled, their code overflows the instruction cache.  The
// update of a 97 x 49 x 33 block with its properties took 240 us with two
// general powers a pair, a reciprocal root a pair of the mixing rule and
// divisions throughout, and the shell as much again.
__device__ __forceinline__ void mixture_properties_point(const Zone &z, const Param &p, const Thermo *th, int64_t id,
                                                         double temperature, double V) {
  const int64_t sz = z.d.plane(z.d.ngg);
  const int ns = p.n_spec;
  double imw = 0, cpm = 0;
  double cp[kMaxSpec], X[kMaxSpec], vis[kMaxSpec], sq[kMaxSpec], rsq[kMaxSpec];
  for (int l = 0; l < ns; ++l) {
    const double y = z.sv[id + l * sz];
    cp[l] = cp_one(th, l, temperature);
    X[l] = y * th->imw[l];
    imw = fma(y, th->imw[l], imw);
    cpm = fma(y, cp[l], cpm);
  }
  const double R = kRu * imw;
  const double gam = cpm / (cpm - R);
  z.gamma[id] = gam;
  const double a = sqrt(gam * R * temperature);
  z.acoustic_speed[id] = a;
  if (z.mach) z.mach[id] = V / a;

  const double mw_total = 1 / imw;
  const double root_t = sqrt(temperature), t_15 = temperature * root_t;
  const double lj_t = 1.147 * pow(temperature, -0.145), t_pow = pow(temperature, -0.15504);
  const double iT = rcp_nr(temperature);
  for (int l = 0; l < ns; ++l) {
    X[l] *= mw_total;
    const double t5 = fma(temperature, th->LJ_potent_inv[l], 0.5);
    vis[l] = th->vis_coeff[l] * root_t * rcp_nr(fma(lj_t, th->LJ_pow[l], rcp_nr(t5 * t5)));
    rsq[l] = rsqrt(vis[l]);
    sq[l] = vis[l] * rsq[l];
  }
  double viscosity = 0, conductivity = 0;
  constexpr double pi = 3.141592653589793;
  for (int m = 0; m < ns; ++m) {
    const double Rm = th->gas_const[m], vm = vis[m];
    double lambda = 15 * 0.25 * vm * Rm;
    const int geom = th->geometry[m];
    if (geom == 1 || geom == 2) {
      const double tRedInv = rcp_nr(temperature * th->kb_over_eps_jk[m][m]);
      const double root = sqrt(tRedInv * pi) * pi;
      const double FT = 1 + 0.5 * root + (2 + 0.25 * pi * pi) * tRedInv + root * tRedInv;
      const double rhoD = th->binary_diffusivity_coeff[m][m] * t_15 * iT *
                          rcp_nr(omega_d(th, m, m, temperature, t_pow) * Rm);
      // 10/3 and 2.5 a rotational degree pair: linear, 5 and 3 A/(pi B) - 2.5: non-linear molecules
      const double rot = geom == 1 ? 10.0 / 3 : 5.0, dof = geom == 1 ? 1.0 : 1.5;
      const double ADivPiB =
          (2.5 * vm - rhoD) * rcp_nr(pi * th->ZRotF298[m] * vm * rcp_nr(FT) + rot * vm + 2.0 * rhoD);
      lambda += -5 * dof * ADivPiB * vm * Rm + rhoD * cp[m] + rhoD * (2 * dof * ADivPiB - 2.5) * Rm;
    }
    double part = 0;
    const double s = sq[m];
    for (int n = 0; n < ns; ++n) {
      const double num = fma(rsq[n] * s, th->WjDivWi_to_One4th[m][n], 1.0);
      part = fma(m == n ? 1.0 : num * num * th->sqrt_WiDivWjPl1Mul8[m][n], X[n], part);
    }
    viscosity += vm * X[m] * rcp_nr(part);
    conductivity += lambda * X[m] * rcp_nr(1.065 * part - 0.065 * X[m]);
  }
  z.mul[id] = viscosity;
  z.thermal_conductivity[id] = conductivity;
  constexpr double eps = 1e-12;
  double sum = 0;
  for (int l = 0; l < ns; ++l) {
    X[l] += eps;
    sum = fma(X[l], th->mw[l], sum);
    vis[l] = 0;
  }
#pragma unroll 1
  for (int l = 0; l < ns; ++l) {
    double acc = vis[l];
    const double xl = X[l];
#pragma unroll 2
    for (int n = l + 1; n < ns; ++n) {
      const double o = omega_d(th, l, n, temperature, t_pow) * th->inv_bdc[l][n];
      acc = fma(X[n], o, acc);
      vis[n] = fma(xl, o, vis[n]);
    }
    z.rho_D[id + l * sz] = fma(-X[l], th->mw[l], sum) * (t_15 * iT * (1.0 / kRu)) * rcp_nr(acc);
  }
}

// Viscous spectral-radius velocity of the mixture (reference
// src/TimeAdvanceFunc.cuh:72-85).
__device__ __forceinline__ double mixture_max_diffuse_vel(const Zone &z, const Param &p, const Thermo *th, int64_t id,
                                                          double iRho) {
  const int64_t sz = z.d.plane(z.d.ngg);
  double cpl[kMaxSpec];
  compute_cp(th, z.bv[id + 5 * sz], cpl);
  double cp = 0, max_rhoD = 0;
  for (int l = 0; l < p.n_spec; ++l) {
    cp += cpl[l] * z.sv[id + l * sz];
    max_rhoD = max(max_rhoD, z.rho_D[id + l * sz]);
  }
  double mdv = z.mul[id] * iRho;
  mdv = max(mdv, z.thermal_conductivity[id] * iRho * z.gamma[id] / cp);
  mdv = max(mdv, max_rhoD * iRho);
  return mdv;
}

}  // namespace cfk
