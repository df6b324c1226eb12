// Scalar WENO5-JS / WENO7-Z reconstructions of the split characteristic
// fluxes at i+1/2 (reference src/WENO.cu:3059-3222): same substencils,
// smoothness indicators and weights, in exact arithmetic; vp[] and vm[] run
// left to right and the result is f+ + f-.
#pragma once

namespace cfk {

// Dot products with a fixed order of FMAs.  Where the compiler chooses which
// product of a sum to fuse, the choice can differ between the instantiations
// of a kernel; the tile shapes of a sweep give bit-identical fluxes.
__device__ __forceinline__ double dot2(double a0, double b0, double a1, double b1) { return fma(a0, b0, a1 * b1); }
__device__ __forceinline__ double dot3(double a0, double b0, double a1, double b1, double a2, double b2) {
  return fma(a0, b0, fma(a1, b1, a2 * b2));
}
// (the product with a zero addend rounds like the product alone)
__device__ __forceinline__ double dot4p(double a0, double b0, double a1, double b1, double a2, double b2, double a3,
                                        double b3, double plus) {
  return fma(a0, b0, fma(a1, b1, fma(a2, b2, fma(a3, b3, plus))));
}

// WENO5-JS, f+ + f-.  Everything is formed from the differences of the stencil
// values, d_i = u_{i+1} - u_i and s_i = d_{i+1} - d_i: the substencil values
// are u2 plus a combination of them, the smoothness indicators
// 13/12 s^2 + (first derivative)^2.  The weights a_k = d_k / (eps + beta_k)^2
// enter only through sum(a_k v_k) / sum(a_k); both sums are multiplied through
// by the product of the three denominators, so one division per side remains.
// The sides are not merged into one division: in flat regions the products are
// O(eps^4) and their cross product would underflow.
__device__ __forceinline__ void weno5_side(double u0, double u1, double u2, double u3, double u4, double eps,
                                           double &num, double &den) {
  constexpr double one6th{1.0 / 6}, one3rd{1.0 / 3}, t12{13.0 / 12};
  const double d0 = u1 - u0, d1 = u2 - u1, d2 = u3 - u2, d3 = u4 - u3;
  const double s0 = d1 - d0, s1 = d2 - d1, s2 = d3 - d2;
  const double h0 = fma(-0.5, s2, d2), h1 = fma(0.5, s1, d1), h2 = fma(0.5, s0, d1);
  const double b0 = fma(t12 * s2, s2, fma(h0, h0, eps));
  const double b1 = fma(t12 * s1, s1, fma(h1, h1, eps));
  const double b2 = fma(t12 * s0, s0, fma(h2, h2, eps));
  const double m01 = b0 * b1, m02 = b0 * b2, m12 = b1 * b2;
  const double a0 = (0.3 * m12) * m12, a1 = (0.6 * m02) * m02, a2 = (0.1 * m01) * m01;
  const double hd = 0.5 * d2;
  const double v0 = fma(-one6th, s2, hd), v1 = fma(-one6th, s1, hd), v2 = fma(one3rd, s0, 0.5 * d1);
  num = fma(a2, v2, fma(a1, v1, a0 * v0));
  den = __dadd_rn(__dadd_rn(a0, a1), a2);  // not contracted with the products
}

__device__ __forceinline__ double weno5_js(const double *vp, const double *vm, double eps) {
  double np, dp, nm, dm;
  weno5_side(vp[0], vp[1], vp[2], vp[3], vp[4], eps, np, dp);
  // mirrored: minus-side substencil k is plus-side substencil 2-k, same linear weights
  weno5_side(vm[4], vm[3], vm[2], vm[1], vm[0], eps, nm, dm);
  return (vp[2] + vm[2]) + fma(np, rcp_nr(dp), nm * rcp_nr(dm));
}

// One side of WENO7-Z: u[0..6] ordered from the far upwind point to the far
// downwind point of the stencil, formed from the first, second and third
// differences d, s, t of the values.  With s1', s2 and s3 the first (shifted by
// s3 / 24), second and third differences at u3 of a substencil, the indicator
// s1^2 + 13/12 s2^2 + 1043/960 s3^2 + s1 s3 / 12 is
// s1'^2 + 13/12 s2^2 + 781/720 s3^2.  The weights c_k (1 + (T / e_k)^2),
// e_k = eps + beta_k, T = e0 + 3 e1 - 3 e2 - e3, take one reciprocal, of
// e0 e1 e2 e3 (>= eps^4, a normal number, see validate() in capi.cu; a product
// of the squares would underflow in flat regions).  Returns numerator and
// denominator of sum(a_k (v_k - u3)) / sum(a_k).  About 75 FP64 instructions
// and one reciprocal a side, against 118 and two divisions when every
// indicator and value is formed from the u[i].
__device__ __forceinline__ void weno7_z_side(double u0, double u1, double u2, double u3, double u4, double u5,
                                             double u6, double eps, double &num, double &den) {
  constexpr double c0{1.0 / 35}, c1{12.0 / 35}, c2{18.0 / 35}, c3{4.0 / 35};
  constexpr double b2{13.0 / 12.0}, b3{781.0 / 720}, one3rd{1.0 / 3}, one6th{1.0 / 6}, one12th{1.0 / 12};
  const double d0 = u1 - u0, d1 = u2 - u1, d2 = u3 - u2, d3 = u4 - u3, d4 = u5 - u4, d5 = u6 - u5;
  const double s0 = d1 - d0, s1 = d2 - d1, s2 = d3 - d2, s3 = d4 - d3, s4 = d5 - d4;
  const double t0 = s1 - s0, t1 = s2 - s1, t2 = s3 - s2, t3 = s4 - s3;
  const double mid = fma(0.5, s2, d2);  // (u4 - u2) / 2
  const double p0 = fma(0.375, t0, fma(0.5, s1, d2)), q0 = s1 + t0;
  const double p1 = fma(-0.125, t1, mid), p2 = fma(-0.125, t2, mid);
  const double p3 = fma(0.375, t3, fma(-0.5, s3, d3)), q3 = s3 - t3;
  const double m12 = fma(b2 * s2, s2, eps);  // shared by the two middle substencils
  const double e0 = fma(b3 * t0, t0, fma(b2 * q0, q0, fma(p0, p0, eps)));
  const double e1 = fma(b3 * t1, t1, fma(p1, p1, m12));
  const double e2 = fma(b3 * t2, t2, fma(p2, p2, m12));
  const double e3 = fma(b3 * t3, t3, fma(b2 * q3, q3, fma(p3, p3, eps)));
  const double tau = fma(3.0, e1 - e2, e0 - e3);
  const double e01 = e0 * e1, e23 = e2 * e3;
  const double r = rcp_nr(e01 * e23) * tau;
  const double r01 = r * e23, r23 = r * e01;  // tau / (e0 e1), tau / (e2 e3)
  const double w0 = r01 * e1, w1 = r01 * e0, w2 = r23 * e3, w3 = r23 * e2;
  const double a0 = fma(c0 * w0, w0, c0), a1 = fma(c1 * w1, w1, c1);
  const double a2 = fma(c2 * w2, w2, c2), a3 = fma(c3 * w3, w3, c3);
  const double hd = 0.5 * d3, mv = fma(-one6th, s2, hd);
  const double v0 = fma(0.25, t0, fma(one3rd, s1, 0.5 * d2));
  const double v1 = fma(-one12th, t1, mv), v2 = fma(-one12th, t2, mv);
  const double v3 = fma(one12th, t3, fma(-one6th, s3, hd));
  num = fma(a3, v3, fma(a2, v2, fma(a1, v1, a0 * v0)));
  den = (a0 + a1) + (a2 + a3);
}

// f+ + f-, one division shared by the two sides (each sum(a_k) >= 1, so the
// product of the two denominators cannot underflow).
__device__ __forceinline__ double weno7_z(const double *vp, const double *vm, double eps) {
  double np, dp, nm, dm;
  weno7_z_side(vp[0], vp[1], vp[2], vp[3], vp[4], vp[5], vp[6], eps, np, dp);
  weno7_z_side(vm[6], vm[5], vm[4], vm[3], vm[2], vm[1], vm[0], eps, nm, dm);
  return fma(fma(np, dm, nm * dp), rcp_nr(dp * dm), vp[3] + vm[3]);
}

// Linear branches of WENO5 / WENO7 used by the hybrid scheme away from
// shocks (reference src/WENO.cu:3100-3113 and 3204-3221): the substencil
// values combined with the optimal weights, which collapse to the 5- and
// 7-point upwind-biased stencils (UD5: (2, -13, 47, 27, -3) / 60;
// UD7: (-3, 25, -101, 319, 214, -38, 4) / 420).  The minus side is the plus
// side read right to left.
__device__ __forceinline__ double ud5_side(double u0, double u1, double u2, double u3, double u4) {
  constexpr double r60{1.0 / 60};
  return r60 * (2 * u0 - 13 * u1 + 47 * u2 + 27 * u3 - 3 * u4);
}

__device__ __forceinline__ double weno5_linear(const double *vp, const double *vm) {
  return ud5_side(vp[0], vp[1], vp[2], vp[3], vp[4]) + ud5_side(vm[4], vm[3], vm[2], vm[1], vm[0]);
}

__device__ __forceinline__ double ud7_side(double u0, double u1, double u2, double u3, double u4, double u5,
                                           double u6) {
  constexpr double r420{1.0 / 420};
  return r420 * (-3 * u0 + 25 * u1 - 101 * u2 + 319 * u3 + 214 * u4 - 38 * u5 + 4 * u6);
}

__device__ __forceinline__ double weno7_linear(const double *vp, const double *vm) {
  return ud7_side(vp[0], vp[1], vp[2], vp[3], vp[4], vp[5], vp[6]) +
         ud7_side(vm[6], vm[5], vm[4], vm[3], vm[2], vm[1], vm[0]);
}

// Hybrid switch of the WENO sweeps (reference src/WENO.cu:839-849, 1580-1590
// and the z sweep): the face between node idf and idf + sd takes the
// nonlinear weights when the sensor of any node idf + ii*sd, ii in
// [-g+1, g], exceeds the threshold.  sensor == nullptr: WENO everywhere.
__device__ __forceinline__ bool face_shocked(const double *sensor, int64_t idf, int64_t sd, int g,
                                             double threshold) {
  if (sensor == nullptr) return true;
  for (int ii = -g + 1; ii <= g; ++ii)
    if (__ldg(sensor + idf + ii * sd) > threshold) return true;
  return false;
}

}  // namespace cfk
