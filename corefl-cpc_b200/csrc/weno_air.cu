// Fused characteristic WENO flux + flux difference, calorically perfect air.
//
// Restates compute_convective_term_weno_{x,y,z} with the air characteristic
// helpers (reference src/WENO.cu:831-1138, 10-244, 414-654) followed by
// compute_derivative_{x,y,z} (reference src/WENO.cu:1544, 2219, 2885), as one
// kernel per direction:
//
//   stage   — each CTA stages the stencil points of a tile (a segment of TN
//             nodes along the sweep direction times C columns) into shared
//             memory: conserved Q[5], the Euler flux G[5] along the face
//             normal, p, J/2 and the spectral radius |U_k| + c|grad k|;
//   faces   — each thread projects the 2R+2 stencil points of one face onto
//             the Roe-averaged left eigenvectors, splits them with the local
//             Lax-Friedrichs bound, reconstructs with WENO5-JS / WENO7-Z (or,
//             for the hybrid scheme, with the linear UD5 / UD7 weights where no
//             stencil node is shocked) and projects back; the face fluxes stay
//             in shared memory;
//   diff    — dq(n) -= F(n+1/2) - F(n-1/2) for the tile's nodes.
//
// The face flux never goes to HBM and dq is read-modified-written once per
// direction instead of through a separate derivative pass.  Loads are
// coalesced along i in every direction: x tiles put consecutive faces on
// consecutive lanes, y/z tiles put consecutive i columns on them.
#include "cfk_common.cuh"
#include "weno.cuh"
#include "weno_tiles.cuh"

namespace cfk {

namespace {

constexpr int kNQ = 13;  // staged values per point: Q0..4, G0..4, p, J/2, lambda

// Tile shapes of a sweep: VAR selects one of the CFK_TILE_VARIANTS shapes
// (nodes per column TN x columns C), chosen per direction by weno_air_tile
// (weno_tiles.cuh) or the tile autotuner.  x tiles run along the lanes,
// y/z tiles put C consecutive i columns on the lanes.  Tiles are small, one or
// two faces a thread of a 128-thread CTA: four CTAs fit an SM and their
// stage, face and difference phases overlap.  With the same 128 registers and
// 16 warps an SM, two 256-thread CTAs took 984 us on the WENO7 sweeps of a
// 161 x 113 x 97 block against 886; fewer warps with 168 registers took 990
// (128 x 3) to 1100 (192 x 2).
template <int DIR, int VAR>
struct TileShape {
  static constexpr int TN = kAirTileNodes[DIR > 0][VAR], C = kAirTileColumns[DIR > 0][VAR];
};

template <int DIR, int ORD, int VAR = 0>
struct AirTile {
  static constexpr int R = ORD == 7 ? 3 : 2;          // stencil reach left of the face node
  static constexpr int NPF = 2 * R + 2;               // points per face
  static constexpr int TN = TileShape<DIR, VAR>::TN;  // nodes per column
  static constexpr int C = TileShape<DIR, VAR>::C;    // columns per CTA
  static constexpr int NF = TN + 1;             // faces per column
  static constexpr int NPT = TN + 2 * R + 2;    // staged points per column
  static constexpr int NT = 128;                // threads
  // shared-memory offset of (value q, column c, point/face t): x tiles are
  // column-major in t (lanes run along t), y/z tiles are row-major in c.
  __device__ static int spt(int q, int c, int t) {
    return DIR == 0 ? (q * C + c) * NPT + t : (q * NPT + t) * C + c;
  }
  __device__ static int sfl(int v, int c, int t) {
    return DIR == 0 ? (v * C + c) * NF + t : (v * NF + t) * C + c;
  }
  static constexpr size_t smem_bytes() { return sizeof(double) * (size_t)(kNQ * C * NPT + 5 * C * NF); }
};

}  // namespace

// The 13 staged values of one stencil point from its conserved variables,
// p, T, the sweep's metric row and J: J/2 times Q and the Euler flux G (the
// split fluxes need nothing else), p, 2/J (which gives the Roe average its
// unscaled state back) and the spectral radius.
template <class T>
__device__ __forceinline__ void air_stage_point(double *s, int c, int t, double q0, double q1, double q2, double q3,
                                                double q4, double pk, double tk, double m0, double m1, double m2,
                                                double jac) {
  const double Uk = dot3(q1, m0, q2, m1, q3, m2) * rcp_nr(q0);
  const double lam = __dadd_rn(abs(Uk), sqrt(dot3(m0, m0, m1, m1, m2, m2) * (kGammaAir * kRAir * tk)));
  const double hj = 0.5 * jac, hp = hj * pk;
  q0 *= hj; q1 *= hj; q2 *= hj; q3 *= hj; q4 *= hj;
  s[T::spt(0, c, t)] = q0;
  s[T::spt(1, c, t)] = q1;
  s[T::spt(2, c, t)] = q2;
  s[T::spt(3, c, t)] = q3;
  s[T::spt(4, c, t)] = q4;
  s[T::spt(5, c, t)] = q0 * Uk;
  s[T::spt(6, c, t)] = fma(q1, Uk, hp * m0);
  s[T::spt(7, c, t)] = fma(q2, Uk, hp * m1);
  s[T::spt(8, c, t)] = fma(q3, Uk, hp * m2);
  s[T::spt(9, c, t)] = __dadd_rn(q4, hp) * Uk;
  s[T::spt(10, c, t)] = pk;
  s[T::spt(11, c, t)] = rcp_nr(hj);
  s[T::spt(12, c, t)] = lam;
}

// Flux of the face between local points t + R and t + R + 1 of column c:
// Roe average, characteristic basis, Lax-Friedrichs split of the 2R + 2
// staged points, WENO (or, away from shocks in the hybrid scheme, the linear
// upwind stencils) and back projection into sflx.  kx, ky, kz: the face
// normal before normalisation.
//
// The five fields are taken as two pairs, the shear fields (1, 2) and the
// acoustic ones (0, 4), and the entropy field 3: the two fields of a pair
// share the loads of the staged points, which at one field at a time kept the
// shared-memory pipe as busy as the FP64 one.  The pair loop is not unrolled:
// unrolled, the stencil loads of all fields are hoisted above the first
// field's arithmetic and spill; __syncwarp keeps them below it (so every lane
// of a warp comes here, with valid = false where it has no face).  FP64-bound:
// the three WENO7 sweeps of a 161 x 113 x 97 block went from 1217 to 793 us,
// WENO5 of 200 x 150 x 150 from 2060 to 1270 us.
template <int ORD, class T>
__device__ __forceinline__ void air_face(const double *s, double *sflx, int c, int t, double kx, double ky, double kz,
                                         double eps_ref, bool shock, bool valid) {
  constexpr int R = T::R, NPF = T::NPF;
  constexpr double gm1 = kGammaAir - 1;
  auto recon = [&](const double *vp, const double *vm) -> double {
    if constexpr (ORD == 7) return shock ? weno7_z(vp, vm, eps_ref) : weno7_linear(vp, vm);
    else return shock ? weno5_js(vp, vm, eps_ref) : weno5_linear(vp, vm);
  };
  const int pc = t + R;  // local point of node f
  const double il = s[T::spt(11, c, pc)], ir = s[T::spt(11, c, pc + 1)];
  const double rho_l = s[T::spt(0, c, pc)] * il, rho_r = s[T::spt(0, c, pc + 1)] * ir;
  const double root = sqrt(rho_l * rho_r);
  const double rlc = rcp_nr(__dadd_rn(rho_l, root)), rrc = rcp_nr(__dadd_rn(root, rho_r));
  const double sl = rlc * il, sr = rrc * ir;  // weights of the scaled conserved variables
  const double um = dot2(sl, s[T::spt(1, c, pc)], sr, s[T::spt(1, c, pc + 1)]);
  const double vm = dot2(sl, s[T::spt(2, c, pc)], sr, s[T::spt(2, c, pc + 1)]);
  const double wm = dot2(sl, s[T::spt(3, c, pc)], sr, s[T::spt(3, c, pc + 1)]);
  const double pr = dot2(rlc, s[T::spt(10, c, pc)], rrc, s[T::spt(10, c, pc + 1)]);  // R T of the Roe average
  const double H = fma(sl, s[T::spt(4, c, pc)], fma(sr, s[T::spt(4, c, pc + 1)], pr));
  const double c2 = kGammaAir * pr, cm = sqrt(c2), ic2 = rcp_nr(c2);

  double nrm = rsqrt(dot3(kx, kx, ky, ky, kz, kz));
  kx *= nrm; ky *= nrm; kz *= nrm;
  const double Uk_bar = dot3(kx, um, ky, vm, kz, wm);
  // rows of the two fields of a pair and their common energy coefficient,
  // first the shear fields: n and q = k x n complete the basis
  double A1 = 0, A2 = 0, A3 = 0;
  if (abs(kx) > 0.8) { A1 = -kz; A3 = kx; }
  else { A2 = kz; A3 = -ky; }
  nrm = rsqrt(dot3(A1, A1, A2, A2, A3, A3));
  A1 *= nrm; A2 *= nrm; A3 *= nrm;
  double B1 = dot2(ky, A3, -kz, A2), B2 = dot2(kz, A1, -kx, A3), B3 = dot2(kx, A2, -ky, A1);
  double A0 = -dot3(A1, um, A2, vm, A3, wm), B0 = -dot3(B1, um, B2, vm, B3, wm), E = 0;
  const double alpha = 0.5 * gm1 * dot3(um, um, vm, vm, wm, wm);

  double lam = 0;
#pragma unroll
  for (int q = 0; q < NPF; ++q) lam = max(lam, s[T::spt(12, c, t + q)]);

  double f1 = 0, f2 = 0, f3 = 0, f4 = 0, ca, cb;
#pragma unroll 1
  for (int pair = 0;; ++pair) {
    __syncwarp();
    double va[NPF - 1], wa[NPF - 1], vb[NPF - 1], wb[NPF - 1];
#pragma unroll
    for (int q = 0; q < NPF; ++q) {
      const int tq = t + q;
      const double g0 = s[T::spt(5, c, tq)], g1 = s[T::spt(6, c, tq)], g2 = s[T::spt(7, c, tq)],
                   g3 = s[T::spt(8, c, tq)], eg = E * s[T::spt(9, c, tq)];
      const double q0 = s[T::spt(0, c, tq)], q1 = s[T::spt(1, c, tq)], q2 = s[T::spt(2, c, tq)],
                   q3 = s[T::spt(3, c, tq)], eq = E * s[T::spt(4, c, tq)];
      const double Fa = dot4p(A0, g0, A1, g1, A2, g2, A3, g3, eg);
      const double Fb = dot4p(B0, g0, B1, g1, B2, g2, B3, g3, eg);
      const double Qa = dot4p(A0, q0, A1, q1, A2, q2, A3, q3, eq);
      const double Qb = dot4p(B0, q0, B1, q1, B2, q2, B3, q3, eq);
      if (q < NPF - 1) { va[q] = fma(lam, Qa, Fa); vb[q] = fma(lam, Qb, Fb); }
      if (q > 0) { wa[q - 1] = fma(-lam, Qa, Fa); wb[q - 1] = fma(-lam, Qb, Fb); }
    }
    ca = recon(va, wa);
    cb = recon(vb, wb);
    if (pair) break;
    // back projection of the shear fields; next the acoustic pair
    f1 = dot2(A1, ca, B1, cb);
    f2 = dot2(A2, ca, B2, cb);
    f3 = dot2(A3, ca, B3, cb);
    f4 = -dot2(A0, ca, B0, cb);
    const double h = 0.5 * ic2;
    E = gm1 * h;
    const double kc = cm * h, a0 = alpha * h;
    A0 = fma(Uk_bar, kc, a0); A1 = -dot2(E, um, kx, kc); A2 = -dot2(E, vm, ky, kc); A3 = -dot2(E, wm, kz, kc);
    B0 = fma(-Uk_bar, kc, a0); B1 = dot2(kx, kc, -E, um); B2 = dot2(ky, kc, -E, vm); B3 = dot2(kz, kc, -E, wm);
  }
  const double f04 = cm * (ca - cb);
  double f034 = ca + cb;
  {
    const double L4 = -gm1 * ic2, L0 = fma(-alpha, ic2, 1.0), L1 = -L4 * um, L2 = -L4 * vm, L3 = -L4 * wm;
    __syncwarp();
    double va[NPF - 1], wa[NPF - 1];
#pragma unroll
    for (int q = 0; q < NPF; ++q) {
      const int tq = t + q;
      const double F = dot4p(L0, s[T::spt(5, c, tq)], L1, s[T::spt(6, c, tq)], L2, s[T::spt(7, c, tq)], L3,
                             s[T::spt(8, c, tq)], L4 * s[T::spt(9, c, tq)]);
      const double Q = dot4p(L0, s[T::spt(0, c, tq)], L1, s[T::spt(1, c, tq)], L2, s[T::spt(2, c, tq)], L3,
                             s[T::spt(3, c, tq)], L4 * s[T::spt(4, c, tq)]);
      if (q < NPF - 1) va[q] = fma(lam, Q, F);
      if (q > 0) wa[q - 1] = fma(-lam, Q, F);
    }
    const double c3 = recon(va, wa);
    f034 += c3;
    f4 = fma(-c2 * (1 / gm1), c3, f4);
  }
  if (!valid) return;
  // right eigenvectors written out (reference src/WENO.cu:229-243)
  sflx[T::sfl(0, c, t)] = f034;
  sflx[T::sfl(1, c, t)] = fma(um, f034, fma(-kx, f04, f1));
  sflx[T::sfl(2, c, t)] = fma(vm, f034, fma(-ky, f04, f2));
  sflx[T::sfl(3, c, t)] = fma(wm, f034, fma(-kz, f04, f3));
  sflx[T::sfl(4, c, t)] = fma(H, f034, fma(-Uk_bar, f04, f4));
}

// HYB: hybrid UD/WENO scheme, the face switches on the shock sensor.
// VAR: tile shape (TileShape).
template <int DIR, int ORD, bool HYB, int VAR>
__global__ void __launch_bounds__(128, 4) weno_air_flux_diff(Zone z, double eps_ref, const double *sensor,
                                                              double threshold) {
  using T = AirTile<DIR, ORD, VAR>;
  constexpr int R = T::R, TN = T::TN, C = T::C, NF = T::NF, NPT = T::NPT;
  static_assert(NF * C % T::NT == 0, "every lane of a warp comes to the __syncwarp of air_face in every round");
  extern __shared__ double sm[];
  double *spts = sm;
  double *sflx = sm + kNQ * C * NPT;

  const Dims d = z.d;
  const int g = d.ngg;
  const int64_t sz = d.plane(g), szq = d.plane(0);
  const int m = d.ext(DIR);

  // tile origin: n0 along DIR, column origin across
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

  const int mmo = 3 * DIR;  // metric offset of this direction's grad(xi_dir)
  // ---- stage ------------------------------------------------------------
  for (int item = threadIdx.x; item < NPT * C; item += T::NT) {
    int c, t;
    split(item, NPT, c, t);
    const int a = n0 - 1 - R + t;
    if (cbase + c >= ncol_max || a > m + R) continue;
    const int64_t id = node_idx(g, c, a);
    const double q0 = z.cv[id], q1 = z.cv[id + sz], q2 = z.cv[id + 2 * sz], q3 = z.cv[id + 3 * sz],
                 q4 = z.cv[id + 4 * sz];
    const double pk = z.bv[id + 4 * sz], tk = z.bv[id + 5 * sz];
    const double m0 = z.metric[id + mmo * sz], m1 = z.metric[id + (mmo + 1) * sz],
                 m2 = z.metric[id + (mmo + 2) * sz];
    const double jac = z.jac[id];
    air_stage_point<T>(spts, c, t, q0, q1, q2, q3, q4, pk, tk, m0, m1, m2, jac);
  }
  __syncthreads();

  // ---- face fluxes ------------------------------------------------------
  for (int item = threadIdx.x; item < NF * C; item += T::NT) {
    int c, t;
    split(item, NF, c, t);
    const int f = n0 - 1 + t;  // face between node f and f+1 along DIR
    const bool valid = cbase + c < ncol_max && f < m;
    // face normal, averaged with the (i+1) node in every direction as the
    // reference does (reference src/WENO.cu:886-888, 1627-1629, 2303-2305)
    const int64_t idf = valid ? node_idx(g, c, f) : 0;
    double kx = 0.5 * (z.metric[idf + mmo * sz] + z.metric[idf + 1 + mmo * sz]);
    double ky = 0.5 * (z.metric[idf + (mmo + 1) * sz] + z.metric[idf + 1 + (mmo + 1) * sz]);
    double kz = 0.5 * (z.metric[idf + (mmo + 2) * sz] + z.metric[idf + 1 + (mmo + 2) * sz]);

    const bool shock = !HYB || (valid && face_shocked(sensor, idf, d.stride(g, DIR), g, threshold));
    air_face<ORD, T>(spts, sflx, c, t, kx, ky, kz, eps_ref, shock, valid);
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
    for (int v = 0; v < 5; ++v) red_add(z.dq + iq + v * szq, sflx[T::sfl(v, c, t)] - sflx[T::sfl(v, c, t + 1)]);
  }
}

template <int DIR, int ORD, int VAR>
static cudaError_t launch_var(const Zone &z, double eps_ref, const double *sensor, double threshold,
                              cudaStream_t st) {
  using T = AirTile<DIR, ORD, VAR>;
  const Dims &d = z.d;
  dim3 grid;
  if (DIR == 0) grid = dim3((d.mx + T::TN - 1) / T::TN, (d.my + T::C - 1) / T::C, d.mz);
  else if (DIR == 1) grid = dim3((d.mx + T::C - 1) / T::C, (d.my + T::TN - 1) / T::TN, d.mz);
  else grid = dim3((d.mx + T::C - 1) / T::C, (d.mz + T::TN - 1) / T::TN, d.my);
  const size_t smem = T::smem_bytes();
  if (sensor) weno_air_flux_diff<DIR, ORD, true, VAR><<<grid, T::NT, smem, st>>>(z, eps_ref, sensor, threshold);
  else weno_air_flux_diff<DIR, ORD, false, VAR><<<grid, T::NT, smem, st>>>(z, eps_ref, nullptr, threshold);
  return cudaGetLastError();
}

template <int DIR, int ORD>
static cudaError_t launch_dir(const Zone &z, double eps_ref, const double *sensor, double threshold, int var,
                              cudaStream_t st) {
  if (var == 1) return launch_var<DIR, ORD, 1>(z, eps_ref, sensor, threshold, st);
  if (var == 2) return launch_var<DIR, ORD, 2>(z, eps_ref, sensor, threshold, st);
  return launch_var<DIR, ORD, 0>(z, eps_ref, sensor, threshold, st);
}

template <int DIR, int ORD, int VAR>
static cudaError_t set_smem_attr() {
  const int b = (int)AirTile<DIR, ORD, VAR>::smem_bytes();
  cudaError_t e = cudaFuncSetAttribute(weno_air_flux_diff<DIR, ORD, false, VAR>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, b);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(weno_air_flux_diff<DIR, ORD, true, VAR>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              b);
}

template <int DIR, int ORD>
static cudaError_t set_smem_attrs() {
  cudaError_t e;
  if ((e = set_smem_attr<DIR, ORD, 0>()) != cudaSuccess) return e;
  if ((e = set_smem_attr<DIR, ORD, 1>()) != cudaSuccess) return e;
  return set_smem_attr<DIR, ORD, 2>();
}

// Opt every instantiation in to its dynamic shared-memory size (> 48 KB for
// the y/z tiles).  Called once per device at context creation, outside any
// stream capture.
cudaError_t weno_air_init_attributes() {
  cudaError_t e;
  if ((e = set_smem_attrs<0, 5>()) != cudaSuccess) return e;
  if ((e = set_smem_attrs<1, 5>()) != cudaSuccess) return e;
  if ((e = set_smem_attrs<2, 5>()) != cudaSuccess) return e;
  if ((e = set_smem_attrs<0, 7>()) != cudaSuccess) return e;
  if ((e = set_smem_attrs<1, 7>()) != cudaSuccess) return e;
  return set_smem_attrs<2, 7>();
}

// One sweep (dir 0/1/2) with tile variant var.
cudaError_t launch_weno_air_dir(const Zone &z, const Param &p, int dir, int var, cudaStream_t st) {
  const double eps_ref = kEpsWeno * p.weno_eps_scale;
  // hybrid UD5/UD7 + WENO when a sensor threshold is set (reference src/Parameter.cpp:236-252)
  const double th = p.sensor_threshold;
  const double *sn = th > 1e-10 ? z.shock_sensor : nullptr;
  const bool w7 = p.inviscid_scheme == 72;
  if (dir == 0) return w7 ? launch_dir<0, 7>(z, eps_ref, sn, th, var, st) : launch_dir<0, 5>(z, eps_ref, sn, th, var, st);
  if (dir == 1) return w7 ? launch_dir<1, 7>(z, eps_ref, sn, th, var, st) : launch_dir<1, 5>(z, eps_ref, sn, th, var, st);
  return w7 ? launch_dir<2, 7>(z, eps_ref, sn, th, var, st) : launch_dir<2, 5>(z, eps_ref, sn, th, var, st);
}

// The tile variant of a sweep that was neither tuned nor set.
int weno_air_default_tile(const Dims &d, int dir, int order, int n_sm) {
  return weno_air_tile(d.ext(dir), dir == 0 ? d.my : d.mx, dir == 2 ? d.my : d.mz, dir, order, n_sm);
}

// Host launcher: x, y and (3-D) z sweeps in the reference's order; var[d]
// is the tile variant of sweep d.
cudaError_t launch_weno_air(const Zone &z, const Param &p, const int *var, cudaStream_t st, int *n_launch) {
  const int nd = z.d.mz > 1 ? 3 : 2;
  for (int dir = 0; dir < nd; ++dir) {
    cudaError_t e = launch_weno_air_dir(z, p, dir, var[dir], st);
    if (e != cudaSuccess) return e;
    *n_launch += 1;
  }
  return cudaSuccess;
}

}  // namespace cfk
