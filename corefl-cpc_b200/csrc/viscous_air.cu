// Second-order viscous flux of calorically perfect air, all three directions
// fused, with the flux differences added to dq.
//
// Restates compute_{f,g,h}v_2nd_order (air branch, reference
// src/ViscousScheme.cu:614-1173) and compute_dFv_dx / dGv_dy / dHv_dz
// (reference src/ViscousScheme.cu:75-127).  The staggered face fluxes stay in
// registers and shared memory, so the vis_flux array of the reference never
// reaches HBM, and every node's inputs are read once per stage.
#include "cfk_common.cuh"

namespace cfk {

// All three directions in one kernel: a CTA owns a 32 x 4 tile of (i, j)
// columns and marches along k through a chunk of planes, keeping two planes
// of per-node values (u, v, w, T, mu, J, metric) with a one-node halo in
// shared memory plus the k-differences f(k+1) - f(k-1) of the current plane.
// Per plane it computes the x and y faces of the plane and the z face above
// each node; the z face below comes from the previous plane.  dq gets the x,
// y and z differences added in that order, the order of the reference's
// per-direction derivative kernels (the ring variant adds their sum).  Every node's inputs are read from HBM
// once per stage and dq once instead of three times.
namespace {
constexpr int kFX = 32, kFY = 4;               // tile; the planes of a chunk: viscous_chunk
constexpr int kCtas = 3;                       // CTAs an SM of the ring form
constexpr int kPX = kFX + 2, kPY = kFY + 2;    // staged points per plane
constexpr int kNV = 15;                        // u v w T mu J metric[9]
constexpr int kFT = kFX * kFY;                 // threads
// the flux's constant factors as products: 1/3 of the normal stresses and
// cp / Pr of the conductivity, formed once (the reference divides by 3 and
// by Pr at every face; the results differ in the last bits)
constexpr double kThird = 1.0 / 3.0;
constexpr double kCpAir = kGammaAir * kRAir / (kGammaAir - 1);

struct FusedSmem {
  double pl[2][kNV][kPY][kPX];   // planes k and k+1 (slots swap)
  double dzp[4][kPY][kPX];       // f(k+1) - f(k-1) of u, v, w, T on plane k
  double fx[4][kFY][kFX + 1];    // x faces of plane k
  double fy[4][kFY + 1][kFX];    // y faces of plane k
};

// Face flux between staged points A = (pa, qa) of slot sa and B = (pb, qb)
// of slot sb, normal to DIR (reference src/ViscousScheme.cu:614-700 and the
// g/h analogues), read straight from shared memory: values are fetched where
// they are used so that the two nodes are never held in registers at once.
// The transverse derivative 0.25 (f(A+) - f(A-) + f(B+) - f(B-)) is summed
// as 0.25 ((f(A+) - f(A-)) + (f(B+) - f(B-))).
template <int DIR>
__device__ __forceinline__ void staged_face(const FusedSmem &S, int sa, int pa, int qa, int sb, int pb, int qb,
                                            double cp_pr, double F[4]) {
  const auto &A = S.pl[sa];
  const auto &B = S.pl[sb];
  // transverse difference of variable q at a point along direction D (0 x, 1 y, 2 z)
  auto tdiff = [&](const double (&p)[kNV][kPY][kPX], int D, int q, int px, int py) -> double {
    if (D == 0) return p[q][py][px + 1] - p[q][py][px - 1];
    if (D == 1) return p[q][py + 1][px] - p[q][py - 1][px];
    return S.dzp[q][py][px];
  };
  constexpr int TLO = DIR == 0 ? 1 : 0, THI = DIR == 2 ? 1 : 2;
  double gm[9];
#pragma unroll
  for (int l = 0; l < 9; ++l) gm[l] = 0.5 * (A[6 + l][qa][pa] + B[6 + l][qb][pb]);
  double dd[4][3];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    dd[q][DIR] = B[q][qb][pb] - A[q][qa][pa];
    dd[q][TLO] = 0.25 * (tdiff(A, TLO, q, pa, qa) + tdiff(B, TLO, q, pb, qb));
    dd[q][THI] = 0.25 * (tdiff(A, THI, q, pa, qa) + tdiff(B, THI, q, pb, qb));
  }
  const double u_x = dd[0][0] * gm[0] + dd[0][1] * gm[3] + dd[0][2] * gm[6];
  const double u_y = dd[0][0] * gm[1] + dd[0][1] * gm[4] + dd[0][2] * gm[7];
  const double u_z = dd[0][0] * gm[2] + dd[0][1] * gm[5] + dd[0][2] * gm[8];
  const double v_x = dd[1][0] * gm[0] + dd[1][1] * gm[3] + dd[1][2] * gm[6];
  const double v_y = dd[1][0] * gm[1] + dd[1][1] * gm[4] + dd[1][2] * gm[7];
  const double v_z = dd[1][0] * gm[2] + dd[1][1] * gm[5] + dd[1][2] * gm[8];
  const double w_x = dd[2][0] * gm[0] + dd[2][1] * gm[3] + dd[2][2] * gm[6];
  const double w_y = dd[2][0] * gm[1] + dd[2][1] * gm[4] + dd[2][2] * gm[7];
  const double w_z = dd[2][0] * gm[2] + dd[2][1] * gm[5] + dd[2][2] * gm[8];
  const double t_x = dd[3][0] * gm[0] + dd[3][1] * gm[3] + dd[3][2] * gm[6];
  const double t_y = dd[3][0] * gm[1] + dd[3][1] * gm[4] + dd[3][2] * gm[7];
  const double t_z = dd[3][0] * gm[2] + dd[3][1] * gm[5] + dd[3][2] * gm[8];
  const double mul = 0.5 * (A[4][qa][pa] + B[4][qb][pb]);
  const double tau_xx = mul * (4 * u_x - 2 * v_y - 2 * w_z) * kThird;
  const double tau_yy = mul * (4 * v_y - 2 * u_x - 2 * w_z) * kThird;
  const double tau_zz = mul * (4 * w_z - 2 * u_x - 2 * v_y) * kThird;
  const double tau_xy = mul * (u_y + v_x);
  const double tau_xz = mul * (u_z + w_x);
  const double tau_yz = mul * (v_z + w_y);
  const double ja = A[5][qa][pa], jb = B[5][qb][pb];
  const double gk0 = 0.5 * (A[6 + 3 * DIR][qa][pa] * ja + B[6 + 3 * DIR][qb][pb] * jb);
  const double gk1 = 0.5 * (A[7 + 3 * DIR][qa][pa] * ja + B[7 + 3 * DIR][qb][pb] * jb);
  const double gk2 = 0.5 * (A[8 + 3 * DIR][qa][pa] * ja + B[8 + 3 * DIR][qb][pb] * jb);
  F[0] = gk0 * tau_xx + gk1 * tau_xy + gk2 * tau_xz;
  F[1] = gk0 * tau_xy + gk1 * tau_yy + gk2 * tau_yz;
  F[2] = gk0 * tau_xz + gk1 * tau_yz + gk2 * tau_zz;
  const double um = 0.5 * (A[0][qa][pa] + B[0][qb][pb]);
  const double vm = 0.5 * (A[1][qa][pa] + B[1][qb][pb]);
  const double wm = 0.5 * (A[2][qa][pa] + B[2][qb][pb]);
  const double conductivity = mul * cp_pr;
  F[3] = um * F[0] + vm * F[1] + wm * F[2] + conductivity * (gk0 * t_x + gk1 * t_y + gk2 * t_z);
}
}  // namespace

__global__ void __launch_bounds__(kFT, 2) viscous_air_fused(Zone z, double Pr, int planes) {
  // 152 registers and 65 KB: three CTAs of 128 threads an SM.  Against 32 x 8
  // tiles of two CTAs and chunks of 32 planes: 161 x 113 x 97 271 -> 194 us, 2048
  // x 512 185 -> 145, 40 x 37 x 33 125 -> 15
  extern __shared__ __align__(16) double fsm[];
  const double cp_pr = kCpAir / Pr;
  FusedSmem &S = *reinterpret_cast<FusedSmem *>(fsm);
  const Dims d = z.d;
  const int g = d.ngg;
  const int64_t sz = d.plane(g), szq = d.plane(0);
  const int i0 = blockIdx.x * kFX, j0 = blockIdx.y * kFY, k0 = blockIdx.z * planes;
  const int tx = threadIdx.x % kFX, ty = threadIdx.x / kFX;
  const bool three_d = d.mz > 1;
  const int k_end = min(k0 + planes, d.mz);

  // per-thread share of a plane's staged points: p = threadIdx.x, + kFT
  auto point_ok = [&](int p, int &px, int &py) {
    py = p / kPX;
    px = p - py * kPX;
    return p < kPX * kPY && i0 - 1 + px <= d.mx && j0 - 1 + py <= d.my;
  };
  // the 15 staged values of point (px, py) of plane k into slot sl
  auto load_point = [&](int k, int px, int py, int sl) {
    const int64_t id = d.idx(g, i0 - 1 + px, j0 - 1 + py, k);
    double v[kNV];
    v[0] = z.bv[id + sz];
    v[1] = z.bv[id + 2 * sz];
    v[2] = z.bv[id + 3 * sz];
    v[3] = z.bv[id + 5 * sz];
    v[4] = z.mul[id];
    v[5] = z.jac[id];
#pragma unroll
    for (int l = 0; l < 9; ++l) v[6 + l] = z.metric[id + l * sz];
#pragma unroll
    for (int q = 0; q < kNV; ++q) S.pl[sl][q][py][px] = v[q];
  };

  // planes k0-1 (slot 0) and k0 (slot 1); the z face k0-1/2 between them
  for (int sl = 0; sl < 2; ++sl)
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      int px, py;
      if (point_ok(threadIdx.x + r * kFT, px, py)) load_point(k0 - 1 + sl, px, py, sl);
    }
  __syncthreads();
  const int i = i0 + tx, j = j0 + ty;
  const bool mine = i < d.mx && j < d.my;
  double fzp[4] = {0, 0, 0, 0};
  if (three_d && mine) {
    staged_face<2>(S, 0, tx + 1, ty + 1, 1, tx + 1, ty + 1, cp_pr, fzp);
  }
  // the first iteration refills slot 0, which the z faces above read at
  // neighbouring points
  __syncthreads();
  int cur = 1;  // slot of plane k
  for (int k = k0; k < k_end; ++k) {
    const int nxt = cur ^ 1;  // holds plane k-1, receives plane k+1
    // dq of this node for plane k: loaded now, used after the faces
    double acc[4];
    const int64_t iq = d.idx(0, i, j, k);
    if (mine) {
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[q] = z.dq[iq + (q + 1) * szq];
    }
    // plane k+1 replaces plane k-1 point by point: every point is read and
    // written by the thread that loads it, so the k-differences
    // f(k+1) - f(k-1) of u, v, w, T come from the old slot value before the
    // new one overwrites it, with no barrier between the two
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      int px, py;
      if (!point_ok(threadIdx.x + r * kFT, px, py)) continue;
      const int64_t id = d.idx(g, i0 - 1 + px, j0 - 1 + py, k + 1);
      double v[kNV];
      v[0] = z.bv[id + sz];
      v[1] = z.bv[id + 2 * sz];
      v[2] = z.bv[id + 3 * sz];
      v[3] = z.bv[id + 5 * sz];
      v[4] = z.mul[id];
      v[5] = z.jac[id];
#pragma unroll
      for (int l = 0; l < 9; ++l) v[6 + l] = z.metric[id + l * sz];
#pragma unroll
      for (int q = 0; q < 4; ++q) S.dzp[q][py][px] = v[q] - S.pl[nxt][q][py][px];
#pragma unroll
      for (int q = 0; q < kNV; ++q) S.pl[nxt][q][py][px] = v[q];
    }
    __syncthreads();
    // x faces (33 per row) and y faces (9 per column) of plane k as one work
    // list, the y part starting on a warp boundary, so that the faces beyond
    // one per thread spread over two warps instead of piling onto the first
    constexpr int kNXF = kFY * (kFX + 1), kNYF = (kFY + 1) * kFX;
    constexpr int kYF0 = (kNXF + 31) / 32 * 32;
    for (int f = threadIdx.x; f < kYF0 + kNYF; f += kFT) {
      if (f < kYF0) {
        if (f >= kNXF) continue;
        const int fy_ = f / (kFX + 1), fx_ = f - fy_ * (kFX + 1);
        if (i0 - 1 + fx_ > d.mx - 1 || j0 + fy_ >= d.my) continue;
        double F[4];
        staged_face<0>(S, cur, fx_, fy_ + 1, cur, fx_ + 1, fy_ + 1, cp_pr, F);
#pragma unroll
        for (int q = 0; q < 4; ++q) S.fx[q][fy_][fx_] = F[q];
      } else {
        const int e = f - kYF0;
        const int fy_ = e / kFX, fx_ = e - fy_ * kFX;
        if (i0 + fx_ >= d.mx || j0 - 1 + fy_ > d.my - 1) continue;
        double F[4];
        staged_face<1>(S, cur, fx_ + 1, fy_, cur, fx_ + 1, fy_ + 1, cp_pr, F);
#pragma unroll
        for (int q = 0; q < 4; ++q) S.fy[q][fy_][fx_] = F[q];
      }
    }
    double fzn[4] = {0, 0, 0, 0};
    if (three_d && mine) {
      staged_face<2>(S, cur, tx + 1, ty + 1, nxt, tx + 1, ty + 1, cp_pr, fzn);
    }
    __syncthreads();
    if (mine) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        double a = acc[q];
        a += S.fx[q][ty][tx + 1] - S.fx[q][ty][tx];
        a += S.fy[q][ty + 1][tx] - S.fy[q][ty][tx];
        if (three_d) a += fzn[q] - fzp[q];
        z.dq[iq + (q + 1) * szq] = a;
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) fzp[q] = fzn[q];
    cur = nxt;
  }
}

// Ring variant: the same tile and march, with only the dynamic
// values (u, v, w, T, mu) staged in shared memory, in a ring of three plane
// slots filled by cp.async: plane k+2 is requested before the faces of plane
// k are computed and lands while they run, so the loads never stall a warp.
// The metric and J (read-only) come from global memory into registers.  41 KB
// of shared memory per CTA, two barriers per plane.  The face flux is term for
// term that of staged_face, and the three differences are summed before they
// are added to dq, so the two agree to the last bits.
namespace {
constexpr int kRV = 5;  // u v w T mu

struct RingSmem {
  double dyn[3][kRV][kPY][kPX];  // planes k-1, k, k+1 (slots rotate; one is refilled with k+2)
  double dzp[4][kPY][kPX];       // f(k+1) - f(k-1) of u, v, w, T on plane k
  double fx[4][kFY][kFX + 1];
  double fy[4][kFY + 1][kFX];
};

__device__ __forceinline__ void cp_async8(double *dst, const double *src) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(src) : "memory");
}
__device__ __forceinline__ void prefetch_l2(const double *p) {
  asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// staged_face with the metric [0..8] and J [9] of the two nodes in registers.
template <int DIR>
__device__ __forceinline__ void ring_face(const RingSmem &S, int sa, int pa, int qa, const double (&ma)[10], int sb,
                                          int pb, int qb, const double (&mb)[10], double cp_pr, double (&F)[4]) {
  const auto &A = S.dyn[sa];
  const auto &B = S.dyn[sb];
  auto tdiff = [&](const double (&p)[kRV][kPY][kPX], int D, int q, int px, int py) -> double {
    if (D == 0) return p[q][py][px + 1] - p[q][py][px - 1];
    if (D == 1) return p[q][py + 1][px] - p[q][py - 1][px];
    return S.dzp[q][py][px];
  };
  constexpr int TLO = DIR == 0 ? 1 : 0, THI = DIR == 2 ? 1 : 2;
  double gm[9];
#pragma unroll
  for (int l = 0; l < 9; ++l) gm[l] = 0.5 * (ma[l] + mb[l]);
  double dd[4][3];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    dd[q][DIR] = B[q][qb][pb] - A[q][qa][pa];
    dd[q][TLO] = 0.25 * (tdiff(A, TLO, q, pa, qa) + tdiff(B, TLO, q, pb, qb));
    dd[q][THI] = 0.25 * (tdiff(A, THI, q, pa, qa) + tdiff(B, THI, q, pb, qb));
  }
  const double u_x = dd[0][0] * gm[0] + dd[0][1] * gm[3] + dd[0][2] * gm[6];
  const double u_y = dd[0][0] * gm[1] + dd[0][1] * gm[4] + dd[0][2] * gm[7];
  const double u_z = dd[0][0] * gm[2] + dd[0][1] * gm[5] + dd[0][2] * gm[8];
  const double v_x = dd[1][0] * gm[0] + dd[1][1] * gm[3] + dd[1][2] * gm[6];
  const double v_y = dd[1][0] * gm[1] + dd[1][1] * gm[4] + dd[1][2] * gm[7];
  const double v_z = dd[1][0] * gm[2] + dd[1][1] * gm[5] + dd[1][2] * gm[8];
  const double w_x = dd[2][0] * gm[0] + dd[2][1] * gm[3] + dd[2][2] * gm[6];
  const double w_y = dd[2][0] * gm[1] + dd[2][1] * gm[4] + dd[2][2] * gm[7];
  const double w_z = dd[2][0] * gm[2] + dd[2][1] * gm[5] + dd[2][2] * gm[8];
  const double t_x = dd[3][0] * gm[0] + dd[3][1] * gm[3] + dd[3][2] * gm[6];
  const double t_y = dd[3][0] * gm[1] + dd[3][1] * gm[4] + dd[3][2] * gm[7];
  const double t_z = dd[3][0] * gm[2] + dd[3][1] * gm[5] + dd[3][2] * gm[8];
  const double mul = 0.5 * (A[4][qa][pa] + B[4][qb][pb]);
  const double tau_xx = mul * (4 * u_x - 2 * v_y - 2 * w_z) * kThird;
  const double tau_yy = mul * (4 * v_y - 2 * u_x - 2 * w_z) * kThird;
  const double tau_zz = mul * (4 * w_z - 2 * u_x - 2 * v_y) * kThird;
  const double tau_xy = mul * (u_y + v_x);
  const double tau_xz = mul * (u_z + w_x);
  const double tau_yz = mul * (v_z + w_y);
  const double gk0 = 0.5 * (ma[3 * DIR] * ma[9] + mb[3 * DIR] * mb[9]);
  const double gk1 = 0.5 * (ma[3 * DIR + 1] * ma[9] + mb[3 * DIR + 1] * mb[9]);
  const double gk2 = 0.5 * (ma[3 * DIR + 2] * ma[9] + mb[3 * DIR + 2] * mb[9]);
  F[0] = gk0 * tau_xx + gk1 * tau_xy + gk2 * tau_xz;
  F[1] = gk0 * tau_xy + gk1 * tau_yy + gk2 * tau_yz;
  F[2] = gk0 * tau_xz + gk1 * tau_yz + gk2 * tau_zz;
  const double um = 0.5 * (A[0][qa][pa] + B[0][qb][pb]);
  const double vm = 0.5 * (A[1][qa][pa] + B[1][qb][pb]);
  const double wm = 0.5 * (A[2][qa][pa] + B[2][qb][pb]);
  const double conductivity = mul * cp_pr;
  F[3] = um * F[0] + vm * F[1] + wm * F[2] + conductivity * (gk0 * t_x + gk1 * t_y + gk2 * t_z);
}
}  // namespace

// MINB: CTAs per SM the register budget is sized for.  PF: with the request of
// plane k+2's dynamic values, also ask L2 for its metric and J, so that the
// faces' reads of them no longer wait on DRAM.
//
// Bound by the L1 and shared-memory pipe and by the barriers of a plane.  A
// thread holds its node's metric and J in registers for its lower x and y faces
// and both its z faces and reads its neighbours' once (30 loads a plane instead
// of some 60).  145 x 130 x 99 (us): faces shared out with every metric read
// from L1 234; the same 32 x 8 tile with the metric held 212; 32 x 4, 128
// threads, four CTAs of 128 registers 180, three of 158 registers 181, which is
// the faster on large blocks (257^3 step 29.02, 28.68 ms).
template <int MINB, bool PF>
__global__ void __launch_bounds__(kFT, MINB) viscous_air_ring(Zone z, double Pr, int planes) {
  extern __shared__ __align__(16) double rsm[];
  const double cp_pr = kCpAir / Pr;
  RingSmem &S = *reinterpret_cast<RingSmem *>(rsm);
  const Dims d = z.d;
  const int g = d.ngg;
  const int64_t sz = d.plane(g), szq = d.plane(0);
  const int64_t srow = d.stride(g, 1), spl = d.stride(g, 2);
  const int i0 = blockIdx.x * kFX, j0 = blockIdx.y * kFY, k0 = blockIdx.z * planes;
  const int tx = threadIdx.x % kFX, ty = threadIdx.x / kFX;
  const bool three_d = d.mz > 1;
  const int k_end = min(k0 + planes, d.mz);
  const double *__restrict__ met = z.metric;
  const double *__restrict__ jac = z.jac;

  auto point_ok = [&](int p, int &px, int &py) {
    py = p / kPX;
    px = p - py * kPX;
    return p < kPX * kPY && i0 - 1 + px <= d.mx && j0 - 1 + py <= d.my;
  };
  // this thread's points of plane k into slot sl (the same points every plane)
  auto request = [&](int k, int sl) {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      int px, py;
      if (!point_ok(threadIdx.x + r * kFT, px, py)) continue;
      const int64_t id = d.idx(g, i0 - 1 + px, j0 - 1 + py, k);
      cp_async8(&S.dyn[sl][0][py][px], z.bv + id + sz);
      cp_async8(&S.dyn[sl][1][py][px], z.bv + id + 2 * sz);
      cp_async8(&S.dyn[sl][2][py][px], z.bv + id + 3 * sz);
      cp_async8(&S.dyn[sl][3][py][px], z.bv + id + 5 * sz);
      cp_async8(&S.dyn[sl][4][py][px], z.mul + id);
    }
  };
  request(k0 - 1, 0);
  request(k0, 1);
  request(k0 + 1, 2);
  cp_async_commit();
  const int i = i0 + tx, j = j0 + ty;
  const bool mine = i < d.mx && j < d.my;
  // the lower x and y faces of the node, also where it is the first beyond the block
  const bool face_x = i <= d.mx && j < d.my, face_y = i < d.mx && j <= d.my;
  auto load_m = [&](int64_t id, double (&m)[10]) {
#pragma unroll
    for (int l = 0; l < 9; ++l) m[l] = __ldg(met + id + l * sz);
    m[9] = __ldg(jac + id);
  };
  // metric and J of this thread's node on plane k: read once, used by its
  // three faces and by the z face of the next plane
  double mc[10];
  const int64_t id0 = d.idx(g, min(i, d.mx), min(j, d.my), k0);
  load_m(id0, mc);
  cp_async_wait_all();
  __syncthreads();
  double fzp[4] = {0, 0, 0, 0};
  if (three_d && mine) {
    double mb[10];
    load_m(id0 - spl, mb);
    ring_face<2>(S, 0, tx + 1, ty + 1, mb, 1, tx + 1, ty + 1, mc, cp_pr, fzp);
  }
  // the first iteration refills slot 0, which the z faces above read at
  // neighbouring points
  __syncthreads();
  int sp = 0, sc = 1, sn = 2;  // slots of planes k-1, k, k+1
  for (int k = k0; k < k_end; ++k) {
    const int64_t id = id0 + (k - k0) * spl;
    // k-differences at this thread's points: its own copies of planes k-1
    // and k+1 are complete, and no other thread reads these points of
    // slot sp before the next barrier
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      int px, py;
      if (!point_ok(threadIdx.x + r * kFT, px, py)) continue;
#pragma unroll
      for (int q = 0; q < 4; ++q) S.dzp[q][py][px] = S.dyn[sn][q][py][px] - S.dyn[sp][q][py][px];
    }
    if (k + 2 <= k_end) request(k + 2, sp);  // plane k+2 into the slot of plane k-1
    if (PF && k + 2 <= k_end && face_x) {
#pragma unroll
      for (int m = 0; m < 9; ++m) prefetch_l2(met + id + 2 * spl + m * sz);
      prefetch_l2(jac + id + 2 * spl);
    }
    cp_async_commit();
    __syncthreads();
    double fx[4], fy[4];
    if (face_x) {
      double ma[10];
      load_m(id - 1, ma);
      ring_face<0>(S, sc, tx, ty + 1, ma, sc, tx + 1, ty + 1, mc, cp_pr, fx);
#pragma unroll
      for (int q = 0; q < 4; ++q) S.fx[q][ty][tx] = fx[q];
    }
    if (face_y) {
      double ma[10];
      load_m(id - srow, ma);
      ring_face<1>(S, sc, tx + 1, ty, ma, sc, tx + 1, ty + 1, mc, cp_pr, fy);
#pragma unroll
      for (int q = 0; q < 4; ++q) S.fy[q][ty][tx] = fy[q];
    }
    // the tile's last y faces and last x faces: a warp each, another one on every plane
    if (ty == (k & (kFY - 1))) {
      if (i < d.mx && j0 + kFY <= d.my) {
        double ma[10], mb[10], F[4];
        const int64_t ida = d.idx(g, i, j0 + kFY - 1, k);
        load_m(ida, ma);
        load_m(ida + srow, mb);
        ring_face<1>(S, sc, tx + 1, kFY, ma, sc, tx + 1, kFY + 1, mb, cp_pr, F);
#pragma unroll
        for (int q = 0; q < 4; ++q) S.fy[q][kFY][tx] = F[q];
      }
    } else if (ty == ((k + kFY / 2) & (kFY - 1)) && tx < kFY) {
      if (j0 + tx < d.my && i0 + kFX <= d.mx) {
        double ma[10], mb[10], F[4];
        const int64_t ida = d.idx(g, i0 + kFX - 1, j0 + tx, k);
        load_m(ida, ma);
        load_m(ida + 1, mb);
        ring_face<0>(S, sc, kFX, tx + 1, ma, sc, kFX + 1, tx + 1, mb, cp_pr, F);
#pragma unroll
        for (int q = 0; q < 4; ++q) S.fx[q][tx][kFX] = F[q];
      }
    }
    double fzn[4] = {0, 0, 0, 0};
    if (three_d) {
      double mn[10];
      load_m(id + spl, mn);
      if (mine) ring_face<2>(S, sc, tx + 1, ty + 1, mc, sn, tx + 1, ty + 1, mn, cp_pr, fzn);
#pragma unroll
      for (int l = 0; l < 10; ++l) mc[l] = mn[l];
    }
    cp_async_wait_all();
    __syncthreads();
    if (mine) {
      // the differences in x, y, z order; one addition to dq
      const int64_t iq = d.idx(0, i, j, k);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        double a = S.fx[q][ty][tx + 1] - fx[q];
        a += S.fy[q][ty + 1][tx] - fy[q];
        if (three_d) a += fzn[q] - fzp[q];
        red_add(z.dq + iq + (q + 1) * szq, a);
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) fzp[q] = fzn[q];
    const int t = sp;
    sp = sc;
    sc = sn;
    sn = t;
  }
}

// Opt the kernels in to their dynamic shared-memory sizes.
cudaError_t viscous_air_init_attributes() {
  cudaError_t e = cudaFuncSetAttribute(viscous_air_fused, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)sizeof(FusedSmem));
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(viscous_air_ring<kCtas, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)sizeof(RingSmem));
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(viscous_air_ring<kCtas, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)sizeof(RingSmem));
}

// Planes a CTA marches through: of all equal cuts of the block along k, the one
// with the fewest plane steps in its last CTA to finish, waves of kCtas CTAs
// an SM times a chunk's planes and the two that its start costs.  With 32 planes
// always, small blocks were a handful of CTAs (us: 40 x 37 x 33 137, 22 with the
// chunks cut to fit; 64 x 257 x 20 96, 45; 90 x 80 x 70 150, 66).
int viscous_chunk(long long tiles, int mz, int n_sm) {
  long long best = -1;
  int planes = mz;
  for (int c = 1; c <= mz; ++c) {
    const int len = (mz + c - 1) / c;
    if (c > 1 && len == (mz + c - 2) / (c - 1)) continue;  // the same chunks with an empty one
    const long long cost = (tiles * c + (long long)kCtas * n_sm - 1) / ((long long)kCtas * n_sm) * (len + 2);
    if (best < 0 || cost < best) {
      best = cost;
      planes = len;
    }
  }
  return planes;
}

// compute_viscous_flux for air (reference src/ViscousScheme.cu:7-40): one
// launch for all directions; var 0 the staged kernel, 1 the ring kernel,
// 2 the ring kernel with the L2 prefetch of the metric two planes ahead.
cudaError_t launch_viscous_air(const Zone &z, const Param &p, cudaStream_t st, int *n_launch, int var, int n_sm) {
  const Dims &d = z.d;
  dim3 grid((d.mx + kFX - 1) / kFX, (d.my + kFY - 1) / kFY);
  const int planes = viscous_chunk((long long)grid.x * grid.y, d.mz, n_sm);
  grid.z = (d.mz + planes - 1) / planes;
  if (var == 1) viscous_air_ring<kCtas, false><<<grid, kFT, sizeof(RingSmem), st>>>(z, p.Pr, planes);
  else if (var == 2) viscous_air_ring<kCtas, true><<<grid, kFT, sizeof(RingSmem), st>>>(z, p.Pr, planes);
  else viscous_air_fused<<<grid, kFT, sizeof(FusedSmem), st>>>(z, p.Pr, planes);
  *n_launch += 1;
  return cudaGetLastError();
}

}  // namespace cfk
