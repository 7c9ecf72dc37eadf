// Semi-implicit viscous scheme of the IO section (visthemflg = 1): the
// viscous terms split into an explicit part, a part treated by
// Crank-Nicolson factors and its density correction; then the factored
// variable-coefficient solves (1 - A_x)(1 - A_z)(1 - A_y) dG = RHS_io.
//
// Restates (paths relative to the CHAPSim1WW project root), channel branches:
//   VISCOUS_PAR_EXPLT_X/Y/Z_io  src/VISCOUS_X_EXPLICIT_io.f90:124-286,
//                           src/VISCOUS_Y_EXPLICIT_io.f90:264-424,
//                           src/VISCOUS_Z_EXPLICIT_io.f90:289-460
//   RHS_MOM_EXPLICIT_io     src/RHS_MOM_EXPLICIT_io.f90:79-95 (implicit branch)
//   MOMFA_io, MOMFA1_X_io, MOMFA2_Z_io, MOMFA3_Y_io  src/MOMFA_io.f90:17-377
//   TDMAIJI_CYC, TDMAIJJ_nonCYC  src/TDMAIJI_CYC.f90:67-157,
//                           src/TDMAIJJ_nonCYC.f90:67-123
//   DENSITY_implicit_add    src/MASSFLUX_CALC_IO.f90:316-399 (in k_io_prep)
//
// The three components' right-hand sides are formed by one kernel before any
// solve: VISCOUS_PAR_EXPLT_*_io and RHS_MOM_EXPLICIT_io of component c read
// Q_io, the convection terms (all formed first by the reference too), the
// pressure and G_io component c only, and MOMFA_io(c) changes G_io component
// c only, so the reference's interleaved order gives the same values.
//
// Line solves: one warp per line with the line in shared memory
// (warp_part_solve: chunked elimination, then parallel cyclic reduction of
// the chunk-end system over shuffles), staged by coalesced loads: x lines are
// rows, z and y lines come in tiles of consecutive x.  The coefficients are
// formed from VISCOUSITY and the MU_STG / RHO_STG fields k_si_stg forms once
// per substep (as MU_Staggered and DENSITY_Staggered do).  Nothing but the
// right-hand sides and the result crosses global memory.
#include <cuda_runtime.h>

#include <string>

#include "chapsim_internal.cuh"
#include "tma.cuh"

#define LAUNCHED()                                                        \
  do {                                                                    \
    ++c->launches;                                                        \
    cudaError_t e_ = cudaGetLastError();                                  \
    if (e_ != cudaSuccess) {                                              \
      c->err = std::string("kernel launch: ") + cudaGetErrorString(e_);   \
      return CHAPSIM_ERR_CUDA;                                            \
    }                                                                     \
  } while (0)

namespace chapsim {
namespace {

constexpr int SI_BX = 32, SI_BY = 8;

__device__ __forceinline__ int wp(int i, int n) { return i + 1 == n ? 0 : i + 1; }
__device__ __forceinline__ int wm(int i, int n) { return i == 0 ? n - 1 : i - 1; }

// MU_Staggered and DENSITY_Staggered (src/MASSFLUX_CALC_IO.f90:147-311) at
// (i, j, k), periodic in i and k, formed from mu, mu0, rho, rho0.
struct StgForm {
  const double *__restrict__ mu;
  const double *__restrict__ mu0;
  const double *__restrict__ D;
  const double *__restrict__ D0;
  const double *__restrict__ wff;
  const double *__restrict__ wfb;
  int nx, ny, nz;
  int64_t sy, sz;
  __device__ __forceinline__ int64_t at(int i, int j, int k) const { return (int64_t)i + sy * j + sz * k; }
  // x-face / y-face edge; wall rows 1 and ny+1 from the ghost cells
  __device__ __forceinline__ double s1(int i, int j, int k) const {
    const int64_t c = at(i, j, k), m = at(wm(i, nx), j, k);
    if (j == 1) return 0.5 * (mu0[c - sy] + mu[c - sy]);
    if (j == ny + 1) return 0.5 * (mu0[c] + mu[c]);
    return ((mu[c] + mu[m] + mu0[c] + mu0[m]) * wff[j] + (mu[c - sy] + mu[m - sy] + mu0[c - sy] + mu0[m - sy]) * wfb[j]) *
           0.5 * 0.5;
  }
  // x-face / z-face edge
  __device__ __forceinline__ double s2(int i, int j, int k) const {
    const int im = wm(i, nx), km = wm(k, nz);
    const int64_t c = at(i, j, k), cx = at(im, j, k), cz = at(i, j, km), cxz = at(im, j, km);
    return (mu[c] + mu[cx] + mu0[c] + mu0[cx] + mu[cz] + mu[cxz] + mu0[cz] + mu0[cxz]) * 0.5 * 0.5 * 0.5;
  }
  // y-face / z-face edge; wall rows from the ghost cells
  __device__ __forceinline__ double s3(int i, int j, int k) const {
    const int64_t c = at(i, j, k), m = at(i, j, wm(k, nz));
    if (j == 1) return 0.5 * (mu0[c - sy] + mu[c - sy]);
    if (j == ny + 1) return 0.5 * (mu0[c] + mu[c]);
    return ((mu[m] + mu[c] + mu0[m] + mu0[c]) * wff[j] + (mu[m - sy] + mu[c - sy] + mu0[m - sy] + mu0[c - sy]) * wfb[j]) *
           0.5 * 0.5;
  }
  __device__ __forceinline__ double r1(int i, int j, int k) const {
    const int64_t c = at(i, j, k), m = at(wm(i, nx), j, k);
    return (D[c] + D[m] + D0[c] + D0[m]) * 0.5 * 0.5;
  }
  // v faces: row 0 keeps the allocation value 1 (never formed by
  // DENSITY_Staggered), rows 1 and ny+1 from the ghost cells
  __device__ __forceinline__ double r2(int i, int j, int k) const {
    if (j == 0) return 1.0;
    const int64_t c = at(i, j, k);
    if (j == 1) return 0.5 * (D0[c - sy] + D[c - sy]);
    if (j == ny + 1) return 0.5 * (D0[c] + D[c]);
    return (wff[j] * (D[c] + D0[c]) + wfb[j] * (D[c - sy] + D0[c - sy])) * 0.5;
  }
  __device__ __forceinline__ double r3(int i, int j, int k) const {
    const int64_t c = at(i, j, k), m = at(i, j, wm(k, nz));
    return (D[c] + D[m] + D0[c] + D0[m]) * 0.5 * 0.5;
  }
};

// MU_STG 1-3 and 1 / RHO_STG 1-3 of the substep into io.stg, once, for the
// right-hand sides and the factor solves: rows 0..ny+1 of the faces that
// have them (s1, s3: 1..ny+1; s2, r1, r3: 1..ny; r2: 0..ny+1).  The solves
// divide by RHO_STG 27 times per cell: three reciprocals here, products there.
__global__ void __launch_bounds__(SI_BX *SI_BY) k_si_stg(TGDev d, IODev io) {
  const int i = blockIdx.x * SI_BX + threadIdx.x;
  const int j = blockIdx.y * SI_BY + threadIdx.y;  // 0..ny+1
  const int k = blockIdx.z;
  if (i >= d.nx || j > d.ny + 1) return;
  const StgForm F{io.mu, io.mu0, io.D, io.D0, d.wff, d.wfb, d.nx, d.ny, d.nz, d.sy, d.sz};
  const int64_t c = F.at(i, j, k);
  if (j >= 1) {
    io.stg[0][c] = F.s1(i, j, k);
    io.stg[2][c] = F.s3(i, j, k);
  }
  if (j >= 1 && j <= d.ny) {
    io.stg[1][c] = F.s2(i, j, k);
    io.stg[3][c] = 1.0 / F.r1(i, j, k);
    io.stg[5][c] = 1.0 / F.r3(i, j, k);
  }
  io.stg[4][c] = 1.0 / F.r2(i, j, k);
}

// VISCOUSITY, MU_STG(1..3) and 1 / RHO_STG(1..3) at (i, j, k) from the fields
// k_si_stg formed; with the energy equation off all of them are 1.
struct Prop {
  const double *__restrict__ mu;
  const double *__restrict__ st1;
  const double *__restrict__ st2;
  const double *__restrict__ st3;
  const double *__restrict__ rs1;
  const double *__restrict__ rs2;
  const double *__restrict__ rs3;
  int nx, ny, nz, th;
  int64_t sy, sz;
  __device__ __forceinline__ int64_t at(int i, int j, int k) const { return (int64_t)i + sy * j + sz * k; }
  __device__ __forceinline__ double vis(int i, int j, int k) const { return th ? mu[at(i, j, k)] : 1.0; }
  __device__ __forceinline__ double s1(int i, int j, int k) const { return th ? st1[at(i, j, k)] : 1.0; }
  __device__ __forceinline__ double s2(int i, int j, int k) const { return th ? st2[at(i, j, k)] : 1.0; }
  __device__ __forceinline__ double s3(int i, int j, int k) const { return th ? st3[at(i, j, k)] : 1.0; }
  __device__ __forceinline__ double ri1(int i, int j, int k) const { return th ? rs1[at(i, j, k)] : 1.0; }
  __device__ __forceinline__ double ri2(int i, int j, int k) const { return th ? rs2[at(i, j, k)] : 1.0; }
  __device__ __forceinline__ double ri3(int i, int j, int k) const { return th ? rs3[at(i, j, k)] : 1.0; }
};

__device__ __forceinline__ Prop make_prop(const TGDev &d, const IODev &io) {
  return Prop{io.mu, io.stg[0], io.stg[1], io.stg[2], io.stg[3], io.stg[4], io.stg[5],
              d.nx, d.ny, d.nz, io.thermal, d.sy, d.sz};
}

// Convection (CONVECTION_*_io), the split viscous terms (VISCOUS_PAR_EXPLT_*_io)
// and RHS_MOM_EXPLICIT_io's implicit branch for component C of one cell
// (one launch per component): RHS_io -> d.rhs[C], EXPLT0_io updated.  Per-block sums of RHS_x / DYFI
// feed DPGRNS.  Row 1 of the v right-hand side is zero (VISCOUS_PAR_EXPLT_Y_io
// clears RHS_io and nothing writes that row before MOMFA3_Y_io).
template <int C, bool TH>
__global__ void __launch_bounds__(SI_BX *SI_BY, 4) k_io_rhs_si(TGDev d, IODev io, double gam, double roh, double alp,
                                                          int cur) {
  __shared__ double red[SI_BX * SI_BY / 32];
  const int nx = d.nx, ny = d.ny, nz = d.nz;
  const int i = blockIdx.x * SI_BX + threadIdx.x;
  const int j = blockIdx.y * SI_BY + threadIdx.y + 1;
  const int k = blockIdx.z;
  double part = 0.0;
  if (i < nx && j <= ny) {
    const int64_t sy = d.sy, sz = d.sz;
    const int ip = wp(i, nx), im = wm(i, nx), kp = wp(k, nz), km = wm(k, nz);
    Prop P = make_prop(d, io);
    P.th = TH;  // compile-time: the property loads and density parts fold away without the energy equation
    constexpr bool th = TH;
    const double *__restrict__ u = d.u, *__restrict__ v = d.v, *__restrict__ w = d.w, *__restrict__ p = d.p;
    const double *__restrict__ gx = io.g[cur][0], *__restrict__ gy = io.g[cur][1], *__restrict__ gz = io.g[cur][2];
    const double *__restrict__ r0 = io.drhoi[0], *__restrict__ r1 = io.drhoi[1], *__restrict__ r2 = io.drhoi[2];
    auto A = [&](const double *f, int ii, int jj, int kk) { return f[(int64_t)ii + sy * jj + sz * kk]; };
    // G_io * DRHOI_STG (and Q_io * DRHOI_STG where the reference writes it)
    auto AD = [&](const double *f, const double *r, int ii, int jj, int kk) {
      const int64_t q = (int64_t)ii + sy * jj + sz * kk;
      return f[q] * r[q];
    };
    const int64_t c = (int64_t)i + sy * j + sz * k;
    const double dxi = d.dxi, dzi = d.dzi, cv = d.cvisc, dt = d.dt, coe2a = alp * dt;
    const double dyfj = d.dyfi[j], dycj = d.dyci[j], dycp = d.dyci[j + 1];
    const double wff = d.wff[j], wfb = d.wfb[j], wffp = d.wff[j + 1], wfbp = d.wfb[j + 1];
    const int64_t oxp = ip - i, oxm = im - i, ozp = sz * (kp - k), ozm = sz * (km - k);
    // ------------------------------------------------ x
    if (C == 0) {
      const double h11 = ((gx[c + oxp] + gx[c]) * (u[c + oxp] + u[c]) - (gx[c] + gx[c + oxm]) * (u[c] + u[c + oxm])) *
                         (dxi * 0.5 * 0.5);
      const double h12 = ((gy[c + sy] + gy[c + sy + oxm]) * (wffp * u[c + sy] + wfbp * u[c]) -
                          (gy[c] + gy[c + oxm]) * (wff * u[c] + wfb * u[c - sy])) * (dyfj * 0.5);
      const double h13 = ((gz[c + ozp] + gz[c + ozp + oxm]) * (u[c + ozp] + u[c]) -
                          (gz[c] + gz[c + oxm]) * (u[c] + u[c + ozm])) * (dzi * 0.5 * 0.5);
      const double conv = -(h11 + h12 + h13);
      const double coe1 = -2.0 / 3.0 * dxi * cv, coe2 = dyfj * cv, coe32 = dzi * cv;
      const double muc = P.vis(i, j, k), mum = P.vis(im, j, k);
      double dudx = (A(u, ip, j, k) - A(u, i, j, k)) * dxi;
      double dvdy = (A(v, i, j + 1, k) - A(v, i, j, k)) * dyfj;
      double dwdz = (A(w, i, j, kp) - A(w, i, j, k)) * dzi;
      const double t11fe = muc * (dvdy + dwdz), t11fi = muc * dudx;
      const double t11fa = th ? muc * ((AD(gx, r0, ip, j, k) - AD(gx, r0, i, j, k)) * dxi) : 0.0;
      dudx = (A(u, i, j, k) - A(u, im, j, k)) * dxi;
      dvdy = (A(v, im, j + 1, k) - A(v, im, j, k)) * dyfj;
      dwdz = (A(w, im, j, kp) - A(w, im, j, k)) * dzi;
      const double t11be = mum * (dvdy + dwdz), t11bi = mum * dudx;
      const double t11ba = th ? mum * ((AD(gx, r0, i, j, k) - AD(gx, r0, im, j, k)) * dxi) : 0.0;
      const double d11e = (t11fe - t11be) * coe1, d11i = (t11fi - t11bi) * coe1 * (-2.0);
      const double d11a = (t11fa - t11ba) * coe1 * (-2.0);
      const double vis12p = P.s1(i, j + 1, k), vis12c = P.s1(i, j, k);
      double dvdx = (A(v, i, j + 1, k) - A(v, im, j + 1, k)) * dxi;
      double dudy = (A(u, i, j + 1, k) - A(u, i, j, k)) * dycp;
      const double t12fe = vis12p * dvdx, t12fi = vis12p * dudy;
      const double t12fa = th ? vis12p * ((AD(gx, r0, i, j + 1, k) - AD(gx, r0, i, j, k)) * dycp) : 0.0;
      dudy = (A(u, i, j, k) - A(u, i, j - 1, k)) * dycj;
      dvdx = (A(v, i, j, k) - A(v, im, j, k)) * dxi;
      const double t12be = vis12c * dvdx, t12bi = vis12c * dudy;
      const double t12ba = th ? vis12c * ((AD(gx, r0, i, j, k) - AD(gx, r0, i, j - 1, k)) * dycj) : 0.0;
      const double d12e = (t12fe - t12be) * coe2, d12i = (t12fi - t12bi) * coe2, d12a = (t12fa - t12ba) * coe2;
      const double vis13p = P.s2(i, j, kp), vis13c = P.s2(i, j, k);
      double dudz = (A(u, i, j, kp) - A(u, i, j, k)) * dzi;
      double dwdx = (A(w, i, j, kp) - A(w, im, j, kp)) * dxi;
      const double t13fe = vis13p * dwdx, t13fi = vis13p * dudz;
      // the density part of tau13 differences Q_io, as the reference writes it
      const double t13fa = th ? vis13p * ((AD(u, r0, i, j, kp) - AD(u, r0, i, j, k)) * dzi) : 0.0;
      dudz = (A(u, i, j, k) - A(u, i, j, km)) * dzi;
      dwdx = (A(w, i, j, k) - A(w, im, j, k)) * dxi;
      const double t13be = vis13c * dwdx, t13bi = vis13c * dudz;
      const double t13ba = th ? vis13c * ((AD(u, r0, i, j, k) - AD(u, r0, i, j, km)) * dzi) : 0.0;
      const double d13e = (t13fe - t13be) * coe32, d13i = (t13fi - t13bi) * coe32, d13a = (t13fa - t13ba) * coe32;
      const double explt = (d11e + d12e + d13e) + conv;
      const double imp = d11i + d12i + d13i, adv = d11a + d12a + d13a;
      double *e0 = (double *)d.h0[0];
      double r = (gam * explt + roh * e0[c]) * dt;
      r = r + coe2a * imp + 0.5 * coe2a * adv;
      e0[c] = explt;
      r -= (p[c] - p[c + oxm]) * (alp * dt * dxi);
      if (io.gravdir == 1) r += (alp * dt * io.f_a) / P.ri1(i, j, k);
      part = r / dyfj;
      ((double *)d.rhs[0])[c] = r;
    }
    // ------------------------------------------------ y (rows 2..ny)
    if (C == 1 && j >= 2) {
      const double h21 = ((wff * gx[c + oxp] + wfb * gx[c + oxp - sy]) * (v[c + oxp] + v[c]) -
                          (wff * gx[c] + wfb * gx[c - sy]) * (v[c] + v[c + oxm])) * (dxi * 0.5);
      const double h22 = ((gy[c + sy] + gy[c]) * (v[c + sy] + v[c]) - (gy[c] + gy[c - sy]) * (v[c] + v[c - sy])) *
                         (dycj * 0.5 * 0.5);
      const double h23 = ((wff * gz[c + ozp] + wfb * gz[c + ozp - sy]) * (v[c + ozp] + v[c]) -
                          (wff * gz[c] + wfb * gz[c - sy]) * (v[c] + v[c + ozm])) * (dzi * 0.5);
      const double conv = -(h21 + h22 + h23);
      const double coe1 = dxi * cv, coe3 = dzi * cv, coe2 = -2.0 / 3.0 * dycj * cv;
      const double muc = P.vis(i, j, k), mub = P.vis(i, j - 1, k);
      double dudx = (A(u, ip, j, k) - A(u, i, j, k)) * dxi;
      double dvdy = (A(v, i, j + 1, k) - A(v, i, j, k)) * dyfj;
      double dwdz = (A(w, i, j, kp) - A(w, i, j, k)) * dzi;
      const double t22fe = muc * (dudx + dwdz), t22fi = muc * dvdy;
      const double t22fa = th ? muc * ((AD(gy, r1, i, j + 1, k) - AD(gy, r1, i, j, k)) * dyfj) : 0.0;
      dudx = (A(u, ip, j - 1, k) - A(u, i, j - 1, k)) * dxi;
      dvdy = (A(v, i, j, k) - A(v, i, j - 1, k)) * d.dyfi[j - 1];
      dwdz = (A(w, i, j - 1, kp) - A(w, i, j - 1, k)) * dzi;
      const double t22be = mub * (dudx + dwdz), t22bi = mub * dvdy;
      const double t22ba = th ? mub * ((AD(gy, r1, i, j, k) - AD(gy, r1, i, j - 1, k)) * d.dyfi[j - 1]) : 0.0;
      const double d22e = (t22fe - t22be) * coe2, d22i = (t22fi - t22bi) * coe2 * (-2.0);
      const double d22a = (t22fa - t22ba) * coe2 * (-2.0);
      const double vis21p = P.s1(ip, j, k), vis21c = P.s1(i, j, k);
      double dvdx = (A(v, ip, j, k) - A(v, i, j, k)) * dxi;
      double dudy = (A(u, ip, j, k) - A(u, ip, j - 1, k)) * dycj;
      const double t21fe = vis21p * dudy, t21fi = vis21p * dvdx;
      const double t21fa = th ? vis21p * ((AD(gy, r1, ip, j, k) - AD(gy, r1, i, j, k)) * dxi) : 0.0;
      dvdx = (A(v, i, j, k) - A(v, im, j, k)) * dxi;
      dudy = (A(u, i, j, k) - A(u, i, j - 1, k)) * dycj;
      const double t21be = vis21c * dudy, t21bi = vis21c * dvdx;
      const double t21ba = th ? vis21c * ((AD(gy, r1, i, j, k) - AD(gy, r1, im, j, k)) * dxi) : 0.0;
      const double d21e = (t21fe - t21be) * coe1, d21i = (t21fi - t21bi) * coe1, d21a = (t21fa - t21ba) * coe1;
      const double vis23p = P.s3(i, j, kp), vis23c = P.s3(i, j, k);
      double dvdz = (A(v, i, j, kp) - A(v, i, j, k)) * dzi;
      double dwdy = (A(w, i, j, kp) - A(w, i, j - 1, kp)) * dycj;
      const double t23fe = vis23p * dwdy, t23fi = vis23p * dvdz;
      const double t23fa = th ? vis23p * ((AD(gy, r1, i, j, kp) - AD(gy, r1, i, j, k)) * dzi) : 0.0;
      dvdz = (A(v, i, j, k) - A(v, i, j, km)) * dzi;
      dwdy = (A(w, i, j, k) - A(w, i, j - 1, k)) * dycj;
      const double t23be = vis23c * dwdy, t23bi = vis23c * dvdz;
      const double t23ba = th ? vis23c * ((AD(gy, r1, i, j, k) - AD(gy, r1, i, j, km)) * dzi) : 0.0;
      const double d23e = (t23fe - t23be) * coe3, d23i = (t23fi - t23bi) * coe3, d23a = (t23fa - t23ba) * coe3;
      const double explt = (d21e + d22e + d23e) + conv;
      const double imp = d21i + d22i + d23i, adv = d21a + d22a + d23a;
      double *e0 = (double *)d.h0[1];
      double r = (gam * explt + roh * e0[c]) * dt;
      r = r + coe2a * imp + 0.5 * coe2a * adv;
      e0[c] = explt;
      r -= (p[c] - p[c - sy]) * (alp * dt * dycj);
      if (io.gravdir == 2) r += (alp * dt * io.f_a) / P.ri2(i, j, k);
      ((double *)d.rhs[1])[c] = r;
    } else if (C == 1) {
      ((double *)d.rhs[1])[c] = 0.0;
    }
    // ------------------------------------------------ z
    if (C == 2) {
      const double h31 = ((gx[c + oxp] + gx[c + oxp + ozm]) * (w[c + oxp] + w[c]) -
                          (gx[c] + gx[c + ozm]) * (w[c] + w[c + oxm])) * (dxi * 0.5 * 0.5);
      const double h32 = ((gy[c + sy] + gy[c + sy + ozm]) * (wffp * w[c + sy] + wfbp * w[c]) -
                          (gy[c] + gy[c + ozm]) * (wff * w[c] + wfb * w[c - sy])) * (dyfj * 0.5);
      const double h33 = ((gz[c + ozp] + gz[c]) * (w[c + ozp] + w[c]) - (gz[c] + gz[c + ozm]) * (w[c] + w[c + ozm])) *
                         (dzi * 0.5 * 0.5);
      const double conv = -(h31 + h32 + h33);
      const double coe1 = dxi * cv, coe3 = -2.0 / 3.0 * dzi * cv, coe2 = dyfj * cv;
      const double muc = P.vis(i, j, k), mub = P.vis(i, j, km);
      double dudx = (A(u, ip, j, k) - A(u, i, j, k)) * dxi;
      double dvdy = (A(v, i, j + 1, k) - A(v, i, j, k)) * dyfj;
      double dwdz = (A(w, i, j, kp) - A(w, i, j, k)) * dzi;
      const double t33fe = muc * (dudx + dvdy), t33fi = muc * dwdz;
      const double t33fa = th ? muc * ((AD(gz, r2, i, j, kp) - AD(gz, r2, i, j, k)) * dzi) : 0.0;
      dudx = (A(u, ip, j, km) - A(u, i, j, km)) * dxi;
      dvdy = (A(v, i, j + 1, km) - A(v, i, j, km)) * dyfj;
      dwdz = (A(w, i, j, k) - A(w, i, j, km)) * dzi;
      const double t33be = mub * (dudx + dvdy), t33bi = mub * dwdz;
      const double t33ba = th ? mub * ((AD(gz, r2, i, j, k) - AD(gz, r2, i, j, km)) * dzi) : 0.0;
      const double d33e = (t33fe - t33be) * coe3, d33i = (t33fi - t33bi) * coe3 * (-2.0);
      const double d33a = (t33fa - t33ba) * coe3 * (-2.0);
      const double vis31p = P.s2(ip, j, k), vis31c = P.s2(i, j, k);
      double dwdx = (A(w, ip, j, k) - A(w, i, j, k)) * dxi;
      double dudz = (A(u, ip, j, k) - A(u, ip, j, km)) * dzi;
      const double t31fe = vis31p * dudz, t31fi = vis31p * dwdx;
      const double t31fa = th ? vis31p * ((AD(gz, r2, ip, j, k) - AD(gz, r2, i, j, k)) * dxi) : 0.0;
      dwdx = (A(w, i, j, k) - A(w, im, j, k)) * dxi;
      dudz = (A(u, i, j, k) - A(u, i, j, km)) * dzi;
      const double t31be = vis31c * dudz, t31bi = vis31c * dwdx;
      const double t31ba = th ? vis31c * ((AD(gz, r2, i, j, k) - AD(gz, r2, im, j, k)) * dxi) : 0.0;
      const double d31e = (t31fe - t31be) * coe1, d31i = (t31fi - t31bi) * coe1, d31a = (t31fa - t31ba) * coe1;
      const double vis32p = P.s3(i, j + 1, k), vis32c = P.s3(i, j, k);
      double dwdy = (A(w, i, j + 1, k) - A(w, i, j, k)) * dycp;
      double dvdz = (A(v, i, j + 1, k) - A(v, i, j + 1, km)) * dzi;
      const double t32fe = vis32p * dvdz, t32fi = vis32p * dwdy;
      const double t32fa = th ? vis32p * ((AD(gz, r2, i, j + 1, k) - AD(gz, r2, i, j, k)) * dycp) : 0.0;
      dwdy = (A(w, i, j, k) - A(w, i, j - 1, k)) * dycj;
      dvdz = (A(v, i, j, k) - A(v, i, j, km)) * dzi;
      const double t32be = vis32c * dvdz, t32bi = vis32c * dwdy;
      const double t32ba = th ? vis32c * ((AD(gz, r2, i, j, k) - AD(gz, r2, i, j - 1, k)) * dycj) : 0.0;
      const double d32e = (t32fe - t32be) * coe2, d32i = (t32fi - t32bi) * coe2, d32a = (t32fa - t32ba) * coe2;
      const double explt = (d31e + d32e + d33e) + conv;
      const double imp = d31i + d32i + d33i, adv = d31a + d32a + d33a;
      double *e0 = (double *)d.h0[2];
      double r = (gam * explt + roh * e0[c]) * dt;
      r = r + coe2a * imp + 0.5 * coe2a * adv;
      e0[c] = explt;
      r -= (p[c] - p[c + ozm]) * (alp * dt * dzi);
      if (io.gravdir == 3) r += (alp * dt * io.f_a) / P.ri3(i, j, k);
      ((double *)d.rhs[2])[c] = r;
    }
  }
  if (C == 0) {
    // fixed-order block sum of RHS_x / DYFI
    for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
    const int tid = threadIdx.x + SI_BX * threadIdx.y;
    if ((tid & 31) == 0) red[tid >> 5] = part;
    __syncthreads();
    if (tid == 0) {
      double s = 0.0;
      for (int q = 0; q < SI_BX * SI_BY / 32; ++q) s += red[q];
      io.part[blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z)] = s;
    }
  }
}

// The same right-hand sides as a 2.5-D stencil, all three components in one
// launch: a block owns a 32 x 8 (x, y) tile and marches along z over nzc
// planes.  Each plane of u, v, w, G, p and, with the energy equation, mu,
// M = mu0 + mu (MU_STG is formed from it) and DRHOI_STG arrives as TMA boxes
// of 36 x 10 doubles (x0-2 .. x0+33, j0-1 .. j0+8) in a ring of four plane
// slots, plane k + 2 in flight while plane k is computed; periodic x
// neighbours outside the box are patched in on the first and last tiles.
// The ring (141 KB) allows one block per SM; its 24 warps are the three
// components of the tile, so that the registers of one component suffice and
// the warps hide each other's shared-memory latency.  The per-component
// kernels above read up to fourteen arrays from global memory, 60 loads per
// cell and component, and wait for them (DRAM 17 %): 3.15 ms for the three at
// 384x192x192 with the energy equation, 1.00 ms here (its bytes: 0.37 ms;
// at 192x96x192 L1 and shared memory 67 %, FP64 pipe 34 % busy).
constexpr int ST_BXW = 36, ST_BYW = 10, ST_PLANE = ST_BXW * ST_BYW, ST_PST = 368;
constexpr int S_U = 0, S_V = 1, S_W = 2, S_GX = 3, S_GY = 4, S_GZ = 5, S_P = 6, S_MU = 7, S_M = 8, S_R = 9;
constexpr int st_fields(bool th) { return th ? 12 : 7; }
constexpr size_t st_smem(bool th) { return (size_t)4 * st_fields(th) * ST_PST * sizeof(double) + 4 * sizeof(uint64_t); }
static_assert((ST_PST * 8) % 128 == 0 && ST_PST >= ST_PLANE, "TMA destinations must stay 128-byte aligned");
struct SiMaps {
  CUtensorMap m[12];  // in the order of S_U .. S_R + 2
};

template <bool TH>
__global__ void __launch_bounds__(3 * SI_BX *SI_BY, 1)
k_io_rhs_si_tma(const __grid_constant__ SiMaps maps, TGDev d, IODev io, double gam, double roh, double alp, int cur,
                int nzc) {
  constexpr int NF = st_fields(TH);
  extern __shared__ __align__(128) unsigned char smem_raw[];
  double *ring = reinterpret_cast<double *>(smem_raw);
  auto slot = [&](int sl) { return ring + (size_t)sl * NF * ST_PST; };
  uint64_t *bar = reinterpret_cast<uint64_t *>(ring + (size_t)4 * NF * ST_PST);
  __shared__ double red[SI_BX * SI_BY / 32];
  __shared__ double ycoef[SI_BY][9];
  __shared__ const double *src[NF];
  const int nx = d.nx, ny = d.ny, nz = d.nz;
  const int tx = threadIdx.x, ty = threadIdx.y, C = threadIdx.z, tid = tx + SI_BX * (ty + SI_BY * C);
  const int x0 = blockIdx.x * SI_BX, j0 = 1 + blockIdx.y * SI_BY;
  const int kbeg = blockIdx.z * nzc, kend = min(kbeg + nzc, nz);
  const int i = x0 + tx, j = j0 + ty;
  const bool active = i < nx && j <= ny;
  const bool left_edge = x0 == 0, right_edge = x0 + SI_BX >= nx;
  const int right_col = nx - x0 + 2;  // smem column of x = nx (wraps to 0)
  if (tid == 0) {
    for (int q = 0; q < 4; ++q) mbar_init(&bar[q], 1);
    fence_mbar_init();
    const double *f[12] = {d.u, d.v, d.w, io.g[cur][0], io.g[cur][1], io.g[cur][2], d.p,
                           io.mu, io.msum, io.drhoi[0], io.drhoi[1], io.drhoi[2]};
    for (int q = 0; q < NF; ++q) src[q] = f[q];
  }
  if (tid < SI_BY * 9) {
    const int r = tid / 9, q = tid - 9 * r, jr = j0 + r;
    double v = 0.0;
    if (jr <= ny) {
      switch (q) {
        case 0: v = d.wff[jr]; break;
        case 1: v = d.wfb[jr]; break;
        case 2: v = d.wff[jr + 1]; break;
        case 3: v = d.wfb[jr + 1]; break;
        case 4: v = d.dyfi[jr]; break;
        case 5: v = d.dyci[jr]; break;
        case 6: v = d.dyci[jr + 1]; break;
        case 7: v = d.dyfi[jr - 1]; break;
        case 8: v = 1.0 / d.dyfi[jr]; break;
      }
    }
    ycoef[r][q] = v;
  }
  __syncthreads();
  auto slot_of = [&](int k) { return (k - kbeg + 1) & 3; };
  auto issue = [&](int k) {
    const int sl = slot_of(k), kz = k < 0 ? k + nz : (k >= nz ? k - nz : k);
    mbar_expect_tx(&bar[sl], (uint32_t)(NF * ST_PLANE * sizeof(double)));
#pragma unroll
    for (int f = 0; f < NF; ++f) tma_load_3d(slot(sl) + f * ST_PST, &maps.m[f], x0 - 2, j0 - 1, kz, &bar[sl]);
  };
  uint32_t par = 0;
  auto wait_plane = [&](int k) -> bool {
    const int sl = slot_of(k);
    const bool ok = mbar_wait(&bar[sl], (par >> sl) & 1u, d.err);
    par ^= 1u << sl;
    const int kz = k < 0 ? k + nz : (k >= nz ? k - nz : k);
    if (left_edge && tid < 10 * NF) {
      const int f = tid / 10, r = tid - f * 10, jr = j0 - 1 + r;
      if (jr <= ny + 1) slot(sl)[f * ST_PST + r * ST_BXW + 1] = src[f][(nx - 1) + d.sy * jr + d.sz * kz];
    }
    if (right_edge && tid >= 384 && tid < 384 + 10 * NF) {
      const int q = tid - 384, f = q / 10, r = q - f * 10, jr = j0 - 1 + r;
      if (jr <= ny + 1) slot(sl)[f * ST_PST + r * ST_BXW + right_col] = src[f][d.sy * jr + d.sz * kz];
    }
    return ok;
  };
  if (tid == 0) {
    issue(kbeg - 1);
    issue(kbeg);
    issue(kbeg + 1);
  }
  bool ok = wait_plane(kbeg - 1);
  ok = wait_plane(kbeg) && ok;
  double part = 0.0;
  const double dxi = d.dxi, dzi = d.dzi, cv = d.cvisc, dt = d.dt, coe2a = alp * dt;
  const double *yc = ycoef[ty];
  const int at0 = (ty + 1) * ST_BXW + tx + 2;
  double *const e0p = (double *)d.h0[C];
  double *const rp = (double *)d.rhs[C];
  for (int k = kbeg; k < kend; ++k) {
    const int64_t c = i + d.sy * j + d.sz * k;
    const double e0 = active ? e0p[c] : 0.0;  // hides behind the plane wait
    ok = wait_plane(k + 1) && ok;
    // one barrier a plane, as in k_io_rhs_tma: no warp reads plane k - 2 after
    // it (momentum stage 3.35 -> 3.26 ms at 384x192x192)
    __syncthreads();
    if (tid == 0 && k + 2 <= kend) {
      fence_proxy_async();
      issue(k + 2);
    }
    if (active && ok) {
      const double *Sm = slot(slot_of(k - 1)) + at0, *Sc = slot(slot_of(k)) + at0, *Sp = slot(slot_of(k + 1)) + at0;
#define A(S, f, dx, dy) S[(f) * ST_PST + (dy) * ST_BXW + (dx)]
// G_io * DRHOI_STG of component q (and Q_io * DRHOI_STG where the reference writes it)
#define AD(S, f, q, dx, dy) (A(S, f, dx, dy) * A(S, S_R + (q), dx, dy))
      const double wff = yc[0], wfb = yc[1], wffp = yc[2], wfbp = yc[3], dyfj = yc[4], dycj = yc[5], dycp = yc[6];
      auto vis = [&](const double *S, int dx, int dy) { return TH ? A(S, S_MU, dx, dy) : 1.0; };
      // MU_STG 1-3 (MU_Staggered): s1 at column dx, row j + dy with that row's weights
      auto s1 = [&](int dx, int dy, double wf, double wb) {
        if (!TH) return 1.0;
        if (j + dy == 1) return 0.5 * A(Sc, S_M, dx, dy - 1);
        if (j + dy == ny + 1) return 0.5 * A(Sc, S_M, dx, dy);
        return ((A(Sc, S_M, dx, dy) + A(Sc, S_M, dx - 1, dy)) * wf +
                (A(Sc, S_M, dx, dy - 1) + A(Sc, S_M, dx - 1, dy - 1)) * wb) * 0.5 * 0.5;
      };
      auto s2 = [&](const double *S, const double *Sb, int dx) {
        if (!TH) return 1.0;
        return (A(S, S_M, dx, 0) + A(S, S_M, dx - 1, 0) + A(Sb, S_M, dx, 0) + A(Sb, S_M, dx - 1, 0)) * 0.5 * 0.5 * 0.5;
      };
      auto s3 = [&](const double *S, const double *Sb, int dy, double wf, double wb) {
        if (!TH) return 1.0;
        if (j + dy == 1) return 0.5 * A(S, S_M, 0, dy - 1);
        if (j + dy == ny + 1) return 0.5 * A(S, S_M, 0, dy);
        return ((A(Sb, S_M, 0, dy) + A(S, S_M, 0, dy)) * wf + (A(Sb, S_M, 0, dy - 1) + A(S, S_M, 0, dy - 1)) * wb) * 0.5 *
               0.5;
      };
      double conv, de, di, da = 0.0, pg, grav = 0.0;
      if (C == 0) {
        const double u0 = A(Sc, S_U, 0, 0);
        const double h11 = ((A(Sc, S_GX, 1, 0) + A(Sc, S_GX, 0, 0)) * (A(Sc, S_U, 1, 0) + u0) -
                            (A(Sc, S_GX, 0, 0) + A(Sc, S_GX, -1, 0)) * (u0 + A(Sc, S_U, -1, 0))) * (dxi * 0.5 * 0.5);
        const double h12 = ((A(Sc, S_GY, 0, 1) + A(Sc, S_GY, -1, 1)) * (wffp * A(Sc, S_U, 0, 1) + wfbp * u0) -
                            (A(Sc, S_GY, 0, 0) + A(Sc, S_GY, -1, 0)) * (wff * u0 + wfb * A(Sc, S_U, 0, -1))) *
                           (dyfj * 0.5);
        const double h13 = ((A(Sp, S_GZ, 0, 0) + A(Sp, S_GZ, -1, 0)) * (A(Sp, S_U, 0, 0) + u0) -
                            (A(Sc, S_GZ, 0, 0) + A(Sc, S_GZ, -1, 0)) * (u0 + A(Sm, S_U, 0, 0))) * (dzi * 0.5 * 0.5);
        conv = -(h11 + h12 + h13);
        const double coe1 = -2.0 / 3.0 * dxi * cv, coe2 = dyfj * cv, coe3 = dzi * cv;
        const double muc = vis(Sc, 0, 0), mum = vis(Sc, -1, 0);
        const double dvwf = (A(Sc, S_V, 0, 1) - A(Sc, S_V, 0, 0)) * dyfj + (A(Sp, S_W, 0, 0) - A(Sc, S_W, 0, 0)) * dzi;
        const double dvwb = (A(Sc, S_V, -1, 1) - A(Sc, S_V, -1, 0)) * dyfj + (A(Sp, S_W, -1, 0) - A(Sc, S_W, -1, 0)) * dzi;
        const double d11e = (muc * dvwf - mum * dvwb) * coe1;
        const double d11i = (muc * ((A(Sc, S_U, 1, 0) - u0) * dxi) - mum * ((u0 - A(Sc, S_U, -1, 0)) * dxi)) * coe1 * (-2.0);
        const double vp = s1(0, 1, wffp, wfbp), vc = s1(0, 0, wff, wfb);
        const double d12e = (vp * ((A(Sc, S_V, 0, 1) - A(Sc, S_V, -1, 1)) * dxi) -
                             vc * ((A(Sc, S_V, 0, 0) - A(Sc, S_V, -1, 0)) * dxi)) * coe2;
        const double d12i = (vp * ((A(Sc, S_U, 0, 1) - u0) * dycp) - vc * ((u0 - A(Sc, S_U, 0, -1)) * dycj)) * coe2;
        const double zp = s2(Sp, Sc, 0), zc = s2(Sc, Sm, 0);
        const double d13e = (zp * ((A(Sp, S_W, 0, 0) - A(Sp, S_W, -1, 0)) * dxi) -
                             zc * ((A(Sc, S_W, 0, 0) - A(Sc, S_W, -1, 0)) * dxi)) * coe3;
        const double d13i = (zp * ((A(Sp, S_U, 0, 0) - u0) * dzi) - zc * ((u0 - A(Sm, S_U, 0, 0)) * dzi)) * coe3;
        if (TH) {
          const double g0 = AD(Sc, S_GX, 0, 0, 0);
          const double d11a = (muc * ((AD(Sc, S_GX, 0, 1, 0) - g0) * dxi) - mum * ((g0 - AD(Sc, S_GX, 0, -1, 0)) * dxi)) *
                              coe1 * (-2.0);
          const double d12a = (vp * ((AD(Sc, S_GX, 0, 0, 1) - g0) * dycp) - vc * ((g0 - AD(Sc, S_GX, 0, 0, -1)) * dycj)) *
                              coe2;
          // the density part of tau13 differences Q_io, as the reference writes it
          const double q0 = AD(Sc, S_U, 0, 0, 0);
          const double d13a = (zp * ((AD(Sp, S_U, 0, 0, 0) - q0) * dzi) - zc * ((q0 - AD(Sm, S_U, 0, 0, 0)) * dzi)) * coe3;
          da = d11a + d12a + d13a;
        }
        de = d11e + d12e + d13e;
        di = d11i + d12i + d13i;
        pg = (A(Sc, S_P, 0, 0) - A(Sc, S_P, -1, 0)) * (alp * dt * dxi);
        if (io.gravdir == 1) grav = (alp * dt * io.f_a) / (TH ? io.stg[3][c] : 1.0);
      } else if (C == 1) {
        const double v0 = A(Sc, S_V, 0, 0), dyfm = yc[7];
        const double h21 = ((wff * A(Sc, S_GX, 1, 0) + wfb * A(Sc, S_GX, 1, -1)) * (A(Sc, S_V, 1, 0) + v0) -
                            (wff * A(Sc, S_GX, 0, 0) + wfb * A(Sc, S_GX, 0, -1)) * (v0 + A(Sc, S_V, -1, 0))) * (dxi * 0.5);
        const double h22 = ((A(Sc, S_GY, 0, 1) + A(Sc, S_GY, 0, 0)) * (A(Sc, S_V, 0, 1) + v0) -
                            (A(Sc, S_GY, 0, 0) + A(Sc, S_GY, 0, -1)) * (v0 + A(Sc, S_V, 0, -1))) * (dycj * 0.5 * 0.5);
        const double h23 = ((wff * A(Sp, S_GZ, 0, 0) + wfb * A(Sp, S_GZ, 0, -1)) * (A(Sp, S_V, 0, 0) + v0) -
                            (wff * A(Sc, S_GZ, 0, 0) + wfb * A(Sc, S_GZ, 0, -1)) * (v0 + A(Sm, S_V, 0, 0))) * (dzi * 0.5);
        conv = -(h21 + h22 + h23);
        const double coe1 = dxi * cv, coe3 = dzi * cv, coe2 = -2.0 / 3.0 * dycj * cv;
        const double muc = vis(Sc, 0, 0), mub = vis(Sc, 0, -1);
        const double duwf = (A(Sc, S_U, 1, 0) - A(Sc, S_U, 0, 0)) * dxi + (A(Sp, S_W, 0, 0) - A(Sc, S_W, 0, 0)) * dzi;
        const double duwb = (A(Sc, S_U, 1, -1) - A(Sc, S_U, 0, -1)) * dxi + (A(Sp, S_W, 0, -1) - A(Sc, S_W, 0, -1)) * dzi;
        const double d22e = (muc * duwf - mub * duwb) * coe2;
        const double d22i = (muc * ((A(Sc, S_V, 0, 1) - v0) * dyfj) - mub * ((v0 - A(Sc, S_V, 0, -1)) * dyfm)) * coe2 * (-2.0);
        const double xp = s1(1, 0, wff, wfb), xc = s1(0, 0, wff, wfb);
        const double d21e = (xp * ((A(Sc, S_U, 1, 0) - A(Sc, S_U, 1, -1)) * dycj) -
                             xc * ((A(Sc, S_U, 0, 0) - A(Sc, S_U, 0, -1)) * dycj)) * coe1;
        const double d21i = (xp * ((A(Sc, S_V, 1, 0) - v0) * dxi) - xc * ((v0 - A(Sc, S_V, -1, 0)) * dxi)) * coe1;
        const double zp = s3(Sp, Sc, 0, wff, wfb), zc = s3(Sc, Sm, 0, wff, wfb);
        const double d23e = (zp * ((A(Sp, S_W, 0, 0) - A(Sp, S_W, 0, -1)) * dycj) -
                             zc * ((A(Sc, S_W, 0, 0) - A(Sc, S_W, 0, -1)) * dycj)) * coe3;
        const double d23i = (zp * ((A(Sp, S_V, 0, 0) - v0) * dzi) - zc * ((v0 - A(Sm, S_V, 0, 0)) * dzi)) * coe3;
        if (TH) {
          const double g0 = AD(Sc, S_GY, 1, 0, 0);
          const double d22a = (muc * ((AD(Sc, S_GY, 1, 0, 1) - g0) * dyfj) - mub * ((g0 - AD(Sc, S_GY, 1, 0, -1)) * dyfm)) *
                              coe2 * (-2.0);
          const double d21a = (xp * ((AD(Sc, S_GY, 1, 1, 0) - g0) * dxi) - xc * ((g0 - AD(Sc, S_GY, 1, -1, 0)) * dxi)) * coe1;
          const double d23a = (zp * ((AD(Sp, S_GY, 1, 0, 0) - g0) * dzi) - zc * ((g0 - AD(Sm, S_GY, 1, 0, 0)) * dzi)) * coe3;
          da = d21a + d22a + d23a;
        }
        de = d21e + d22e + d23e;
        di = d21i + d22i + d23i;
        pg = (A(Sc, S_P, 0, 0) - A(Sc, S_P, 0, -1)) * (alp * dt * dycj);
        if (io.gravdir == 2) grav = (alp * dt * io.f_a) / (TH ? io.stg[4][c] : 1.0);
      } else {
        const double w0 = A(Sc, S_W, 0, 0);
        const double h31 = ((A(Sc, S_GX, 1, 0) + A(Sm, S_GX, 1, 0)) * (A(Sc, S_W, 1, 0) + w0) -
                            (A(Sc, S_GX, 0, 0) + A(Sm, S_GX, 0, 0)) * (w0 + A(Sc, S_W, -1, 0))) * (dxi * 0.5 * 0.5);
        const double h32 = ((A(Sc, S_GY, 0, 1) + A(Sm, S_GY, 0, 1)) * (wffp * A(Sc, S_W, 0, 1) + wfbp * w0) -
                            (A(Sc, S_GY, 0, 0) + A(Sm, S_GY, 0, 0)) * (wff * w0 + wfb * A(Sc, S_W, 0, -1))) * (dyfj * 0.5);
        const double h33 = ((A(Sp, S_GZ, 0, 0) + A(Sc, S_GZ, 0, 0)) * (A(Sp, S_W, 0, 0) + w0) -
                            (A(Sc, S_GZ, 0, 0) + A(Sm, S_GZ, 0, 0)) * (w0 + A(Sm, S_W, 0, 0))) * (dzi * 0.5 * 0.5);
        conv = -(h31 + h32 + h33);
        const double coe1 = dxi * cv, coe3 = -2.0 / 3.0 * dzi * cv, coe2 = dyfj * cv;
        const double muc = vis(Sc, 0, 0), mub = vis(Sm, 0, 0);
        const double duvf = (A(Sc, S_U, 1, 0) - A(Sc, S_U, 0, 0)) * dxi + (A(Sc, S_V, 0, 1) - A(Sc, S_V, 0, 0)) * dyfj;
        const double duvb = (A(Sm, S_U, 1, 0) - A(Sm, S_U, 0, 0)) * dxi + (A(Sm, S_V, 0, 1) - A(Sm, S_V, 0, 0)) * dyfj;
        const double d33e = (muc * duvf - mub * duvb) * coe3;
        const double d33i = (muc * ((A(Sp, S_W, 0, 0) - w0) * dzi) - mub * ((w0 - A(Sm, S_W, 0, 0)) * dzi)) * coe3 * (-2.0);
        const double xp = s2(Sc, Sm, 1), xc = s2(Sc, Sm, 0);
        const double d31e = (xp * ((A(Sc, S_U, 1, 0) - A(Sm, S_U, 1, 0)) * dzi) -
                             xc * ((A(Sc, S_U, 0, 0) - A(Sm, S_U, 0, 0)) * dzi)) * coe1;
        const double d31i = (xp * ((A(Sc, S_W, 1, 0) - w0) * dxi) - xc * ((w0 - A(Sc, S_W, -1, 0)) * dxi)) * coe1;
        const double yp = s3(Sc, Sm, 1, wffp, wfbp), yb = s3(Sc, Sm, 0, wff, wfb);
        const double d32e = (yp * ((A(Sc, S_V, 0, 1) - A(Sm, S_V, 0, 1)) * dzi) -
                             yb * ((A(Sc, S_V, 0, 0) - A(Sm, S_V, 0, 0)) * dzi)) * coe2;
        const double d32i = (yp * ((A(Sc, S_W, 0, 1) - w0) * dycp) - yb * ((w0 - A(Sc, S_W, 0, -1)) * dycj)) * coe2;
        if (TH) {
          const double g0 = AD(Sc, S_GZ, 2, 0, 0);
          const double d33a = (muc * ((AD(Sp, S_GZ, 2, 0, 0) - g0) * dzi) - mub * ((g0 - AD(Sm, S_GZ, 2, 0, 0)) * dzi)) *
                              coe3 * (-2.0);
          const double d31a = (xp * ((AD(Sc, S_GZ, 2, 1, 0) - g0) * dxi) - xc * ((g0 - AD(Sc, S_GZ, 2, -1, 0)) * dxi)) * coe1;
          const double d32a = (yp * ((AD(Sc, S_GZ, 2, 0, 1) - g0) * dycp) - yb * ((g0 - AD(Sc, S_GZ, 2, 0, -1)) * dycj)) *
                              coe2;
          da = d31a + d32a + d33a;
        }
        de = d31e + d32e + d33e;
        di = d31i + d32i + d33i;
        pg = (A(Sc, S_P, 0, 0) - A(Sm, S_P, 0, 0)) * (alp * dt * dzi);
        if (io.gravdir == 3) grav = (alp * dt * io.f_a) / (TH ? io.stg[5][c] : 1.0);
      }
#undef AD
#undef A
      if (C == 1 && j == 1) {
        rp[c] = 0.0;
      } else {
        const double explt = de + conv;
        double r = (gam * explt + roh * e0) * dt;
        r = r + coe2a * di + 0.5 * coe2a * da;
        e0p[c] = explt;
        r -= pg;
        r += grav;
        rp[c] = r;
        if (C == 0) part += r * yc[8];  // RHS_x / DYFI
      }
    }
  }
  // every issued plane has been waited for, so no bulk copy is in flight at
  // exit; fixed-order block sum of RHS_x / DYFI
  for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
  if (C == 0 && tx == 0) red[ty] = part;
  __syncthreads();
  if (tid == 0) {
    double s = 0.0;
    for (int q = 0; q < SI_BY; ++q) s += red[q];
    io.part[blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z)] = s;
  }
}

// Coefficients a x(-1) + b x(0) + c x(+1) of MOMFA1_X_io, MOMFA2_Z_io and
// MOMFA3_Y_io (axis AX: 0 x, 1 y, 2 z) for component C at value c of the
// fields, its neighbours along the line at offsets om and op.  The component's
// own axis takes VISCOUSITY of the cells on either side, the others MU_STG of
// the two edges; D holds 1 / RHO_STG of the component.
template <int C, int AX> struct LineCoef {
  static constexpr bool OWN = (AX == 0 && C == 0) || (AX == 1 && C == 1) || (AX == 2 && C == 2);
  const double *__restrict__ F, *__restrict__ D, *__restrict__ mu;
  int th;
  __device__ __forceinline__ explicit LineCoef(const IODev &io)
      : F(OWN ? io.mu : io.stg[AX == 0 ? C - 1 : (AX == 1 ? C : C + 1)]), D(io.stg[3 + C]), mu(io.mu), th(io.thermal) {}
  __device__ __forceinline__ double f(int64_t q) const { return th ? F[q] : 1.0; }
  __device__ __forceinline__ double r(int64_t q) const { return th ? D[q] : 1.0; }
  // periodic lines; w = - the factor of both edges
  __device__ __forceinline__ void cyc(int64_t c, int64_t om, int64_t op, double w, double &a, double &b,
                                      double &cc) const {
    const double amu = w * f(OWN ? c + om : c), apu = w * f(OWN ? c : c + op);
    a = amu * r(c + om);
    cc = apu * r(c + op);
    b = 1.0 - (amu + apu) * r(c);
  }
  // y lines, interior form of row j in 1..ny (every value it reads exists, so
  // that the staging loop has no branches); wm, wp: the row's factors
  __device__ __forceinline__ void row(int64_t c, int64_t sy, double wm, double wp, double &a, double &b,
                                      double &cc) const {
    const double amu = wm * f(OWN ? c - sy : c), apu = wp * f(OWN ? c : c + sy);
    a = amu * r(c - sy);
    cc = apu * r(OWN ? c : c + sy);  // v rows divide by the v face j itself, as written
    b = 1.0 - (amu + apu) * r(c);
  }
  // the wall rows j = 1 (lo) and ny: a wall edge takes the mean of the
  // viscosity across it (wm, wp: AMVR1, APVRN there), and with zero boundary
  // values the end couplings drop
  __device__ __forceinline__ void wall(int64_t c, int64_t sy, bool lo, double wm, double wp, double &a, double &b,
                                       double &cc) const {
    row(c, sy, wm, wp, a, b, cc);
    if (OWN) {
      if (lo) cc = wp * f(c) * r(c + sy);
    } else {
      const double edge = th ? (mu[c] + mu[lo ? c - sy : c + sy]) * 0.5 : 1.0;
      const double amu = wm * (lo ? edge : f(c)), apu = wp * (lo ? f(c + sy) : edge);
      a = amu * r(c - sy);
      cc = apu * r(c + sy);
      b = 1.0 - (amu + apu) * r(c);
    }
    if (lo) a = 0.0; else cc = 0.0;
  }
};

// ------------------------------------------------------------ line solves
// Warp partition solver for one tridiagonal line of n unknowns,
// a x(i-1) + b x(i) + c x(i+1) = r, cyclic (CYC) or with a(0) = c(n-1) = 0.
// The line is split into P equal chunks of m = n / P (P a power of two, at
// most 32, m >= 2: part_count).  Lane p eliminates its chunk's first m-1
// unknowns in terms of the chunk-end values L(p-1) and L(p) (one Thomas sweep
// with three right-hand sides), which leaves a P-unknown tridiagonal system
// for the chunk ends, cyclic when the line is; parallel cyclic reduction over
// shuffles solves it; then every lane back-substitutes its chunk.  The
// arrays live in shared memory with element i = p m + t at t Q + p
// (Q = P + 1, SlotWalk), so the lanes' sweeps touch consecutive words.  The result overwrites R.
__host__ __device__ inline int part_count(int n) {
  int P = 1;
  while (P < 32 && n % (2 * P) == 0 && n / (2 * P) >= 2) P *= 2;
  return P;
}
// Shared-memory layout of one line: element i at (i % m) * Q + i / m, rows of
// pitch Q = P + 1, so the lanes' chunk walks (row t, lane p: t * Q + p) read
// consecutive words and the coalesced staging loops, whose lanes take
// consecutive i, spread over the banks instead of hitting one bank at stride P.
// SlotWalk: the slots of i, i + step, i + 2 step, ... with one division at the start.
struct SlotWalk {
  int t, p, dt, dp, m, Q;
  __device__ __forceinline__ SlotWalk(int i, int step, int m_, int Q_)
      : t(i % m_), p(i / m_), dt(step % m_), dp(step / m_), m(m_), Q(Q_) {}
  __device__ __forceinline__ int slot() const { return t * Q + p; }
  __device__ __forceinline__ void next() {
    t += dt;
    p += dp;
    if (t >= m) {
      t -= m;
      ++p;
    }
  }
};
// values of one line array: m rows of pitch P + 1
__host__ __device__ inline int part_len(int n) {
  const int P = part_count(n);
  return (n / P) * (P + 1);
}
// stride of the lines of a z / y block (4 arrays), = 2 (mod 16) words: the
// staging loops' 8 lines x 2 elements per half-warp then fall in 16 banks
__host__ __device__ inline int zy_stride(int n) {
  const int s = 4 * part_len(n);
  return s + ((2 - s) % 16 + 16) % 16;
}

template <bool CYC>
__device__ void warp_part_solve(double *__restrict__ A, double *__restrict__ B, double *__restrict__ Cc,
                                double *__restrict__ R, int P, int Q, int m, int lane) {
  const bool act = lane < P;
  double yl = 0.0, vl = 0.0, wl = 0.0, yf = 0.0, vf = 0.0, wf = 0.0;
  double ae = 0.0, be = 1.0, ce = 0.0, re = 0.0;
  if (act) {
    double h = 0.0, y = 0.0, v = 0.0, w = 0.0;
    for (int t = 0; t <= m - 2; ++t) {
      const int q = t * Q + lane;
      const double a = A[q], b = B[q], c = Cc[q], r = R[q];
      const double al = t == 0 ? 0.0 : a;       // first row: a couples to L(p-1)
      const double cu = t == m - 2 ? 0.0 : c;   // last interior row: c couples to L(p)
      const double inv = 1.0 / (b - al * h);
      h = cu * inv;
      y = (r - al * y) * inv;
      v = ((t == 0 ? -a : 0.0) - al * v) * inv;
      w = ((t == m - 2 ? -c : 0.0) - al * w) * inv;
      Cc[q] = h; R[q] = y; A[q] = v; B[q] = w;
    }
    yl = y; vl = v; wl = w;
    for (int t = m - 3; t >= 0; --t) {
      const int q = t * Q + lane;
      const double hq = Cc[q];
      y = R[q] - hq * y;
      v = A[q] - hq * v;
      w = B[q] - hq * w;
      R[q] = y; A[q] = v; B[q] = w;
    }
    yf = y; vf = v; wf = w;
    const int qe = (m - 1) * Q + lane;
    ae = A[qe]; be = B[qe]; ce = Cc[qe]; re = R[qe];
  }
  const unsigned full = 0xffffffffu;
  const int nxt = act ? (lane + 1) % P : lane;
  const double yn = __shfl_sync(full, yf, nxt), vn = __shfl_sync(full, vf, nxt), wn = __shfl_sync(full, wf, nxt);
  // chunk-end equation: row e with x(e-1) = yl + vl L(p-1) + wl L(p) and
  // x(e+1) = yn + vn L(p) + wn L(p+1)
  double Ap = ae * vl, Bp = ae * wl + be + ce * vn, Cp = ce * wn, Rp = re - ae * yl - ce * yn;
  if (!act) { Ap = 0.0; Bp = 1.0; Cp = 0.0; Rp = 0.0; }
  // Each step squares the couplings (they fall by the chunk's diagonal
  // dominance), so the reduction ends where they no longer reach a double:
  // below 2^-100 of every diagonal, usually after the first of five steps.
  for (int hs = 1; hs < P; hs <<= 1) {
    if (!__any_sync(full, !(fabs(Ap) + fabs(Cp) < 0x1p-100 * fabs(Bp)))) break;
    const int lm = act ? (lane - hs + P) % P : lane, lp = act ? (lane + hs) % P : lane;
    double Am = __shfl_sync(full, Ap, lm), Bm = __shfl_sync(full, Bp, lm), Cm = __shfl_sync(full, Cp, lm),
           Rm = __shfl_sync(full, Rp, lm);
    double Aq = __shfl_sync(full, Ap, lp), Bq = __shfl_sync(full, Bp, lp), Cq = __shfl_sync(full, Cp, lp),
           Rq = __shfl_sync(full, Rp, lp);
    if (!CYC) {
      if (lane - hs < 0) { Am = 0.0; Bm = 1.0; Cm = 0.0; Rm = 0.0; }
      if (lane + hs >= P) { Aq = 0.0; Bq = 1.0; Cq = 0.0; Rq = 0.0; }
    }
    if (act) {
      const double k1 = Ap / Bm, k2 = Cp / Bq;
      const double nA = -Am * k1, nC = -Cq * k2;
      const double nB = Bp - Cm * k1 - Aq * k2;
      const double nR = Rp - Rm * k1 - Rq * k2;
      Ap = nA; Bp = nB; Cp = nC; Rp = nR;
    }
  }
  // couplings now reach distance P: the unknown itself (cyclic) or nothing
  const double L = CYC ? Rp / (Ap + Bp + Cp) : Rp / Bp;
  double Lm = __shfl_sync(full, L, act ? (lane - 1 + P) % P : lane);
  if (!CYC && lane == 0) Lm = 0.0;
  if (act) {
    for (int t = 0; t <= m - 2; ++t) {
      const int q = t * Q + lane;
      R[q] = R[q] + A[q] * Lm + B[q] * L;
    }
    R[(m - 1) * Q + lane] = L;
  }
}

// MOMFA1_X_io (TDMAIJI_CYC along x) for component C: one warp per (j, k) row;
// the row and its coefficients are staged in shared memory with coalesced
// loads, solved by warp_part_solve and written back in place.  x-momentum
// subtracts DPGRNS from RHS_io as it is read.
template <int C>
__global__ void __launch_bounds__(256) k_si_x(TGDev d, IODev io, double coe1, double coe2, int use_dpg) {
  extern __shared__ double xs_smem[];
  const int nx = d.nx, j0 = C == 1 ? 2 : 1, nj = d.ny - j0 + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int line = blockIdx.x * nw + warp;
  if (line >= nj * d.nz) return;  // whole warp leaves together
  const int j = j0 + line % nj, k = line / nj;
  const int P = part_count(nx), m = nx / P, Q = P + 1, len = m * Q;
  double *A = xs_smem + (size_t)warp * 4 * len, *B = A + len, *Cc = B + len, *Rs = Cc + len;
  const LineCoef<C, 0> co(io);
  const int64_t row = d.sy * j + d.sz * k;
  const double w = -(C == 0 ? coe1 : coe2);
  double *__restrict__ R = (double *)d.rhs[C] + row;
  const double sub = (C == 0 && use_dpg) ? *io.dpg : 0.0;
  SlotWalk sl(lane, 32, m, Q);
#pragma unroll 4
  for (int i = lane; i < nx; i += 32, sl.next()) {
    double a, b, cc;
    co.cyc(row + i, i == 0 ? nx - 1 : -1, i + 1 == nx ? 1 - nx : 1, w, a, b, cc);
    const int q = sl.slot();
    A[q] = a; B[q] = b; Cc[q] = cc; Rs[q] = R[i] - sub;
  }
  __syncwarp();
  warp_part_solve<true>(A, B, Cc, Rs, P, Q, m, lane);
  __syncwarp();
  SlotWalk so(lane, 32, m, Q);
  for (int i = lane; i < nx; i += 32, so.next()) R[i] = Rs[so.slot()];
}

// Lines along z (MOMFA2_Z_io, cyclic) or y (MOMFA3_Y_io, rows 1..ny, zero
// boundary values) for component C: a block stages LB lines of consecutive x
// (each row of the tile one coalesced load), its warps solve them in turn.
// The y solve ends with G* = G + dG in the other G buffer from row N2I.
// Four blocks per SM (64 registers, a few spilled words) with 8 lines each at
// n = 192: the blocks' stage / solve / store phases overlap better than two
// blocks of 16 lines.  Bound by instruction issue (47-56 %), so the staging
// loops carry no divisions (1 / RHO_STG once per cell in k_si_stg, slots by
// SlotWalk) and no branches (wall rows apart), and the reduction ends early:
// x / z / y lines of one component at 384x192x192 260 / 335 / 560 -> 169 / 203
// / 280 us, their bytes 70 / 70 / 110 us.
template <int C, bool Y>
__global__ void __launch_bounds__(256, 4) k_si_zy(TGDev d, IODev io, double coe1, double coe2, int LB, int cur) {
  extern __shared__ double zs_smem[];
  const int nx = d.nx, ny = d.ny;
  const int n = Y ? ny : d.nz;
  const int j0 = C == 1 ? 2 : 1;
  const int i0 = blockIdx.x * LB;
  const int nl = min(LB, nx - i0);
  // z lines: blockIdx.y = row j - j0; y lines: blockIdx.y = plane k
  const int jz = Y ? 0 : j0 + (int)blockIdx.y, ky = Y ? (int)blockIdx.y : 0;
  const int P = part_count(n), m = n / P, Q = P + 1, len = m * Q, S = zy_stride(n);
  const LineCoef<C, Y ? 1 : 2> co(io);
  const int64_t st = Y ? d.sy : d.sz;
  const int64_t base = (Y ? d.sz * ky + d.sy : d.sy * jz) + i0;  // + l, + st * (index along the line)
  double *__restrict__ R = (double *)d.rhs[C];
  // thread -> line l of the tile and every (blockDim / LB)-th element of it;
  // LB is a power of two
  const int l = threadIdx.x & (LB - 1), e0 = threadIdx.x >> (__ffs(LB) - 1), de = blockDim.x / LB;
  double *const L = zs_smem + (size_t)l * S;
  const double w = -(C == 2 ? coe1 : coe2);  // z lines
  double *const rw = zs_smem + (size_t)LB * S;  // y lines: the rows' factors, minus then plus side
  if (Y) {
    for (int e = threadIdx.x; e < n; e += blockDim.x) {
      const double f = C == 1 ? -coe1 * 4.0 / 3.0 : -coe1;
      rw[e] = f * (C != 1 && e == 0 ? io.amvr1 : d.amvr[C][e + 1]);
      rw[n + e] = f * (C != 1 && e + 1 == n ? io.apvrn : d.apvr[C][e + 1]);
    }
    __syncthreads();
  }
  SlotWalk sl(e0, de, m, Q);
  if (l < nl) {
#pragma unroll 4
    for (int e = e0; e < n; e += de, sl.next()) {
      double a, b, cc;
      const int64_t g = base + l + st * e;
      if (Y)
        co.row(g, st, rw[e], rw[n + e], a, b, cc);
      else
        co.cyc(g, e == 0 ? st * (n - 1) : -st, e + 1 == n ? st * (1 - n) : st, w, a, b, cc);
      const int q = sl.slot();
      L[q] = a; L[len + q] = b; L[2 * len + q] = cc; L[3 * len + q] = R[g];
    }
    if (Y) {  // the wall rows again, by the threads that staged them
      double a, b, cc;
      if (e0 == 0) {
        co.wall(base + l, st, true, rw[0], rw[n], a, b, cc);
        L[0] = a; L[len] = b; L[2 * len] = cc;
      }
      if ((n - 1) % de == e0) {
        const int q = (m - 1) * Q + P - 1;
        co.wall(base + l + st * (n - 1), st, false, rw[n - 1], rw[2 * n - 1], a, b, cc);
        L[q] = a; L[len + q] = b; L[2 * len + q] = cc;
      }
    }
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int q = warp; q < nl; q += nw) {
    double *T = zs_smem + (size_t)q * S;
    warp_part_solve<!Y>(T, T + len, T + 2 * len, T + 3 * len, P, Q, m, lane);
  }
  __syncthreads();
  SlotWalk so(e0, de, m, Q);
  if (l < nl)
    for (int e = e0; e < n; e += de, so.next()) {
      const double x = L[3 * len + so.slot()];
      const int64_t g = base + l + st * e;
      if (!Y)
        R[g] = x;
      else if (e + 1 >= j0)
        io.g[1 - cur][C][g] = x + io.g[cur][C][g];
    }
}

inline dim3 si_cell_grid(const TGDev &d) { return dim3((d.nx + SI_BX - 1) / SI_BX, (d.ny + SI_BY - 1) / SI_BY, d.nz); }

}  // namespace

// Shared-memory limit of the z-marching right-hand side; the tensor maps of mu
// and DRHOI_STG are made beside the explicit kernel's (io_init_maps).
int io_si_setup(chapsim_ctx *c) {
  int optin = 0;
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device);
  if ((size_t)optin < st_smem(true) + 2048) return CHAPSIM_OK;
  if (cudaFuncSetAttribute(k_io_rhs_si_tma<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)st_smem(true)) != cudaSuccess ||
      cudaFuncSetAttribute(k_io_rhs_si_tma<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)st_smem(false)) != cudaSuccess) {
    c->err = "semi-implicit right-hand side: cannot raise the shared-memory limit";
    return CHAPSIM_ERR_CUDA;
  }
  c->use_tma_si = true;
  return CHAPSIM_OK;
}

// Right-hand sides of the semi-implicit momentum stage; *npart receives the
// number of block partials written for DPGRNS.
int io_mom_si(chapsim_ctx *c, int ns, int *npart) {
  TGDev &d = c->d;
  IODev &io = c->io;
  const SubParams &sp = c->sp[ns];
  const dim3 grid = si_cell_grid(d);
  if (io.thermal) {
    k_si_stg<<<dim3(grid.x, (d.ny + 2 + SI_BY - 1) / SI_BY, d.nz), dim3(SI_BX, SI_BY), 0, c->stream>>>(d, io);
    LAUNCHED();
  }
  if (c->use_tma_si) {
    SiMaps maps;
    const int id[7] = {0, 1, 2, 5 + 3 * c->io_cur, 6 + 3 * c->io_cur, 7 + 3 * c->io_cur, 3};
    for (int q = 0; q < 7; ++q) maps.m[q] = c->io_maps[id[q]];
    maps.m[S_M] = c->io_maps[4];
    maps.m[S_MU] = c->si_maps[0];
    for (int q = 0; q < 3; ++q) maps.m[S_R + q] = c->si_maps[1 + q];
    const int nzc = rhs_march(c);
    const dim3 g2(grid.x, grid.y, (d.nz + nzc - 1) / nzc), blk(SI_BX, SI_BY, 3);
    if (io.thermal)
      k_io_rhs_si_tma<true><<<g2, blk, st_smem(true), c->stream>>>(maps, d, io, sp.gam, sp.roh, sp.alp, c->io_cur, nzc);
    else
      k_io_rhs_si_tma<false><<<g2, blk, st_smem(false), c->stream>>>(maps, d, io, sp.gam, sp.roh, sp.alp, c->io_cur, nzc);
    LAUNCHED();
    *npart = (int)(g2.x * g2.y * g2.z);
    return CHAPSIM_OK;
  }
  // grids too small for the boxes: one kernel per component, a third of the
  // live values each
  if (io.thermal) {
    k_io_rhs_si<0, true><<<grid, dim3(SI_BX, SI_BY), 0, c->stream>>>(d, io, sp.gam, sp.roh, sp.alp, c->io_cur);
    LAUNCHED();
    k_io_rhs_si<1, true><<<grid, dim3(SI_BX, SI_BY), 0, c->stream>>>(d, io, sp.gam, sp.roh, sp.alp, c->io_cur);
    LAUNCHED();
    k_io_rhs_si<2, true><<<grid, dim3(SI_BX, SI_BY), 0, c->stream>>>(d, io, sp.gam, sp.roh, sp.alp, c->io_cur);
    LAUNCHED();
  } else {
    k_io_rhs_si<0, false><<<grid, dim3(SI_BX, SI_BY), 0, c->stream>>>(d, io, sp.gam, sp.roh, sp.alp, c->io_cur);
    LAUNCHED();
    k_io_rhs_si<1, false><<<grid, dim3(SI_BX, SI_BY), 0, c->stream>>>(d, io, sp.gam, sp.roh, sp.alp, c->io_cur);
    LAUNCHED();
    k_io_rhs_si<2, false><<<grid, dim3(SI_BX, SI_BY), 0, c->stream>>>(d, io, sp.gam, sp.roh, sp.alp, c->io_cur);
    LAUNCHED();
  }
  *npart = (int)(grid.x * grid.y * grid.z);
  return CHAPSIM_OK;
}

// MOMFA_io for the three components: x, z and y factor solves, G* into the
// other G buffer.
namespace {
int zy_lines_per_block(int n) {
  // lines of one z / y block: as many as fit in 50 KB (4 arrays of n values),
  // so that four blocks share an SM
  // (a power of two)
  const int fit = (int)(50 * 1024 / ((size_t)32 * n));
  int lb = 1;
  while (2 * lb <= fit && lb < 32) lb *= 2;
  return lb;
}
template <int C>
int si_solves(chapsim_ctx *c, double facoe, double cx1, double cx2, double cz1, double cz2) {
  TGDev &d = c->d;
  IODev &io = c->io;
  const int j0 = C == 1 ? 2 : 1, nj = d.ny - j0 + 1;
  {
    // rows per block: as many as fit in 110 KB (4 arrays of nx values each)
    int wpb = (int)(110 * 1024 / ((size_t)32 * d.nx));
    wpb = wpb < 1 ? 1 : (wpb > 8 ? 8 : wpb);
    const size_t sm = (size_t)wpb * 4 * part_len(d.nx) * sizeof(double);
    k_si_x<C><<<(nj * d.nz + wpb - 1) / wpb, 32 * wpb, sm, c->stream>>>(d, io, cx1, cx2, 1);
    LAUNCHED();
  }
  {
    const int lb = zy_lines_per_block(d.nz);
    k_si_zy<C, false><<<dim3((d.nx + lb - 1) / lb, nj), 256, (size_t)lb * zy_stride(d.nz) * sizeof(double), c->stream>>>(
        d, io, cz1, cz2, lb, c->io_cur);
    LAUNCHED();
  }
  {
    const int lb = zy_lines_per_block(d.ny);
    k_si_zy<C, true><<<dim3((d.nx + lb - 1) / lb, d.nz), 256, ((size_t)lb * zy_stride(d.ny) + 2 * d.ny) * sizeof(double), c->stream>>>(
        d, io, facoe, 0.0, lb, c->io_cur);
    LAUNCHED();
  }
  return CHAPSIM_OK;
}
}  // namespace

int io_factor_si(chapsim_ctx *c, int ns) {
  TGDev &d = c->d;
  const double facoe = 0.5 * c->sp[ns].alp * d.dt * d.cvisc;  // FACOE_io
  const double cx1 = facoe * 4.0 / 3.0 * d.dxqi, cx2 = facoe * d.dxqi;
  const double cz1 = facoe * 4.0 / 3.0 * d.dzqi, cz2 = facoe * d.dzqi;
  if (!c->si_smem_set) {
    // dynamic shared memory above 48 KB (k_si_zy at ny = 192 takes 51 KB):
    // the limit is set per device, with that device current, by every
    // context before its first solve; setting it again is harmless and it
    // involves no process-wide bookkeeping shared between host threads
    int optin = 0;
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device);
    const void *fns[] = {(const void *)k_si_x<0>, (const void *)k_si_x<1>, (const void *)k_si_x<2>,
                         (const void *)k_si_zy<0, false>, (const void *)k_si_zy<1, false>,
                         (const void *)k_si_zy<2, false>, (const void *)k_si_zy<0, true>,
                         (const void *)k_si_zy<1, true>, (const void *)k_si_zy<2, true>};
    for (const void *f : fns)
      if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, optin) != cudaSuccess) {
        cudaGetLastError();
        c->err = "semi-implicit line solves: cannot raise the shared-memory limit";
        return CHAPSIM_ERR_CUDA;
      }
    c->si_smem_set = true;
  }
  int rc;
  if ((rc = si_solves<0>(c, facoe, cx1, cx2, cz1, cz2))) return rc;
  if ((rc = si_solves<1>(c, facoe, cx1, cx2, cz1, cz2))) return rc;
  return si_solves<2>(c, facoe, cx1, cx2, cz1, cz2);
}

}  // namespace chapsim
