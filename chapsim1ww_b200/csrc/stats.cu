// On-device flow statistics of the TG channel: the xz-plane averages of
// PP_MEAN_ZX_FLOW_TG (src/processing/PP_MEAN_ZX.f90:1-294) and their running
// time average PP_MEAN_T_TG (src/processing/PP_MEAN_T.f90:322-370), so that a
// host needs no per-step download of the field to keep its statistics.
//
// Per y-row j the 122 values are, in this order:
//   U1 (4)     mean of the cell-centred u, v, w (x 0.5 x 2) and p
//   UP (3)     u_i p
//   U2 (6)     u_i u_j, upper triangle (11 12 13 22 23 33)
//   U3 (10)    u_i u_j u_k, upper tetrahedron (111 112 113 122 123 133 222 223 233 333)
//   DVDL1 (9)  du_m/dx_n, row-major (m, n)
//   DVDLP (9)  du_m/dx_n p
//   DVDL2 (81) (du_m/dx_h)(du_n/dx_p), row (m,h), column (n,p)
// with the reference's scaling (VL1313 = 1/(nx nz) and the 0.5 factors of the
// cell-centred sums).
//
// Reduction: grid (ny, NBK k-chunks, 2 groups); every block sums its cells in
// a fixed order and writes one partial per accumulator; a second kernel adds
// the NBK partials of each row in order and applies the scaling, so the
// result is bit-reproducible.  Group 0 holds U1, UP, U2, U3, DVDL1, DVDLP
// (41 values), group 1 the upper triangle of the symmetric DVDL2 (45).
//
// IO section (x-periodic): PP_MEAN_ZX_FLOW_Xperiodic_IO
// (src/processing/PP_MEAN_ZX.f90:299-872) and PP_MEAN_T_Xperiodic_IO
// (src/processing/PP_MEAN_T.f90:436-520, the xz fields): 360 values per row
// (141 flow, 219 with the energy equation; the order is stated at
// io_source).  Every value is the xz-mean of a product of at most four
// per-cell quantities (U, p, G, the velocity gradient D, T, rho, h, mu, k
// and the gradients of h and T); k_io_stats_part forms the 288 distinct
// products, grid (ny, ST_NBK k-chunks).
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>
#include <vector>

#include "chapsim_internal.cuh"

namespace chapsim {
namespace {

constexpr int ST_NV = 122, ST_G0 = 41, ST_G1 = 45, ST_NBK = 4, ST_TPB = 128;

#define CK(call)                                                          \
  do {                                                                    \
    cudaError_t e_ = (call);                                              \
    if (e_ != cudaSuccess) {                                              \
      c->err = std::string(#call) + ": " + cudaGetErrorString(e_);        \
      return CHAPSIM_ERR_CUDA;                                            \
    }                                                                     \
  } while (0)

#define LAUNCHED()                                                        \
  do {                                                                    \
    ++c->launches;                                                        \
    cudaError_t e_ = cudaGetLastError();                                  \
    if (e_ != cudaSuccess) {                                              \
      c->err = std::string("kernel launch: ") + cudaGetErrorString(e_);   \
      return CHAPSIM_ERR_CUDA;                                            \
    }                                                                     \
  } while (0)

// The 13 per-cell quantities: U_cct(1..3), p, and DVDL_cct(3x3) (unscaled).
struct CellQ {
  double U[3], p, D[9];
};

__device__ __forceinline__ CellQ cell_quantities(const TGDev &d, int i, int j, int k) {
  const int nx = d.nx, nz = d.nz;
  const int ip = i + 1 == nx ? 0 : i + 1, im = i == 0 ? nx - 1 : i - 1;
  const int kp = k + 1 == nz ? 0 : k + 1, km = k == 0 ? nz - 1 : k - 1;
  const int64_t sy = d.sy, sz = d.sz;
  const int64_t c = i + sy * j + sz * k;
  const int64_t oxp = ip - i, oxm = im - i, ozp = sz * (kp - k), ozm = sz * (km - k);
  const double *u = d.u, *v = d.v, *w = d.w;
  CellQ q;
  // U_cct and its neighbours (src/processing/PP_MEAN_ZX.f90:79-121, channel branch)
  const double u0 = u[c] + u[c + oxp];
  const double ujp = u[c + sy] + u[c + sy + oxp], ujm = u[c - sy] + u[c - sy + oxp];
  const double ukp = u[c + ozp] + u[c + ozp + oxp], ukm = u[c + ozm] + u[c + ozm + oxp];
  const double w0 = w[c] + w[c + ozp];
  const double wip = w[c + oxp] + w[c + oxp + ozp], wim = w[c + oxm] + w[c + oxm + ozp];
  const double wjp = w[c + sy] + w[c + sy + ozp], wjm = w[c - sy] + w[c - sy + ozp];
  const double v0 = v[c] + v[c + sy];
  const double vip = v[c + oxp] + v[c + oxp + sy], vim = v[c + oxm] + v[c + oxm + sy];
  const double vkp = v[c + ozp] + v[c + ozp + sy], vkm = v[c + ozm] + v[c + ozm + sy];
  q.U[0] = u0; q.U[1] = v0; q.U[2] = w0;
  q.p = d.p[c];
  const double dycp = d.dyci[j + 1], dycj = d.dyci[j];
  q.D[0] = u[c + oxp] - u[c];
  q.D[1] = (ujp - u0) * dycp + (u0 - ujm) * dycj;
  q.D[2] = ukp - ukm;
  q.D[3] = vip - vim;
  q.D[4] = (v[c + sy] - v[c]) * d.dyfi[j];
  q.D[5] = vkp - vkm;
  q.D[6] = wip - wim;
  q.D[7] = (wjp - w0) * dycp + (w0 - wjm) * dycj;
  q.D[8] = w[c + ozp] - w[c];
  return q;
}

template <int G>
__global__ void __launch_bounds__(ST_TPB) k_stats_part(TGDev d, double *part) {
  constexpr int NA = G == 0 ? ST_G0 : ST_G1;
  __shared__ double red[ST_TPB / 32][NA];
  const int j = blockIdx.x + 1;
  const int nx = d.nx, nz = d.nz;
  const int k0 = (int)((int64_t)nz * blockIdx.y / ST_NBK), k1 = (int)((int64_t)nz * (blockIdx.y + 1) / ST_NBK);
  double acc[NA];
#pragma unroll
  for (int a = 0; a < NA; ++a) acc[a] = 0.0;
  const int ncell = nx * (k1 - k0);
  for (int t = threadIdx.x; t < ncell; t += ST_TPB) {
    const int kk = k0 + t / nx, i = t % nx;
    const CellQ q = cell_quantities(d, i, j, kk);
    if (G == 0) {
      int a = 0;
#pragma unroll
      for (int m = 0; m < 3; ++m) acc[a++] += q.U[m];
      acc[a++] += q.p;
#pragma unroll
      for (int m = 0; m < 3; ++m) acc[a++] += q.U[m] * q.p;
#pragma unroll
      for (int m = 0; m < 3; ++m)
#pragma unroll
        for (int n = m; n < 3; ++n) acc[a++] += q.U[m] * q.U[n];
#pragma unroll
      for (int m = 0; m < 3; ++m)
#pragma unroll
        for (int n = m; n < 3; ++n)
#pragma unroll
          for (int h = n; h < 3; ++h) acc[a++] += q.U[m] * q.U[n] * q.U[h];
#pragma unroll
      for (int m = 0; m < 9; ++m) acc[a++] += q.D[m];
#pragma unroll
      for (int m = 0; m < 9; ++m) acc[a++] += q.D[m] * q.p;
    } else {
      int a = 0;
#pragma unroll
      for (int l1 = 0; l1 < 9; ++l1)
#pragma unroll
        for (int l2 = l1; l2 < 9; ++l2) acc[a++] += q.D[l1] * q.D[l2];
    }
  }
  // fixed-order block reduction: warp tree, then the warps in order
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int a = 0; a < NA; ++a) {
    double v = acc[a];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) red[wid][a] = v;
  }
  __syncthreads();
  for (int a = threadIdx.x; a < NA; a += ST_TPB) {
    double s = 0.0;
    for (int q = 0; q < ST_TPB / 32; ++q) s += red[q][a];
    part[((size_t)(j - 1) * ST_NBK + blockIdx.y) * (ST_G0 + ST_G1) + (G == 0 ? 0 : ST_G0) + a] = s;
  }
}

// Sum the k-chunk partials of each row in order, scale as the reference does,
// expand the DVDL2 triangle, and (accumulate != 0) fold into the time average.
__global__ void k_stats_final(TGDev d, const double *part, double *xz, double *xzt, double coe2, double coe3,
                              int accumulate) {
  const int j = blockIdx.x + 1;
  const double vl = 1.0 / ((double)d.nx * (double)d.nz);
  const double cog1[9] = {vl * d.dxi, vl * 0.25, vl * 0.25 * d.dzi, vl * 0.25 * d.dxi, vl,
                          vl * 0.25 * d.dzi, vl * 0.25 * d.dxi, vl * 0.25, vl * d.dzi};
  double *out = xz + (size_t)(j - 1) * ST_NV;
  for (int a = threadIdx.x; a < ST_G0 + 81; a += blockDim.x) {
    // source accumulator index and scale of output value a (group-0 part and
    // the 81 DVDL2 entries from the upper triangle)
    int src;
    double sc;
    int o;
    if (a < ST_G0) {
      src = a;
      o = a;
      if (a < 3) sc = vl * 0.5;                   // U1 u, v, w
      else if (a == 3) sc = vl;                   // U1 p
      else if (a < 7) sc = vl * 0.5;              // UP
      else if (a < 13) sc = vl * (0.5 * 0.5);     // U2
      else if (a < 23) sc = vl * (0.5 * 0.5 * 0.5);  // U3
      else if (a < 32) sc = cog1[a - 23];         // DVDL1
      else sc = cog1[a - 32];                     // DVDLP
    } else {
      const int e = a - ST_G0, l1 = e / 9, l2 = e % 9;
      const int lo = l1 < l2 ? l1 : l2, hi = l1 < l2 ? l2 : l1;
      src = ST_G0 + lo * 9 - lo * (lo - 1) / 2 + (hi - lo);
      o = ST_G0 + e;
      sc = cog1[l1] * cog1[l2];
    }
    double s = 0.0;
    for (int b = 0; b < ST_NBK; ++b) s += part[((size_t)(j - 1) * ST_NBK + b) * (ST_G0 + ST_G1) + src];
    const double val = s * sc;
    out[o] = val;
    if (accumulate) {
      double *t = xzt + (size_t)(j - 1) * ST_NV + o;
      *t = coe3 * *t + coe2 * val;
    }
  }
}

// ------------------------------------------------------------- IO section
// The 288 distinct sums behind the 360 IO statistics (DVDL2 and DVDL2M are
// symmetric), in six groups of 48 so that one thread keeps a group's sums in
// registers.  With D(l) the nine velocity gradients:
//   0  D, D p, D D (upper triangle, rows 0-2), dh, dh p
//   1  D D (rows 3-8), dh mu D
//   2  D mu, D mu h, D D mu (rows 0-2), T, rho, h, mu, T T, rho rho
//   3  D D mu (rows 3-8), D mu U
//   4  dT k, dT k U, dT k D, h U, h G, h h, h rho, h p
//   5  U, p, G, U p, U U, U G, U U U, U G U, rho h U U
constexpr int SI_NV = 360, SI_NG = 6, SI_GN = 48, SI_NS = SI_NG * SI_GN, SI_TOP = 24;  // SI_TOP: triangle rows 0-2
// per-cell quantities in shared memory: U, G, p, D, dh, dT k, T, rho, h, mu
enum { B_U = 0, B_G = 3, B_P = 6, B_D = 7, B_DH = 16, B_DTK = 19, B_T = 22, B_R = 23, B_H = 24, B_M = 25, SI_NB = 26 };
constexpr int SI_CH = 64, SI_TPB = SI_NG * SI_CH;  // cells per chunk, threads per block

// the sum that holds each of the 360 output values, in output order
std::vector<uint16_t> io_source() {
  std::vector<uint16_t> t;
  auto run = [&](int g, int a, int n) {
    for (int q = 0; q < n; ++q) t.push_back((uint16_t)(SI_GN * g + a + q));
  };
  auto sym = [&](int g, int a, int b) {  // a 9 x 9 symmetric matrix: its triangle in group g from a, then g + 1 from b
    for (int l1 = 0; l1 < 9; ++l1)
      for (int l2 = 0; l2 < 9; ++l2) {
        const int lo = l1 < l2 ? l1 : l2, hi = l1 < l2 ? l2 : l1, q = lo * 9 - lo * (lo - 1) / 2 + (hi - lo);
        q < SI_TOP ? run(g, a + q, 1) : run(g + 1, b + q - SI_TOP, 1);
      }
  };
  run(5, 0, 4);    // U1: u, v, w, p
  run(5, 4, 3);    // G1
  run(5, 7, 3);    // UP
  run(5, 10, 6);   // U2
  run(5, 16, 6);   // UG
  run(5, 22, 10);  // U3
  run(5, 32, 10);  // UGU
  run(0, 0, 9);    // DVDL1
  run(0, 9, 9);    // DVDLP
  sym(0, 18, 0);   // DVDL2
  run(2, 42, 4);   // T1 D1 H1 M1
  run(2, 46, 2);   // T2 D2
  run(4, 45, 3);   // H2 DH PH
  run(2, 0, 9);    // DVDL1M
  run(2, 9, 9);    // DVDL1MH
  run(3, 21, 27);  // DVDL1MU
  sym(2, 18, 0);   // DVDL2M
  run(4, 39, 3);   // UH
  run(4, 42, 3);   // GH
  run(5, 42, 6);   // U2DH
  run(0, 42, 3);   // DhDL1
  run(0, 45, 3);   // DhDLP
  run(4, 0, 3);    // DTDLK
  run(4, 3, 9);    // DTDLKU
  run(4, 12, 27);  // DTDLKDVDL
  run(1, 21, 27);  // DHDLMDVDL
  return t;
}

struct IOStatFields {
  const double *g[3];  // current mass flux G
};

// A share of the per-cell quantities of cell (i, j, k) (0-based i, k; row j):
// part 0 the u row (U and the three gradients, central differences as in the
// reference), 1 the v row, 2 the w row, 3 p, G, rho, mu, 4 h and its
// gradient, 5 T and its gradient times k.  The raw values are loaded first
// (SiRaw), so that a chunk's loads are in flight while the chunk before it is
// summed, and combined later.
struct SiRaw {
  double a[10];
};
// the row's coefficients, loaded once per block
struct SiRow {
  double dycp, dycj, dyfj, hdx, hdz;  // hdx, hdz: dxi / 2 and dzi / 2
};
__device__ __forceinline__ void si_load(const TGDev &d, const IODev &io, const IOStatFields &f, int part, int64_t c,
                                        int oxp, int oxm, int64_t ozp, int64_t ozm, SiRaw &r) {
  const int64_t sy = d.sy;
  if (part < 3) {
    // the component's own staggering is along o1; 0, 1: its two faces, then
    // the face pairs of the four neighbours across
    const double *u = (part == 0 ? d.u : (part == 1 ? d.v : d.w)) + c;
    const int64_t o1 = part == 0 ? oxp : (part == 1 ? sy : ozp);
    const double *q[4] = {u + (part == 0 ? sy : oxp), u + (part == 0 ? -sy : oxm), u + (part == 2 ? sy : ozp),
                          u + (part == 2 ? -sy : ozm)};
    r.a[0] = u[0];
    r.a[1] = u[o1];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      r.a[2 + 2 * m] = q[m][0];
      r.a[3 + 2 * m] = q[m][o1];
    }
  } else if (part == 3) {
    r.a[0] = d.p[c];
    r.a[1] = f.g[0][c];
    r.a[2] = f.g[0][c + oxp];
    r.a[3] = f.g[1][c];
    r.a[4] = f.g[1][c + sy];
    r.a[5] = f.g[2][c];
    r.a[6] = f.g[2][c + ozp];
    if (io.thermal) {
      r.a[7] = io.D[c];
      r.a[8] = io.mu[c];
    }
  } else if (io.thermal) {
    const double *h = (part == 4 ? io.h : io.T) + c;
    r.a[0] = h[0];
    r.a[1] = h[oxp];
    r.a[2] = h[oxm];
    r.a[3] = h[sy];
    r.a[4] = h[-sy];
    r.a[5] = h[ozp];
    r.a[6] = h[ozm];
    if (part == 5) r.a[7] = io.kap[c];
  }
}
__device__ __forceinline__ void si_store(const TGDev &d, const IODev &io, const SiRow &y, int part, const SiRaw &r,
                                         double *b) {  // b: column of the chunk, quantities SI_CH apart
  if (part < 3) {
    const double c0 = (r.a[0] + r.a[1]) * 0.5;
    double n[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) n[m] = (r.a[2 + 2 * m] + r.a[3 + 2 * m]) * 0.5;
    double *D = b + (B_D + 3 * part) * SI_CH;
    b[(B_U + part) * SI_CH] = c0;
    const double own = r.a[1] - r.a[0];
    D[0] = part == 0 ? own * d.dxi : (n[0] - n[1]) * y.hdx;
    const double up = part == 0 ? n[0] : n[2], dn = part == 0 ? n[1] : n[3];
    D[SI_CH] = part == 1 ? own * y.dyfj : ((up - c0) * y.dycp + (c0 - dn) * y.dycj) * 0.5;
    D[2 * SI_CH] = part == 2 ? own * d.dzi : (n[2] - n[3]) * y.hdz;
  } else if (part == 3) {
    b[B_P * SI_CH] = r.a[0];
#pragma unroll
    for (int m = 0; m < 3; ++m) b[(B_G + m) * SI_CH] = (r.a[1 + 2 * m] + r.a[2 + 2 * m]) * 0.5;
    b[B_R * SI_CH] = io.thermal ? r.a[7] : 0.0;
    b[B_M * SI_CH] = io.thermal ? r.a[8] : 0.0;
  } else {
    // without the energy equation these quantities are zero
    const double *h = r.a;
    const bool th = io.thermal, iT = part == 5;
    const double kk = iT && th ? r.a[7] : 1.0;
    double *g = b + (iT ? B_DTK : B_DH) * SI_CH;
    b[(iT ? B_T : B_H) * SI_CH] = th ? h[0] : 0.0;
    g[0] = th ? (h[1] - h[2]) * y.hdx * kk : 0.0;
    g[SI_CH] = th ? ((h[3] - h[0]) * y.dycp + (h[0] - h[4]) * y.dycj) * 0.5 * kk : 0.0;
    g[2 * SI_CH] = th ? (h[5] - h[6]) * y.hdz * kk : 0.0;
  }
}

// One cell's contribution to the sums of group G.
template <int G>
__device__ __forceinline__ void si_accumulate(const double (*b)[SI_CH], int col, double (&acc)[SI_GN]) {
  int a = 0;
  double U[3], D[9];
  if (G >= 3) {
#pragma unroll
    for (int m = 0; m < 3; ++m) U[m] = b[B_U + m][col];
  }
  if (G != 5) {
#pragma unroll
    for (int l = 0; l < 9; ++l) D[l] = b[B_D + l][col];
  }
  if (G == 0) {
    const double p = b[B_P][col];
#pragma unroll
    for (int l = 0; l < 9; ++l) acc[a++] += D[l];
#pragma unroll
    for (int l = 0; l < 9; ++l) acc[a++] += D[l] * p;
#pragma unroll
    for (int l1 = 0; l1 < 3; ++l1)
#pragma unroll
      for (int l2 = l1; l2 < 9; ++l2) acc[a++] += D[l1] * D[l2];
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      const double dh = b[B_DH + m][col];
      acc[a + m] += dh;
      acc[a + 3 + m] += dh * p;
    }
  } else if (G == 1) {
    const double M = b[B_M][col];
#pragma unroll
    for (int l1 = 3; l1 < 9; ++l1)
#pragma unroll
      for (int l2 = l1; l2 < 9; ++l2) acc[a++] += D[l1] * D[l2];
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      const double e = b[B_DH + m][col] * M;
#pragma unroll
      for (int l = 0; l < 9; ++l) acc[a++] += e * D[l];
    }
  } else if (G == 2) {
    const double M = b[B_M][col], h = b[B_H][col], T = b[B_T][col], R = b[B_R][col];
    double e[3];
#pragma unroll
    for (int l = 0; l < 9; ++l) {
      const double q = D[l] * M;
      if (l < 3) e[l] = q;
      acc[l] += q;
      acc[9 + l] += q * h;
    }
    a = 18;
#pragma unroll
    for (int l1 = 0; l1 < 3; ++l1)
#pragma unroll
      for (int l2 = l1; l2 < 9; ++l2) acc[a++] += e[l1] * D[l2];
    acc[a++] += T;
    acc[a++] += R;
    acc[a++] += h;
    acc[a++] += M;
    acc[a++] += T * T;
    acc[a++] += R * R;
  } else if (G == 3) {
    const double M = b[B_M][col];
    double e[9];
#pragma unroll
    for (int l = 0; l < 9; ++l) e[l] = D[l] * M;
#pragma unroll
    for (int l1 = 3; l1 < 9; ++l1)
#pragma unroll
      for (int l2 = l1; l2 < 9; ++l2) acc[a++] += e[l1] * D[l2];
#pragma unroll
    for (int l = 0; l < 9; ++l)
#pragma unroll
      for (int m = 0; m < 3; ++m) acc[a++] += e[l] * U[m];
  } else if (G == 4) {
    const double h = b[B_H][col];
    double e[3];
#pragma unroll
    for (int m = 0; m < 3; ++m) e[m] = b[B_DTK + m][col];
#pragma unroll
    for (int m = 0; m < 3; ++m) acc[a++] += e[m];
#pragma unroll
    for (int m = 0; m < 3; ++m)
#pragma unroll
      for (int n = 0; n < 3; ++n) acc[a++] += e[m] * U[n];
#pragma unroll
    for (int m = 0; m < 3; ++m)
#pragma unroll
      for (int l = 0; l < 9; ++l) acc[a++] += e[m] * D[l];
#pragma unroll
    for (int m = 0; m < 3; ++m) acc[a++] += h * U[m];
#pragma unroll
    for (int m = 0; m < 3; ++m) acc[a++] += h * b[B_G + m][col];
    acc[a++] += h * h;
    acc[a++] += h * b[B_R][col];
    acc[a++] += h * b[B_P][col];
  } else {
    double g[3];
    const double p = b[B_P][col], rh = b[B_R][col] * b[B_H][col];
#pragma unroll
    for (int m = 0; m < 3; ++m) g[m] = b[B_G + m][col];
#pragma unroll
    for (int m = 0; m < 3; ++m) acc[a++] += U[m];
    acc[a++] += p;
#pragma unroll
    for (int m = 0; m < 3; ++m) acc[a++] += g[m];
#pragma unroll
    for (int m = 0; m < 3; ++m) acc[a++] += U[m] * p;
#pragma unroll
    for (int m = 0; m < 3; ++m)
#pragma unroll
      for (int n = m; n < 3; ++n) acc[a++] += U[m] * U[n];
#pragma unroll
    for (int m = 0; m < 3; ++m)
#pragma unroll
      for (int n = m; n < 3; ++n) acc[a++] += U[m] * g[n];
#pragma unroll
    for (int m = 0; m < 3; ++m)
#pragma unroll
      for (int n = m; n < 3; ++n) {
        const double uu = U[m] * U[n];
#pragma unroll
        for (int h = n; h < 3; ++h) acc[a++] += uu * U[h];
      }
#pragma unroll
    for (int m = 0; m < 3; ++m)
#pragma unroll
      for (int n = m; n < 3; ++n) {
        const double ug = U[m] * g[n];
#pragma unroll
        for (int h = n; h < 3; ++h) acc[a++] += ug * U[h];
      }
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      const double ru = rh * U[m];
#pragma unroll
      for (int n = m; n < 3; ++n) acc[a++] += ru * U[n];
    }
  }
}

// Partial sums of one row and k-chunk.  A block of twelve warps walks its
// cells in chunks of 64: 6 x 64 threads load and combine the per-cell
// quantities of the next chunk into the other half of shared memory while
// each warp adds half of the current chunk to one group's sums (two warps per
// group, one per 32 cells).  Every quantity is formed once per cell, every
// product once, and the sums stay in registers: about 330 FP64 operations and
// 80 shared-memory loads per cell.  What bounds it is the issue of those and
// of the address arithmetic by the twelve warps that the registers allow
// (1.7 instructions per cycle; FP64 pipe 23 %, DRAM 10 % busy).  A sample of
// the 384x192x192 channel with both averages read back takes 1.79 ms; the
// generic kernel that looked up the factors of each of the 360 products took
// 8.86 ms.  Group copies of the whole loop overflow the instruction cache
// (2.8x slower).
__global__ void __launch_bounds__(SI_TPB, 1) k_io_stats_part(TGDev d, IODev io, IOStatFields f, double *part) {
  __shared__ double b[2][SI_NB][SI_CH];
  __shared__ double red[2][SI_NS];
  const int j = blockIdx.x + 1, nx = d.nx, nz = d.nz;
  const int k0 = (int)((int64_t)nz * blockIdx.y / ST_NBK), k1 = (int)((int64_t)nz * (blockIdx.y + 1) / ST_NBK);
  const int ncell = nx * (k1 - k0);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = w % SI_NG, half = w / SI_NG;
  const int slice = threadIdx.x / SI_CH, col = threadIdx.x % SI_CH;
  const SiRow y{d.dyci[j + 1], d.dyci[j], d.dyfi[j], d.dxi * 0.5, d.dzi * 0.5};
  // this thread's cell of the chunk being loaded, advanced by 64 cells a chunk
  const int di = SI_CH % nx, dk = SI_CH / nx;
  int i = col % nx, k = k0 + col / nx;
  const int64_t wrapz = d.sz * (nz - 1), row = d.sy * j;
  auto load = [&](SiRaw &r) {
    si_load(d, io, f, slice, i + row + d.sz * k, i + 1 == nx ? 1 - nx : 1, i == 0 ? nx - 1 : -1,
            k + 1 == nz ? -wrapz : d.sz, k == 0 ? wrapz : -d.sz, r);
  };
  double acc[SI_GN];
#pragma unroll
  for (int a = 0; a < SI_GN; ++a) acc[a] = 0.0;
  SiRaw r;
  if (k < k1) {
    load(r);
    si_store(d, io, y, slice, r, &b[0][0][col]);
  }
  __syncthreads();
  int buf = 0;
  const int c = half * 32 + lane;
  for (int t0 = 0; t0 < ncell; t0 += SI_CH) {
    i += di;
    k += dk;
    if (i >= nx) {
      i -= nx;
      ++k;
    }
    const bool more = k < k1;
    if (more) load(r);
    if (t0 + c < ncell) switch (g) {  // warp-uniform
        case 0: si_accumulate<0>(b[buf], c, acc); break;
        case 1: si_accumulate<1>(b[buf], c, acc); break;
        case 2: si_accumulate<2>(b[buf], c, acc); break;
        case 3: si_accumulate<3>(b[buf], c, acc); break;
        case 4: si_accumulate<4>(b[buf], c, acc); break;
        default: si_accumulate<5>(b[buf], c, acc); break;
      }
    buf ^= 1;
    if (more) si_store(d, io, y, slice, r, &b[buf][0][col]);
    __syncthreads();
  }
#pragma unroll
  for (int a = 0; a < SI_GN; ++a) {
    double v = acc[a];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) red[half][SI_GN * g + a] = v;
  }
  __syncthreads();
  for (int a = threadIdx.x; a < SI_NS; a += SI_TPB)
    part[((size_t)(j - 1) * ST_NBK + blockIdx.y) * SI_NS + a] = red[0][a] + red[1][a];
}

// Sum the k-chunk partials of each row in order, scale by 1/(nx nz) and
// (accumulate != 0) fold into the time average.
__global__ void k_io_stats_final(int nx, int nz, const double *part, const uint16_t *source, double *xz, double *xzt,
                                 double coe2, double coe3, int accumulate) {
  const int j = blockIdx.x + 1;
  const double vl = 1.0 / ((double)nx * (double)nz);
  for (int a = threadIdx.x; a < SI_NV; a += blockDim.x) {
    double s = 0.0;
    const int src = source[a];
    for (int b = 0; b < ST_NBK; ++b) s += part[((size_t)(j - 1) * ST_NBK + b) * SI_NS + src];
    const double val = s * vl;
    xz[(size_t)(j - 1) * SI_NV + a] = val;
    if (accumulate) {
      double *t = xzt + (size_t)(j - 1) * SI_NV + a;
      *t = coe3 * *t + coe2 * val;
    }
  }
}

// Values per row and partials per row of the context's statistics.
int nv_of(const chapsim_ctx *c) { return c->domain == CHAPSIM_IIO ? SI_NV : ST_NV; }
size_t npart_of(const chapsim_ctx *c) {
  return (size_t)c->d.ny * ST_NBK * (c->domain == CHAPSIM_IIO ? SI_NS : ST_G0 + ST_G1);
}

}  // namespace

int stats_run(chapsim_ctx *c, int accumulate) {
  if (c->domain == CHAPSIM_IIO) {
    TGDev &d = c->d;
    const size_t np = npart_of(c), nv = (size_t)d.ny * SI_NV;
    if (!c->stats_buf) {
      void *p = nullptr;
      // partials, xz, xzt, then the table of the output values' sums
      CK(cudaMalloc(&p, (np + 2 * nv) * sizeof(double) + SI_NV * sizeof(uint16_t)));
      c->allocs.push_back(p);
      c->stats_buf = (double *)p;
      CK(cudaMemsetAsync(p, 0, (np + 2 * nv) * sizeof(double), c->stream));
      const std::vector<uint16_t> t = io_source();
      CK(cudaMemcpyAsync(c->stats_buf + np + 2 * nv, t.data(), SI_NV * sizeof(uint16_t), cudaMemcpyHostToDevice,
                         c->stream));
      CK(cudaStreamSynchronize(c->stream));  // the host table goes out of scope
    }
    double *part = c->stats_buf, *xz = part + np, *xzt = xz + nv;
    const uint16_t *source = reinterpret_cast<const uint16_t *>(xzt + nv);
    IOStatFields f;
    for (int m = 0; m < 3; ++m) f.g[m] = c->io.g[c->io_cur][m];
    k_io_stats_part<<<dim3(d.ny, ST_NBK), SI_TPB, 0, c->stream>>>(d, c->io, f, part);
    LAUNCHED();
    double coe2 = 0.0, coe3 = 0.0;
    if (accumulate) {  // T_Asymptotic_Average
      c->nstatis += 1;
      coe2 = 1.0 / (double)c->nstatis;
      coe3 = (double)(c->nstatis - 1) / (double)c->nstatis;
    }
    k_io_stats_final<<<d.ny, 128, 0, c->stream>>>(d.nx, d.nz, part, source, xz, xzt, coe2, coe3, accumulate);
    LAUNCHED();
    return CHAPSIM_OK;
  }
  TGDev &d = c->d;
  if (!c->stats_buf) {
    const size_t np = (size_t)d.ny * ST_NBK * (ST_G0 + ST_G1), nv = (size_t)d.ny * ST_NV;
    void *p = nullptr;
    CK(cudaMalloc(&p, (np + 2 * nv) * sizeof(double)));
    c->allocs.push_back(p);
    c->stats_buf = (double *)p;
    CK(cudaMemsetAsync(p, 0, (np + 2 * nv) * sizeof(double), c->stream));
  }
  double *part = c->stats_buf, *xz = part + (size_t)d.ny * ST_NBK * (ST_G0 + ST_G1), *xzt = xz + (size_t)d.ny * ST_NV;
  k_stats_part<0><<<dim3(d.ny, ST_NBK), ST_TPB, 0, c->stream>>>(d, part);
  LAUNCHED();
  k_stats_part<1><<<dim3(d.ny, ST_NBK), ST_TPB, 0, c->stream>>>(d, part);
  LAUNCHED();
  double coe2 = 0.0, coe3 = 0.0;
  if (accumulate) {  // T_Asymptotic_Average
    c->nstatis += 1;
    coe2 = 1.0 / (double)c->nstatis;
    coe3 = (double)(c->nstatis - 1) / (double)c->nstatis;
  }
  k_stats_final<<<d.ny, 128, 0, c->stream>>>(d, part, xz, xzt, coe2, coe3, accumulate);
  LAUNCHED();
  return CHAPSIM_OK;
}

int stats_reset(chapsim_ctx *c) {
  c->nstatis = 0;
  if (!c->stats_buf) return CHAPSIM_OK;
  const size_t nv = (size_t)c->d.ny * nv_of(c);
  double *xzt = c->stats_buf + npart_of(c) + nv;
  CK(cudaMemsetAsync(xzt, 0, nv * sizeof(double), c->stream));
  return CHAPSIM_OK;
}

int stats_get(chapsim_ctx *c, int which, double *host, int64_t n) {
  TGDev &d = c->d;
  if (!c->stats_buf || n != (int64_t)d.ny * nv_of(c)) return CHAPSIM_ERR_ARG;
  const double *xz = c->stats_buf + npart_of(c);
  const double *src = which == 0 ? xz : xz + (size_t)d.ny * nv_of(c);
  CK(cudaMemcpyAsync(host, src, (size_t)n * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
  CK(cudaStreamSynchronize(c->stream));
  return CHAPSIM_OK;
}

}  // namespace chapsim
