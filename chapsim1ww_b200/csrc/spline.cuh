// Table cubic splines shared by the property engine and the IO energy
// path: the Forsythe-Malcolm-Moler spline of CUBIC_SPLINE
// (src/Flow_State.f90:1693-1787) built on the host, evaluated on the device
// with the binary search of NIST_SLEVAL_* (src/Flow_State.f90:1015-1070)
// started from a uniform bucket table.
#pragma once
#include <cuda_runtime.h>

#include <vector>

namespace chapsim_spl {

// Spline of y over x: coefficients b, c, d (Forsythe, Malcolm & Moler),
// also packed per interval as one 32-byte record {y, b, c, d}.
struct Spline {
  const double *x, *y, *b, *c, *d;
  const double4 *ybcd;
  const int *blo;    // bucket -> first candidate interval
  const int2 *brng;  // bucket -> search range {blo[b], min(n - 1, blo[b + 1] + 3)}
  double x0, binv;
  double xlo, xhi;   // x[0] and x[n - 1], held by value for the range test
  int n, nb;
};

// Interval i with x[i] <= u < x[i+1] (u strictly inside the table); the
// bucket gives a short range for the same binary search as the reference.
__device__ __forceinline__ int spline_find(const Spline &s, double u) {
  int b = (int)((u - s.x0) * s.binv);
  b = b < 0 ? 0 : (b >= s.nb ? s.nb - 1 : b);
  const int2 rg = __ldg(s.brng + b);
  int i = rg.x, j = rg.y;
  while (j > i + 1) {
    const int k = (i + j) >> 1;
    if (u < __ldg(s.x + k)) j = k; else i = k;
  }
  return i;
}
__device__ __forceinline__ double spline_at(const Spline &s, int i, double u) {
  const double2 r0 = __ldg(reinterpret_cast<const double2 *>(s.ybcd + i));
  const double2 r1 = __ldg(reinterpret_cast<const double2 *>(s.ybcd + i) + 1);
  const double4 r = make_double4(r0.x, r0.y, r1.x, r1.y);
  const double dx = u - __ldg(s.x + i);
  return r.x + dx * (r.y + dx * (r.z + dx * r.w));
}

// ---------------------------------------------------------------- IO tables
// The table of an IO context, laid out for look-ups by a warp of cells whose
// enthalpies lie within a hundred or so intervals.  The L1 cache serves a
// gather one 128-byte line per cycle, so a look-up costs the lines that its
// gathers touch: coefficients sit in arrays of pairs (a hundred intervals are
// 13 lines; records of a whole interval are 26 to 100), the search starts
// from one 4-byte index per bucket, and the caller keeps the last interval's
// values (Poly), so that a second look-up in it loads nothing.
struct PropTable {
  const int *hb, *tb;                 // bucket of the uniform search grid -> first candidate interval
  const double *hx, *tx;              // the grids of h and T
  const double2 *hc[2];               // T(h): {c0, c1}, {c2, c3} per interval
  const double2 *rho[2], *mu[2], *k[2];  // of T
  double h0, hbinv, t0, tbinv;
  double hlo, hhi, tlo, thi;
  int n, nb;
};

__device__ __forceinline__ bool inside_h(const PropTable &p, double h) { return h > p.hlo && h < p.hhi; }
__device__ __forceinline__ bool inside_t(const PropTable &p, double T) { return T > p.tlo && T < p.thi; }

// One interval [x, xn) and the coefficients of one function on it:
// c0 + dx (c1 + dx (c2 + dx c3)), dx = u - x.
struct Poly {
  double x, xn;
  double2 a, b;
  __device__ __forceinline__ bool holds(double u) const { return u >= x && u < xn; }
  __device__ __forceinline__ double at(double u) const {
    const double dx = u - x;
    return a.x + dx * (a.y + dx * (b.x + dx * b.y));
  }
  __device__ __forceinline__ void coef(const double2 *const (&c)[2], int i) {
    a = __ldg(c[0] + i);
    b = __ldg(c[1] + i);
  }
  // Interval i with x[i] <= u < x[i + 1], u strictly inside the table: from
  // the bucket's first candidate a few steps up, then by bisection (tables
  // whose points crowd into few buckets).
  __device__ __forceinline__ int find(const int *bucket, int nb, double x0, double binv, const double *grid, int n,
                                      double u) {
    int q = (int)((u - x0) * binv);
    q = q < 0 ? 0 : (q >= nb ? nb - 1 : q);
    int i = __ldg(bucket + q);
    x = __ldg(grid + i);
    xn = __ldg(grid + i + 1);
#pragma unroll 1
    for (int step = 0; u >= xn; ++step) {
      if (step == 4) {
        int j = n - 1;
        ++i;
        while (j > i + 1) {
          const int m = (i + j) >> 1;
          if (u < __ldg(grid + m)) j = m; else i = m;
        }
        x = __ldg(grid + i);
        xn = __ldg(grid + i + 1);
        break;
      }
      ++i;
      x = xn;
      xn = __ldg(grid + i + 1);
    }
    return i;
  }
};

__device__ __forceinline__ bool inside(const Spline &s, double u) { return u > s.xlo && u < s.xhi; }


// Host restatement of CUBIC_SPLINE (Forsythe-Malcolm-Moler, 1977).
inline void fmm_spline(int n, const double *x, const double *y, double *b, double *c, double *d) {
  const int nm1 = n - 1;
  d[0] = x[1] - x[0];
  c[1] = (y[1] - y[0]) / d[0];
  for (int i = 1; i < nm1; ++i) {
    d[i] = x[i + 1] - x[i];
    b[i] = 2.0 * (d[i - 1] + d[i]);
    c[i + 1] = (y[i + 1] - y[i]) / d[i];
    c[i] = c[i + 1] - c[i];
  }
  b[0] = -d[0];
  b[n - 1] = -d[n - 2];
  c[0] = 0.0;
  c[n - 1] = 0.0;
  if (n > 3) {
    c[0] = c[2] / (x[3] - x[1]) - c[1] / (x[2] - x[0]);
    c[n - 1] = c[n - 2] / (x[n - 1] - x[n - 3]) - c[n - 3] / (x[n - 2] - x[n - 4]);
    c[0] = c[0] * d[0] * d[0] / (x[3] - x[0]);
    c[n - 1] = -c[n - 1] * d[n - 2] * d[n - 2] / (x[n - 1] - x[n - 4]);
  }
  for (int i = 1; i < n; ++i) {
    const double t = d[i - 1] / b[i - 1];
    b[i] = b[i] - t * d[i - 1];
    c[i] = c[i] - t * c[i - 1];
  }
  c[n - 1] = c[n - 1] / b[n - 1];
  for (int l = 1; l <= nm1; ++l) {
    const int i = n - 1 - l;
    c[i] = (c[i] - d[i] * c[i + 1]) / b[i];
  }
  b[n - 1] = (y[n - 1] - y[nm1 - 1]) / d[nm1 - 1] + d[nm1 - 1] * (c[nm1 - 1] + 2.0 * c[n - 1]);
  for (int i = 0; i < nm1; ++i) {
    b[i] = (y[i + 1] - y[i]) / d[i] - d[i] * (c[i + 1] + 2.0 * c[i]);
    d[i] = (c[i + 1] - c[i]) / d[i];
    c[i] = 3.0 * c[i];
  }
  c[n - 1] = 3.0 * c[n - 1];
  d[n - 1] = d[n - 2];
}

// Bucket table over nb uniform buckets of [x_1, x_n]: blo[b] = I(start_b) - 1
// with I(v) = max{i : x_i <= v}, so every u in bucket b satisfies
// x[blo[b]] <= u < x[min(n-1, blo[b+1] + 3)] (one interval of slack each way
// for rounding); the binary search between them finds the reference's i.
inline void bucket_table(int n, const double *x, int nb, double &x0, double &binv, std::vector<int> &blo) {
  x0 = x[0];
  binv = nb / (x[n - 1] - x[0]);
  blo.assign(nb + 1, 0);
  int i = 0;
  for (int b = 0; b <= nb; ++b) {
    const double start = x0 + b / binv;
    while (i + 1 < n && x[i + 1] <= start) ++i;
    int l = i - 1;
    l = l < 0 ? 0 : l;
    blo[b] = l < n - 2 ? l : n - 2;
  }
}


// Search range of each bucket for spline_find: {blo[b], min(n - 1, blo[b + 1] + 3)}.
inline std::vector<int2> bucket_ranges(const std::vector<int> &blo, int n, int nb) {
  std::vector<int2> rng(nb);
  for (int q = 0; q < nb; ++q) rng[q] = make_int2(blo[q], blo[q + 1] + 3 < n - 1 ? blo[q + 1] + 3 : n - 1);
  return rng;
}

// First candidate interval of nb uniform buckets: the last one that starts
// before the bucket, with a margin of 2^-48 of the table's width, far above
// the rounding of the bucket index.
inline std::vector<int> first_intervals(int n, const double *x, int nb, double &x0, double &binv) {
  x0 = x[0];
  binv = nb / (x[n - 1] - x[0]);
  const double tol = (x[n - 1] - x[0]) * 0x1p-48;
  std::vector<int> f(nb);
  int i = 0;
  for (int b = 0; b < nb; ++b) {
    const double start = x0 + b / binv - tol;
    while (i + 2 < n && x[i + 1] <= start) ++i;
    f[b] = i;
  }
  return f;
}

// Build the IO table of T(h), rho(T), mu(T), k(T) (FMM splines) on the host
// and upload it; every allocation is appended to allocs (freed by the owner).
inline cudaError_t upload_props(std::vector<void *> &allocs, const std::vector<double> &H, const std::vector<double> &T,
                                const std::vector<double> &D, const std::vector<double> &M,
                                const std::vector<double> &K, PropTable &p) {
  const int n = (int)H.size();
  auto up = [&](const void *src, size_t bytes, const void **dst) {
    void *q = nullptr;
    cudaError_t e = cudaMalloc(&q, bytes);
    if (e != cudaSuccess) return e;
    allocs.push_back(q);
    *dst = q;
    return cudaMemcpy(q, src, bytes, cudaMemcpyHostToDevice);
  };
  auto fit = [&](const std::vector<double> &x, const std::vector<double> &y, const double2 *(&c)[2]) {
    std::vector<double> b(n), cc(n), d(n);
    fmm_spline(n, x.data(), y.data(), b.data(), cc.data(), d.data());
    std::vector<double2> lo(n), hi(n);
    for (int i = 0; i < n; ++i) {
      lo[i] = make_double2(y[i], b[i]);
      hi[i] = make_double2(cc[i], d[i]);
    }
    const cudaError_t e = up(lo.data(), n * sizeof(double2), (const void **)&c[0]);
    return e != cudaSuccess ? e : up(hi.data(), n * sizeof(double2), (const void **)&c[1]);
  };
  p.n = n;
  p.nb = 4 * n;
  const std::vector<int> hb = first_intervals(n, H.data(), p.nb, p.h0, p.hbinv),
                         tb = first_intervals(n, T.data(), p.nb, p.t0, p.tbinv);
  p.hlo = H[0]; p.hhi = H[n - 1];
  p.tlo = T[0]; p.thi = T[n - 1];
  cudaError_t e;
  if ((e = fit(H, T, p.hc)) != cudaSuccess || (e = fit(T, D, p.rho)) != cudaSuccess ||
      (e = fit(T, M, p.mu)) != cudaSuccess || (e = fit(T, K, p.k)) != cudaSuccess)
    return e;
  if ((e = up(hb.data(), hb.size() * sizeof(int), (const void **)&p.hb)) != cudaSuccess) return e;
  if ((e = up(tb.data(), tb.size() * sizeof(int), (const void **)&p.tb)) != cudaSuccess) return e;
  if ((e = up(H.data(), n * sizeof(double), (const void **)&p.hx)) != cudaSuccess) return e;
  return up(T.data(), n * sizeof(double), (const void **)&p.tx);
}

}  // namespace chapsim_spl
