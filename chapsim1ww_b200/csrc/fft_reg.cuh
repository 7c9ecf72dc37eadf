// Register-blocked complex FP64 transforms: a line of n = R0 R1 (R2) points
// passes through two or three stages of one large radix each.  A thread holds
// a whole butterfly (up to 16 points) in registers; the first stage takes its
// points straight from global memory and the last one writes its results
// there, so that a two-stage line crosses shared memory once.
//
// The stages are those of the self-sorting Stockham transform (fft_smem.cuh):
// stage s with radix R and Ns = product of the earlier radices maps, for j in
// [0, n / R),
//   v_r = in[j + r n / R] w^{r (j mod Ns) n / (Ns R)},  V = DFT_R(v),
//   out[(j / Ns) Ns R + (j mod Ns) + s Ns] = V_s.
// Composite radices split once more inside the registers (Cooley-Tukey), odd
// prime ones pair the points r and R - r (cosines multiply sums, sines
// differences: a quarter of the multiplications of the plain sum).
#pragma once
#include <cuda_runtime.h>

#include "chapsim_internal.cuh"
#include "fft_smem.cuh"

namespace chapsim {

// cos and sin of 2 pi m / R for the radices below
template <int R> __host__ __device__ constexpr double dft_cos(int m);
template <int R> __host__ __device__ constexpr double dft_sin(int m);
template <> __host__ __device__ constexpr double dft_cos<3>(int m) {
  constexpr double t[3] = {1.0, -0.5, -0.5};
  return t[m];
}
template <> __host__ __device__ constexpr double dft_sin<3>(int m) {
  constexpr double t[3] = {0.0, 0.8660254037844386, -0.8660254037844386};
  return t[m];
}
template <> __host__ __device__ constexpr double dft_cos<5>(int m) {
  constexpr double t[5] = {1.0, 0.30901699437494745, -0.8090169943749475, -0.8090169943749475, 0.30901699437494745};
  return t[m];
}
template <> __host__ __device__ constexpr double dft_sin<5>(int m) {
  constexpr double t[5] = {0.0, 0.9510565162951535, 0.5877852522924731, -0.5877852522924731, -0.9510565162951535};
  return t[m];
}
template <> __host__ __device__ constexpr double dft_cos<6>(int m) {
  constexpr double t[6] = {1.0, 0.5, -0.5, -1.0, -0.5, 0.5};
  return t[m];
}
template <> __host__ __device__ constexpr double dft_sin<6>(int m) {
  constexpr double t[6] = {0.0, 0.8660254037844386, 0.8660254037844386, 0.0, -0.8660254037844386,
                           -0.8660254037844386};
  return t[m];
}
template <> __host__ __device__ constexpr double dft_cos<7>(int m) {
  constexpr double t[7] = {1.0, 0.6234898018587335, -0.2225209339563144, -0.9009688679024191, -0.9009688679024191,
                           -0.2225209339563144, 0.6234898018587335};
  return t[m];
}
template <> __host__ __device__ constexpr double dft_sin<7>(int m) {
  constexpr double t[7] = {0.0, 0.7818314824680298, 0.9749279121818236, 0.4338837391175581, -0.4338837391175581,
                           -0.9749279121818236, -0.7818314824680298};
  return t[m];
}
template <> __host__ __device__ constexpr double dft_cos<9>(int m) {
  constexpr double t[9] = {1.0, 0.766044443118978, 0.17364817766693036, -0.5, -0.9396926207859084,
                           -0.9396926207859084, -0.5, 0.17364817766693036, 0.766044443118978};
  return t[m];
}
template <> __host__ __device__ constexpr double dft_sin<9>(int m) {
  constexpr double t[9] = {0.0, 0.6427876096865394, 0.984807753012208, 0.8660254037844386, 0.3420201433256687,
                           -0.3420201433256687, -0.8660254037844386, -0.984807753012208, -0.6427876096865394};
  return t[m];
}
template <> __host__ __device__ constexpr double dft_cos<10>(int m) {
  constexpr double t[10] = {1.0, 0.8090169943749475, 0.30901699437494745, -0.30901699437494745,
                           -0.8090169943749475, -1.0, -0.8090169943749475, -0.30901699437494745,
                           0.30901699437494745, 0.8090169943749475};
  return t[m];
}
template <> __host__ __device__ constexpr double dft_sin<10>(int m) {
  constexpr double t[10] = {0.0, 0.5877852522924731, 0.9510565162951535, 0.9510565162951535, 0.5877852522924731,
                           0.0, -0.5877852522924731, -0.9510565162951535, -0.9510565162951535, -0.5877852522924731};
  return t[m];
}
template <> __host__ __device__ constexpr double dft_cos<11>(int m) {
  constexpr double t[11] = {1.0, 0.8412535328311812, 0.41541501300188644, -0.14231483827328514,
                           -0.6548607339452851, -0.9594929736144974, -0.9594929736144974, -0.6548607339452851,
                           -0.14231483827328514, 0.41541501300188644, 0.8412535328311812};
  return t[m];
}
template <> __host__ __device__ constexpr double dft_sin<11>(int m) {
  constexpr double t[11] = {0.0, 0.5406408174555976, 0.9096319953545183, 0.9898214418809327, 0.7557495743542583,
                           0.28173255684142967, -0.28173255684142967, -0.7557495743542583, -0.9898214418809327,
                           -0.9096319953545183, -0.5406408174555976};
  return t[m];
}
template <> __host__ __device__ constexpr double dft_cos<12>(int m) {
  constexpr double t[12] = {1.0, 0.8660254037844386, 0.5, 0.0, -0.5, -0.8660254037844386, -1.0,
                           -0.8660254037844386, -0.5, 0.0, 0.5, 0.8660254037844386};
  return t[m];
}
template <> __host__ __device__ constexpr double dft_sin<12>(int m) {
  constexpr double t[12] = {0.0, 0.5, 0.8660254037844386, 1.0, 0.8660254037844386, 0.5, 0.0, -0.5,
                           -0.8660254037844386, -1.0, -0.8660254037844386, -0.5};
  return t[m];
}
template <> __host__ __device__ constexpr double dft_cos<14>(int m) {
  constexpr double t[14] = {1.0, 0.9009688679024191, 0.6234898018587335, 0.2225209339563144, -0.2225209339563144,
                           -0.6234898018587335, -0.9009688679024191, -1.0, -0.9009688679024191,
                           -0.6234898018587335, -0.2225209339563144, 0.2225209339563144, 0.6234898018587335,
                           0.9009688679024191};
  return t[m];
}
template <> __host__ __device__ constexpr double dft_sin<14>(int m) {
  constexpr double t[14] = {0.0, 0.4338837391175581, 0.7818314824680298, 0.9749279121818236, 0.9749279121818236,
                           0.7818314824680298, 0.4338837391175581, 0.0, -0.4338837391175581, -0.7818314824680298,
                           -0.9749279121818236, -0.9749279121818236, -0.7818314824680298, -0.4338837391175581};
  return t[m];
}
template <> __host__ __device__ constexpr double dft_cos<15>(int m) {
  constexpr double t[15] = {1.0, 0.9135454576426009, 0.6691306063588582, 0.30901699437494745, -0.10452846326765347,
                           -0.5, -0.8090169943749475, -0.9781476007338057, -0.9781476007338057,
                           -0.8090169943749475, -0.5, -0.10452846326765347, 0.30901699437494745,
                           0.6691306063588582, 0.9135454576426009};
  return t[m];
}
template <> __host__ __device__ constexpr double dft_sin<15>(int m) {
  constexpr double t[15] = {0.0, 0.4067366430758002, 0.7431448254773942, 0.9510565162951535, 0.9945218953682733,
                           0.8660254037844386, 0.5877852522924731, 0.20791169081775934, -0.20791169081775934,
                           -0.5877852522924731, -0.8660254037844386, -0.9945218953682733, -0.9510565162951535,
                           -0.7431448254773942, -0.4067366430758002};
  return t[m];
}
template <> __host__ __device__ constexpr double dft_cos<16>(int m) {
  constexpr double t[16] = {1.0, 0.9238795325112867, 0.7071067811865476, 0.3826834323650898, 0.0,
                           -0.3826834323650898, -0.7071067811865476, -0.9238795325112867, -1.0,
                           -0.9238795325112867, -0.7071067811865476, -0.3826834323650898, 0.0, 0.3826834323650898,
                           0.7071067811865476, 0.9238795325112867};
  return t[m];
}
template <> __host__ __device__ constexpr double dft_sin<16>(int m) {
  constexpr double t[16] = {0.0, 0.3826834323650898, 0.7071067811865476, 0.9238795325112867, 1.0,
                           0.9238795325112867, 0.7071067811865476, 0.3826834323650898, 0.0, -0.3826834323650898,
                           -0.7071067811865476, -0.9238795325112867, -1.0, -0.9238795325112867,
                           -0.7071067811865476, -0.3826834323650898};
  return t[m];
}

// v <- DFT_R(v) with root exp(SG 2 pi i / R), natural order in and out
template <int R, int SG> struct Dft;

template <int SG> struct Dft<2, SG> {
  static __device__ __forceinline__ void run(double2 (&v)[2]) {
    const double2 a = v[0];
    v[0] = cadd(a, v[1]);
    v[1] = csub(a, v[1]);
  }
};
template <int SG> struct Dft<4, SG> {
  static __device__ __forceinline__ void run(double2 (&v)[4]) { dft4(v[0], v[1], v[2], v[3], SG); }
};
template <int SG> struct Dft<8, SG> {
  static __device__ __forceinline__ void run(double2 (&v)[8]) { dft_small<double2, 8>(v, nullptr, 8, SG); }
};
// odd prime
template <int R, int SG> struct DftPrime {
  static __device__ __forceinline__ void run(double2 (&v)[R]) {
    constexpr int H = (R - 1) / 2;
    double2 s[H], d[H];
    double2 x0 = v[0];
#pragma unroll
    for (int r = 0; r < H; ++r) {
      s[r] = cadd(v[r + 1], v[R - 1 - r]);
      d[r] = csub(v[r + 1], v[R - 1 - r]);
      x0 = cadd(x0, s[r]);
    }
#pragma unroll
    for (int k = 1; k <= H; ++k) {
      double2 a = v[0], b = make_double2(0.0, 0.0);
#pragma unroll
      for (int r = 0; r < H; ++r) {
        const double c = dft_cos<R>((r + 1) * k % R), q = SG * dft_sin<R>((r + 1) * k % R);
        a.x += c * s[r].x;
        a.y += c * s[r].y;
        b.x -= q * d[r].y;  // i q d
        b.y += q * d[r].x;
      }
      // k and R - k: a +- b; the sums s, d are still needed, so v[1..] is
      // rewritten only here
      v[k] = cadd(a, b);
      v[R - k] = csub(a, b);
    }
    v[0] = x0;
  }
};
template <int SG> struct Dft<3, SG> : DftPrime<3, SG> {};
template <int SG> struct Dft<5, SG> : DftPrime<5, SG> {};
template <int SG> struct Dft<7, SG> : DftPrime<7, SG> {};
template <int SG> struct Dft<11, SG> : DftPrime<11, SG> {};
// R = A B: columns of A, twiddles, rows of B
template <int A, int B, int SG> struct DftSplit {
  static __device__ __forceinline__ void run(double2 (&v)[A * B]) {
    constexpr int R = A * B;
    double2 y[B][A];
#pragma unroll
    for (int q = 0; q < B; ++q) {
#pragma unroll
      for (int p = 0; p < A; ++p) y[q][p] = v[B * p + q];
      Dft<A, SG>::run(y[q]);
#pragma unroll
      for (int p = 1; p < A; ++p)
        if (q) y[q][p] = cmul(y[q][p], make_double2(dft_cos<R>(q * p), SG * dft_sin<R>(q * p)));
    }
#pragma unroll
    for (int p = 0; p < A; ++p) {
      double2 z[B];
#pragma unroll
      for (int q = 0; q < B; ++q) z[q] = y[q][p];
      Dft<B, SG>::run(z);
#pragma unroll
      for (int q = 0; q < B; ++q) v[p + A * q] = z[q];
    }
  }
};
template <int SG> struct Dft<6, SG> : DftSplit<2, 3, SG> {};
template <int SG> struct Dft<9, SG> : DftSplit<3, 3, SG> {};
template <int SG> struct Dft<10, SG> : DftSplit<2, 5, SG> {};
template <int SG> struct Dft<12, SG> : DftSplit<4, 3, SG> {};
template <int SG> struct Dft<14, SG> : DftSplit<2, 7, SG> {};
template <int SG> struct Dft<15, SG> : DftSplit<3, 5, SG> {};
template <int SG> struct Dft<16, SG> : DftSplit<4, 4, SG> {};

// The plan of n points: two radices up to `most`, else three (up to 16 where
// `most` does not suffice), chosen for the smallest largest one (registers),
// then the smallest sum.
inline RegPlan reg_plan(int n, int most = 16) {
  static const int rad[] = {2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 14, 15, 16};
  RegPlan p{n, 0, 0, {1, 1, 1}, nullptr};
  int best = 1 << 30;
  auto take = [&](int a, int b, int c) {
    const int m = a > b ? (a > c ? a : c) : (b > c ? b : c), cost = 64 * m + a + b + c;
    if (m > most || cost >= best) return;
    best = cost;
    p.nst = c > 1 ? 3 : 2;
    p.rmax = m;
    p.R[0] = a;
    p.R[1] = b;
    p.R[2] = c;
  };
  for (int a : rad)
    for (int b : rad)
      if (a * b == n) take(a, b, 1);
  if (p.nst) return p;
  for (int a : rad)
    for (int b : rad)
      for (int c : rad)
        if (a * b * c == n) take(a, b, c);
  if (!p.nst && most < 16) return reg_plan(n);
  return p;
}

// Butterflies of the stage that has most: threads per line
inline int reg_per(const RegPlan &p) {
  if (!p.nst) return 0;
  int m = p.R[0] < p.R[1] ? p.R[0] : p.R[1];
  if (p.nst == 3 && p.R[2] < m) m = p.R[2];
  return p.n / m;
}

// f(integral constant R) for the plan's radix r, R <= RMAX
template <int R> struct RadixTag { static constexpr int value = R; };
template <int RMAX, typename F> __device__ __forceinline__ void with_radix(int r, F f) {
  switch (r) {
    case 2: f(RadixTag<2>()); break;
    case 3: f(RadixTag<3>()); break;
    case 4: f(RadixTag<4>()); break;
    case 5: f(RadixTag<5>()); break;
    case 6: f(RadixTag<6>()); break;
    case 7: f(RadixTag<7>()); break;
    case 8: f(RadixTag<8>()); break;
    case 9: if (RMAX > 8) f(RadixTag<9>()); break;
    case 10: if (RMAX > 8) f(RadixTag<10>()); break;
    case 11: if (RMAX > 8) f(RadixTag<11>()); break;
    case 12: if (RMAX > 8) f(RadixTag<12>()); break;
    case 14: if (RMAX > 8) f(RadixTag<14>()); break;
    case 15: if (RMAX > 8) f(RadixTag<15>()); break;
    case 16: if (RMAX > 8) f(RadixTag<16>()); break;
  }
}

// v_r *= w^{r m}, table entries (exp(-2 pi i m / n)); r m < n
template <int R, int SG> __device__ __forceinline__ void reg_twiddle(double2 (&v)[R], const double2 *__restrict__ tw, int m) {
#pragma unroll
  for (int r = 1; r < R; ++r) {
    double2 t = __ldg(tw + r * m);
    if (SG > 0) t.y = -t.y;
    v[r] = cmul(v[r], t);
  }
}

// Position of element p of a line-major buffer: the low three bits XORed with
// the two groups of three above them, a permutation inside every aligned
// group of eight. The first stage writes at stride R (8 or 16 elements of 16
// bytes); permuted, those writes and the contiguous reads spread over all
// banks.
__device__ __forceinline__ int swz2(int p) { return p ^ ((p >> 3) & 7) ^ ((p >> 6) & 7); }

// One line of pl.n points at `base` of the buffer A, butterfly j of every
// stage by the calling thread: load(i) gives point i, store(k, value) takes
// result k.  Every thread of the block calls it (act: the line exists).  KEEP
// puts a barrier before the stores, for a store that writes A.
template <int RMAX, int SG, bool KEEP, typename L, typename S>
__device__ __forceinline__ void reg_line(const RegPlan &pl, double2 *A, int base, int j, bool act, L load, S store) {
  const int n = pl.n;
  with_radix<RMAX>(pl.R[0], [&](auto tag) {
    constexpr int R = decltype(tag)::value;
    const int nb = n / R;
    if (act && j < nb) {
      double2 v[R];
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = load(j + r * nb);
      Dft<R, SG>::run(v);
#pragma unroll
      for (int r = 0; r < R; ++r) A[swz2(base + j * R + r)] = v[r];
    }
  });
  __syncthreads();
  int Ns = pl.R[0];
  if (pl.nst == 3) {
    with_radix<RMAX>(pl.R[1], [&](auto tag) {
      constexpr int R = decltype(tag)::value;
      const int nb = n / R, jq = j / Ns, k = j - jq * Ns;
      double2 v[R];
      if (act && j < nb) {
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = A[swz2(base + j + r * nb)];
        reg_twiddle<R, SG>(v, pl.tw, k * (n / (Ns * R)));
        Dft<R, SG>::run(v);
      }
      __syncthreads();
      if (act && j < nb) {
#pragma unroll
        for (int r = 0; r < R; ++r) A[swz2(base + jq * Ns * R + k + r * Ns)] = v[r];
      }
    });
    __syncthreads();
    Ns *= pl.R[1];
  }
  with_radix<RMAX>(pl.nst == 3 ? pl.R[2] : pl.R[1], [&](auto tag) {
    constexpr int R = decltype(tag)::value;
    const int nb = n / R;  // = Ns
    double2 v[R];
    if (act && j < nb) {
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = A[swz2(base + j + r * nb)];
      reg_twiddle<R, SG>(v, pl.tw, j);
      Dft<R, SG>::run(v);
    }
    if (KEEP) __syncthreads();
    if (act && j < nb) {
#pragma unroll
      for (int r = 0; r < R; ++r) store(j + r * nb, v[r]);
    }
  });
}

}  // namespace chapsim
