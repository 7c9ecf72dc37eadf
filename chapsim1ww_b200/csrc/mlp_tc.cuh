// Learned property model: inference core on the sm_100a tensor cores
// (tcgen05.mma, BF16 operands, FP32 accumulators in tensor memory).
//
// The model maps x = (h - hmid) / hhalf to the five properties (T, rho, mu,
// k, cp) as a least-squares polynomial base of degree 5 per output plus an
// MLP 1 -> 64 -> 64 -> 5 (tanh) that carries the standardised residual:
//   out_o = base_o(x) + mean_o + std_o * (W3 tanh(W2 tanh(W1 x + b1) + b2) + b3)_o
// The reference has no such model (its THERM_PROP_UPDATE interpolates the
// table by cubic splines, src/THERM_PROP_UPDATE.f90:129-205,
// src/Flow_State.f90:1015-1070,1420-1581); the splines stay as the fallback.
//
// A group of 128 threads evaluates tiles of 128 cells (one cell per thread,
// the MMA's M = 128 rows); a CTA holds one group, or four that share the
// weights (the energy substep):
//  - layer 1 on the CUDA cores in FP32 (tanh.approx.f32), the affine parts
//    and every other elementwise step on packed FP32 pairs (.f32x2);
//  - each activation vector is split into BF16 hi + lo parts (lo = the
//    rounding error of hi), the weights likewise, and every layer runs as
//    three BF16 MMAs accumulating in FP32 (hi*hi + hi*lo + lo*hi), which
//    carries about 16 mantissa bits: plain BF16 operands (8 bits) leave the
//    outputs about 1e-3 off, above the 1e-4 bound the model is gated on;
//  - layer 2 (K = 64, N = 64) and layer 3 (K = 64, N = 16, rows 5..15 zero)
//    are issued by one thread as tcgen05.mma kind::f16 from shared-memory
//    operands in the canonical no-swizzle K-major layout, committed to one
//    mbarrier; every thread reads its row back with tcgen05.ld.
// Each group holds 128 tensor-memory columns (layer 2 at columns 0..63, layer 3
// at 64..79, or with the derivative chains of tile_eval_d: z2 0..63 and dz2
// 64..127, then y 0..15 and dy 16..31).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "tma.cuh"

namespace chapsim_mlp {

using chapsim::mbar_init;
using chapsim::mbar_wait;
using chapsim::smem_u32;

constexpr int NH = 64, NO = 5, NOP = 16;  // hidden width, outputs, layer-3 N (padded)
constexpr int TILE = 128;                 // cells per tile = MMA M
constexpr int NBASE = 6;                  // polynomial base: degree 5
constexpr int NP = NH + NH + NH * NH + NH + NO * NH + NO;  // 4613 FP32 parameters
constexpr int O_W1 = 0, O_B1 = NH, O_W2 = 2 * NH, O_B2 = 2 * NH + NH * NH, O_W3 = O_B2 + NH, O_B3 = O_W3 + NO * NH;
constexpr int TMEM_COLS = 128;
constexpr int kMaxGateBins = 4096;
// gate mask bits: output o may come from the model in a bin when bit o is set
constexpr unsigned kStepMask = 0xF;  // T, rho, mu, k: what THERM_PROP_UPDATE produces

// Bytes of one operand tile of `rows` rows x 64 BF16 (K) in the canonical
// no-swizzle K-major layout: 8-row groups of eight 8x16-byte core matrices.
__host__ __device__ constexpr int tile_bytes(int rows) { return rows * NH * 2; }
// Byte offset of element (r, k) in such a tile: core matrices of one 8-row
// group follow each other along K (LBO = 128 B), groups follow at SBO = 1024 B.
__host__ __device__ constexpr int tile_off(int r, int k) {
  return (r >> 3) * 1024 + (k >> 3) * 128 + (r & 7) * 16 + (k & 7) * 2;
}

// Model parameters on the device, passed by value to the kernels.
struct MlpDev {
  const float *par;      // NP FP32 parameters (W1, b1, W2, b2, W3, b3)
  const uint16_t *wt;    // W2 hi, W2 lo (64 rows), W3 hi, W3 lo (16 rows): canonical tiles
  const uint8_t *gate;   // per h-bin output mask
  double hmid, hhalf;
  double mean[NO], stdv[NO], base[NO][NBASE];  // base in powers of x, lowest first
  double g0, ginv;       // gate bins: bin = (h - g0) * ginv
  int nbins;
};

// The FP32 weights of tile_eval_d, a kernel parameter: every thread reads the
// same one at a time, which from the constant bank costs no shared-memory
// bandwidth (a broadcast load still delivers its bytes to all 32 lanes).
struct __align__(16) MlpW {
  float w1[NH], b1[NH], b2[NH];
  float2 w3p[NH / 2][NO];  // W3 by pairs of hidden units: (W3[o][2q], W3[o][2q + 1])
  float b3[NO];
};
inline void set_weights(MlpW &w, const float *par) {
  for (int k = 0; k < NH; ++k) {
    w.w1[k] = par[O_W1 + k];
    w.b1[k] = par[O_B1 + k];
    w.b2[k] = par[O_B2 + k];
  }
  for (int q = 0; q < NH / 2; ++q)
    for (int o = 0; o < NO; ++o) w.w3p[q][o] = {par[O_W3 + o * NH + 2 * q], par[O_W3 + o * NH + 2 * q + 1]};
  for (int o = 0; o < NO; ++o) w.b3[o] = par[O_B3 + o];
}

// Shared memory of a CTA of G groups of 128 threads, each with operand tiles,
// a tensor-memory window and an mbarrier of its own; the weights are shared.
// Four groups with the derivative tile fill an SM (221 KB, all 512
// tensor-memory columns): 16 warps against 12 with three one-group CTAs.
// NOPS operand tiles a group: the activations hi and lo and, for tile_eval_d,
// the BF16 forward-mode derivative of the activations.
template <int G_, int NOPS_>
struct __align__(1024) Smem {
  static constexpr int G = G_, NOPS = NOPS_;
  uint16_t ops[G][NOPS][TILE * NH];  // 16 KB each
  uint16_t w2_hi[NH * NH];           // 8 KB each
  uint16_t w2_lo[NH * NH];
  uint16_t w3_hi[NOP * NH];          // 2 KB each
  uint16_t w3_lo[NOP * NH];
  alignas(16) float w1[NH];          // read as 16-byte vectors
  alignas(16) float b1[NH];
  alignas(16) float b2[NH];
  alignas(16) float b3[NOP];
  uint32_t gstep[kMaxGateBins / 32];  // bit b: bin b cleared for all of kStepMask
  uint64_t bar[G];
  uint32_t tmem;
  int fail[G];
};
using Smem1 = Smem<1, 2>;  // values only, one group, four CTAs per SM
using SmemD = Smem<4, 3>;  // with the derivative, four groups, one CTA per SM (221 KB)

// One group's view of the CTA: its thread's row of the tile, its tensor
// memory and its index.
struct Grp {
  int r, g;
  uint32_t tm;  // first tensor-memory column of the group
};
template <class S>
__device__ __forceinline__ Grp grp_of(const S &s) {
  if constexpr (S::G == 1) return {(int)threadIdx.x, 0, s.tmem};  // a group index known to be 0
  const int g = threadIdx.x / TILE;
  return {(int)threadIdx.x % TILE, g, s.tmem + (uint32_t)(TMEM_COLS * g)};
}
// Barrier over the group's 128 threads (barrier 0 is the CTA's; the warps are
// converged first, the tensor-memory loads after it need whole warps).
template <class S>
__device__ __forceinline__ void grp_sync(const S &, const Grp &q) {
  if constexpr (S::G == 1) {
    __syncthreads();
  } else {
    __syncwarp();
    asm volatile("barrier.sync %0, %1;" ::"r"(q.g + 1), "n"(TILE) : "memory");
    __syncwarp();
  }
}
// The same with the group's "or" of v.
template <class S>
__device__ __forceinline__ bool grp_or(const S &, const Grp &q, bool v) {
  uint32_t any;
  __syncwarp();
  asm volatile(
      "{\n\t.reg .pred p, o;\n\tsetp.ne.u32 p, %3, 0;\n\t"
      "barrier.red.or.pred o, %1, %2, p;\n\tselp.u32 %0, 1, 0, o;\n\t}"
      : "=r"(any)
      : "r"(q.g + 1), "n"(TILE), "r"((uint32_t)v)
      : "memory");
  __syncwarp();
  return any != 0;
}

// ---------------------------------------------------------------- PTX
__device__ __forceinline__ float tanh_approx(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Instruction descriptor of kind::f16: D FP32 (bits 4-5 = 1), A and B BF16
// (bits 7-9, 10-12 = 1), both K-major (bits 15, 16 = 0), N >> 3 at bits
// 17-22, M >> 4 at bits 24-28.
__host__ __device__ constexpr uint32_t idesc_bf16(int m, int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// Shared-memory matrix descriptor: start address, LBO and SBO in 16-byte
// units, descriptor version 1 (bits 46-47), no swizzle (bits 61-63 = 0).
__device__ __forceinline__ uint64_t sdesc(uint32_t saddr) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)(128u >> 4) << 16) | ((uint64_t)(1024u >> 4) << 32) |
         (1ull << 46);
}

// D (+)= A B^T with every output lane enabled (the four 32-bit
// disable-output-lane masks zero); acc = 0 overwrites D.
__device__ __forceinline__ void umma(uint32_t dtm, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  const uint32_t z = 0;
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}" ::"r"(dtm),
      "l"(a), "l"(b), "r"(idesc), "r"(acc), "r"(z), "r"(z), "r"(z), "r"(z)
      : "memory");
}

__device__ __forceinline__ void umma_commit(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 32 consecutive FP32 columns of this thread's TMEM lane, waited for in the
// same statement so no use of the registers can be scheduled before the wait.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float *v) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// Two runs of 32 columns under one wait.
__device__ __forceinline__ void tmem_ld32x2(uint32_t ta, uint32_t tb, float *u, float *v) {
  uint32_t r[64];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%64];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%32,%33,%34,%35,%36,%37,%38,%39,%40,%41,%42,%43,%44,%45,%46,%47,"
      "%48,%49,%50,%51,%52,%53,%54,%55,%56,%57,%58,%59,%60,%61,%62,%63}, [%65];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]),
        "=r"(r[32]), "=r"(r[33]), "=r"(r[34]), "=r"(r[35]), "=r"(r[36]), "=r"(r[37]), "=r"(r[38]), "=r"(r[39]),
        "=r"(r[40]), "=r"(r[41]), "=r"(r[42]), "=r"(r[43]), "=r"(r[44]), "=r"(r[45]), "=r"(r[46]), "=r"(r[47]),
        "=r"(r[48]), "=r"(r[49]), "=r"(r[50]), "=r"(r[51]), "=r"(r[52]), "=r"(r[53]), "=r"(r[54]), "=r"(r[55]),
        "=r"(r[56]), "=r"(r[57]), "=r"(r[58]), "=r"(r[59]), "=r"(r[60]), "=r"(r[61]), "=r"(r[62]), "=r"(r[63])
      : "r"(ta), "r"(tb)
      : "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    u[i] = __uint_as_float(r[i]);
    v[i] = __uint_as_float(r[32 + i]);
  }
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float *v) {
  uint32_t r[8];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
      : "r"(taddr)
      : "memory");
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

// ------------------------------------------------------ packed FP32 pairs
// sm_100 issues two FP32 operations per instruction on a register pair
// (add/sub/mul/fma .f32x2); the elementwise work between the layers runs on
// such pairs, element 2i in the low word.
__device__ __forceinline__ uint64_t pk(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ uint64_t pku(uint32_t a, uint32_t b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ void upk(uint64_t r, float &a, float &b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(r));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t sub2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// Split of a pair of activations into BF16 hi + lo words: hi = x rounded to
// nearest-even BF16 (one cvt.rn.bf16x2.f32; measured 1.5 % faster over the
// whole kernel than rounding by integer add and byte permute), lo = x - hi (exact in
// FP32: at most 16 significant bits) truncated to BF16, so hi + lo carries x
// to about 2^-16 of its magnitude.
__device__ __forceinline__ void split2(uint64_t p, uint32_t &hi, uint32_t &lo) {
  float x0, x1;
  upk(p, x0, x1);
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(hi) : "f"(x1), "f"(x0));  // x0 in the low half
  const uint64_t l = sub2(p, pku(hi << 16, hi & 0xFFFF0000u));
  float l0, l1;
  upk(l, l0, l1);
  lo = __byte_perm(__float_as_uint(l0), __float_as_uint(l1), 0x7632);
}

// Write 32 of a thread's activations into columns c0 .. c0 + 31 of row r of
// the hi and lo operand tiles.
__device__ __forceinline__ void store_split32(uint16_t *a_hi, uint16_t *a_lo, int r, int c0, const float *a) {
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) split2(pk(a[8 * c + 2 * q], a[8 * c + 2 * q + 1]), hi[q], lo[q]);
    const int off = tile_off(r, c0 + 8 * c);
    *reinterpret_cast<uint4 *>(reinterpret_cast<char *>(a_hi) + off) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<uint4 *>(reinterpret_cast<char *>(a_lo) + off) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
  }
}

// The CTA's Smem inside its dynamic shared memory, placed on a 1024-byte
// boundary (the kernels request sizeof(S) + 1024 bytes).
template <class S>
__device__ __forceinline__ S &smem_of(unsigned char *raw) {
  const uint32_t a = smem_u32(raw);
  return *reinterpret_cast<S *>(raw + ((1024u - (a & 1023u)) & 1023u));
}
constexpr size_t kSmemBytes = sizeof(Smem1) + 1024;
constexpr size_t kSmemDBytes = sizeof(SmemD) + 1024;
static_assert(kSmemDBytes <= 227 * 1024, "one CTA per SM");

// ------------------------------------------------------------ CTA set-up
// Load the weights into shared memory, initialise the mbarriers and allocate
// the CTA's tensor memory (warp 0).  Every thread of the CTA calls it.
template <class S>
__device__ __forceinline__ void cta_setup(S &s, const MlpDev &M) {
  const int t = threadIdx.x;
  const uint4 *src = reinterpret_cast<const uint4 *>(M.wt);  // 16-byte aligned (host contract)
  uint4 *dst = reinterpret_cast<uint4 *>(s.w2_hi);  // w2_hi, w2_lo, w3_hi, w3_lo are contiguous
  constexpr int n16 = (2 * NH * NH + 2 * NOP * NH) * 2 / 16;
  for (int q = t; q < n16; q += blockDim.x) dst[q] = src[q];
  if (t < NH) {
    s.w1[t] = M.par[O_W1 + t];
    s.b1[t] = M.par[O_B1 + t];
    s.b2[t] = M.par[O_B2 + t];
  }
  if (t < NOP) s.b3[t] = t < NO ? M.par[O_B3 + t] : 0.f;
  for (int w = t; w < kMaxGateBins / 32; w += blockDim.x) {
    uint32_t bits = 0;
    for (int b = 0; b < 32; ++b)
      if (32 * w + b < M.nbins && (M.gate[32 * w + b] & kStepMask) == kStepMask) bits |= 1u << b;
    s.gstep[w] = bits;
  }
  if (t == 0) {
    for (int g = 0; g < S::G; ++g) {
      mbar_init(&s.bar[g], 1);
      s.fail[g] = 0;
    }
    chapsim::fence_mbar_init();
  }
  if (t < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s.tmem)),
                 "r"(TMEM_COLS * S::G)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  chapsim::fence_proxy_async();  // weight tiles written by plain stores, read by the MMA
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
}

template <class S>
__device__ __forceinline__ void cta_teardown(S &s) {
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (threadIdx.x < 32)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(s.tmem), "r"(TMEM_COLS * S::G)
                 : "memory");
}

// Issue one layer: D[:, 0:n) = A_hi W_hi^T + A_hi W_lo^T + A_lo W_hi^T over
// K = 64 (four K = 16 steps each).
__device__ __forceinline__ void issue_layer(const uint16_t *a_hi, const uint16_t *a_lo, uint32_t dtm,
                                            const uint16_t *w_hi, const uint16_t *w_lo, int n) {
  const uint32_t idesc = idesc_bf16(TILE, n);
  const uint32_t ah = smem_u32(a_hi), al = smem_u32(a_lo), bh = smem_u32(w_hi), bl = smem_u32(w_lo);
  const uint32_t as[3] = {ah, ah, al}, bs[3] = {bh, bl, bh};
#pragma unroll
  for (int part = 0; part < 3; ++part)
#pragma unroll
    for (int ks = 0; ks < 4; ++ks)
      umma(dtm, sdesc(as[part] + 256u * ks), sdesc(bs[part] + 256u * ks), idesc, (part | ks) ? 1u : 0u);
}

// One plain BF16 chain D[:, 0:n) = A W^T (K = 64) from the operand tiles a and w.
__device__ __forceinline__ void issue_chain(uint32_t dtm, const uint16_t *a, const uint16_t *w, int n) {
  const uint32_t idesc = idesc_bf16(TILE, n);
  const uint32_t aa = smem_u32(a), bb = smem_u32(w);
#pragma unroll
  for (int ks = 0; ks < 4; ++ks) umma(dtm, sdesc(aa + 256u * ks), sdesc(bb + 256u * ks), idesc, ks ? 1u : 0u);
}

// Round 32 values to BF16 (nearest-even, cvt.rn.bf16x2.f32) into columns
// c0 .. c0 + 31 of row r of a single operand tile.
__device__ __forceinline__ void store_bf16_32(uint16_t *tile, int r, int c0, const float *v) {
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    uint32_t w[4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
      asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(w[q]) : "f"(v[8 * c + 2 * q + 1]), "f"(v[8 * c + 2 * q]));
    *reinterpret_cast<uint4 *>(reinterpret_cast<char *>(tile) + tile_off(r, c0 + 8 * c)) =
        make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// Group-uniform bounded wait for the layer's commit: false on every thread
// when any thread's wait ran out (the error word is set by mbar_wait).
template <class S>
__device__ __forceinline__ bool layer_wait(S &s, const Grp &q, uint32_t &phase, int *err) {
  const bool ok = mbar_wait(&s.bar[q.g], phase, err);
  phase ^= 1u;
  if (!ok) s.fail[q.g] = 1;
  grp_sync(s, q);
  tc_fence_after();
  return s.fail[q.g] == 0;
}

// 32 units of layer 1 of one cell: a = tanh(w1 x + b1), the affine part on
// FP32 pairs.
__device__ __forceinline__ void layer1_32(const float *w1, const float *b1, float x, float *a) {
  const uint64_t xx = pk(x, x);
  const uint4 *w = reinterpret_cast<const uint4 *>(w1), *b = reinterpret_cast<const uint4 *>(b1);
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const uint4 wq = w[q], bq = b[q];
    upk(fma2(pku(wq.x, wq.y), xx, pku(bq.x, bq.y)), a[4 * q], a[4 * q + 1]);
    upk(fma2(pku(wq.z, wq.w), xx, pku(bq.z, bq.w)), a[4 * q + 2], a[4 * q + 3]);
  }
#pragma unroll
  for (int k = 0; k < 32; ++k) a[k] = tanh_approx(a[k]);
}

// a = tanh(a + bias) over 32 hidden units, the adds on FP32 pairs.
__device__ __forceinline__ void bias_tanh32(const float *bias, float *a) {
  const uint4 *b = reinterpret_cast<const uint4 *>(bias);
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const uint4 bq = b[q];
    upk(add2(pk(a[4 * q], a[4 * q + 1]), pku(bq.x, bq.y)), a[4 * q], a[4 * q + 1]);
    upk(add2(pk(a[4 * q + 2], a[4 * q + 3]), pku(bq.z, bq.w)), a[4 * q + 2], a[4 * q + 3]);
  }
#pragma unroll
  for (int k = 0; k < 32; ++k) a[k] = tanh_approx(a[k]);
}

// t[k] = (1 - a[k]^2) g[k] for 32 consecutive units, on FP32 pairs: the
// forward-mode factor of tanh' applied to the incoming derivative g.
__device__ __forceinline__ void dtanh32(const float *a, const float *g, float *t) {
#pragma unroll
  for (int q = 0; q < 16; ++q) {
    const uint64_t aa = pk(a[2 * q], a[2 * q + 1]), gg = pk(g[2 * q], g[2 * q + 1]);
    upk(sub2(gg, mul2(mul2(aa, aa), gg)), t[2 * q], t[2 * q + 1]);
  }
}

// Evaluate the MLP on the tile: thread r holds cell r's normalised input x
// and receives y[0..4] (standardised residual outputs, b3 included).  Every
// thread of the group calls it together.  Returns false when a wait ran out
// (then y is not valid and the caller stops).
template <class S>
__device__ __forceinline__ bool tile_eval(S &s, const Grp &q, float x, float (&y)[NO], uint32_t &phase, int *err) {
  uint16_t *a_hi = s.ops[q.g][0], *a_lo = s.ops[q.g][1];
  const uint32_t lane_base = q.tm + ((uint32_t)(q.r & ~31) << 16);
  // halves of the hidden units in registers at a time: both with the 128
  // registers of four one-group CTAs per SM, one beside the energy substep's
  // own values (THERM_PROP_UPDATE at 384x192x192: 1055 us, 1083 with one at a
  // time; 1043 with the group index of a one-group CTA known, grp_of)
  constexpr int HP = S::G == 1 ? 2 : 1;
  float a[32 * HP];
#pragma unroll
  for (int h0 = 0; h0 < 2; h0 += HP) {
#pragma unroll
    for (int h = 0; h < HP; ++h) layer1_32(s.w1 + 32 * (h0 + h), s.b1 + 32 * (h0 + h), x, a + 32 * h);
#pragma unroll
    for (int h = 0; h < HP; ++h) store_split32(a_hi, a_lo, q.r, 32 * (h0 + h), a + 32 * h);
  }
  chapsim::fence_proxy_async();
  tc_fence_before();
  grp_sync(s, q);
  if (q.r == 0) {
    tc_fence_after();
    issue_layer(a_hi, a_lo, q.tm, s.w2_hi, s.w2_lo, NH);
    umma_commit(&s.bar[q.g]);
  }
  if (!layer_wait(s, q, phase, err)) return false;
#pragma unroll
  for (int h0 = 0; h0 < 2; h0 += HP) {  // the layer-2 MMAs have completed: the A tiles are free
    if constexpr (HP == 2)
      tmem_ld32x2(lane_base, lane_base + 32, a, a + 32);
    else
      tmem_ld32(lane_base + 32 * h0, a);
#pragma unroll
    for (int h = 0; h < HP; ++h) bias_tanh32(s.b2 + 32 * (h0 + h), a + 32 * h);
#pragma unroll
    for (int h = 0; h < HP; ++h) store_split32(a_hi, a_lo, q.r, 32 * (h0 + h), a + 32 * h);
  }
  chapsim::fence_proxy_async();
  tc_fence_before();
  grp_sync(s, q);
  if (q.r == 0) {
    tc_fence_after();
    issue_layer(a_hi, a_lo, q.tm + NH, s.w3_hi, s.w3_lo, NOP);
    umma_commit(&s.bar[q.g]);
  }
  if (!layer_wait(s, q, phase, err)) return false;
  float o[8];
  tmem_ld8(lane_base + NH, o);
#pragma unroll
  for (int k = 0; k < NO; ++k) y[k] = o[k] + s.b3[k];
  tc_fence_before();  // the next tile's MMAs overwrite these columns after its first group barrier
  return true;
}

// The model at x together with its derivative with respect to x, by forward
// mode through the same layers: da1 = (1 - a1^2) w1, dz2 = W2 da1,
// da2 = (1 - a2^2) dz2, dy = W3 da2.  Layers 1 and 2 are computed exactly as
// in tile_eval, the layer-2 derivative as one plain BF16 chain next to the
// value chains (the derivative only ever multiplies a step of at most
// kTaylorMax, so its ~4e-3 relative precision adds below 1e-5).  Layer 3
// (64 -> 5), value and derivative, runs on the CUDA cores in FP32 on packed
// pairs from the activations in registers: it costs more instructions than
// its MMAs but saves their round trip through shared memory, the tensor
// pipe and tensor memory (one block barrier and one wait per tile), and its
// FP32 products are more accurate than the split BF16 ones.  Tensor memory:
// z2 in columns 0..63, dz2 in 64..127.  Every thread of the group calls it
// together.  The layer-2 wait has no group barrier after it (nothing it
// guards is shared: each thread reads its own tensor-memory lane after
// seeing the commit itself); a wait that ran out sets s.fail, which the
// caller reads after its next group barrier (the results are then
// discarded).
__device__ __forceinline__ void tile_eval_d(SmemD &s, const MlpW &W, const Grp &q, float x, float (&y)[NO],
                                            float (&dy)[NO], uint32_t &phase, int *err) {
  uint16_t *a_hi = s.ops[q.g][0], *a_lo = s.ops[q.g][1], *d_hi = s.ops[q.g][2];
  const uint32_t lane_base = q.tm + ((uint32_t)(q.r & ~31) << 16);
  float a[32], t[32];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    layer1_32(W.w1 + 32 * h, W.b1 + 32 * h, x, a);
    store_split32(a_hi, a_lo, q.r, 32 * h, a);
    dtanh32(a, W.w1 + 32 * h, t);
    store_bf16_32(d_hi, q.r, 32 * h, t);
  }
  chapsim::fence_proxy_async();
  tc_fence_before();
  grp_sync(s, q);
  if (q.r == 0) {
    tc_fence_after();
    issue_layer(a_hi, a_lo, q.tm, s.w2_hi, s.w2_lo, NH);
    issue_chain(q.tm + NH, d_hi, s.w2_hi, NH);
    umma_commit(&s.bar[q.g]);
  }
  if (!mbar_wait(&s.bar[q.g], phase, err)) s.fail[q.g] = 1;
  phase ^= 1u;
  tc_fence_after();
  uint64_t acc[NO], dacc[NO];
#pragma unroll
  for (int o = 0; o < NO; ++o) acc[o] = dacc[o] = 0ull;  // (+0.0f, +0.0f)
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    tmem_ld32x2(lane_base + 32 * h, lane_base + NH + 32 * h, a, t);
    bias_tanh32(W.b2 + 32 * h, a);
    dtanh32(a, t, t);  // da2 for units 32 h .. 32 h + 31
#pragma unroll
    for (int p = 0; p < 16; ++p) {
      const uint64_t ap = pk(a[2 * p], a[2 * p + 1]), gp = pk(t[2 * p], t[2 * p + 1]);
#pragma unroll
      for (int o = 0; o < NO; ++o) {
        const uint64_t w = *reinterpret_cast<const uint64_t *>(&W.w3p[16 * h + p][o]);
        acc[o] = fma2(w, ap, acc[o]);
        dacc[o] = fma2(w, gp, dacc[o]);
      }
    }
  }
#pragma unroll
  for (int o = 0; o < NO; ++o) {
    float e0, e1;
    upk(acc[o], e0, e1);
    y[o] = (e0 + e1) + W.b3[o];
    upk(dacc[o], e0, e1);
    dy[o] = e0 + e1;
  }
  tc_fence_before();  // the next tile's MMAs overwrite the columns read here after its first group barrier
}

// Largest step |x_new - x_old| over which a tile takes the properties at the
// second enthalpy from the first-order expansion of the model's residual
// (the polynomial base is evaluated exactly): the dropped second-order term is
// below std_o |y''| dx^2 / 2, about 1e-5 of each property's range for the
// model's curvature here; a larger step in any cell of the tile evaluates the
// model a second time.
constexpr double kTaylorMax = 1e-3;

// Assemble output o from the standardised residual y at input x (FP64).
__device__ __forceinline__ double assemble(const MlpDev &M, int o, double x, float y) {
  double b = M.base[o][NBASE - 1];
#pragma unroll
  for (int p = NBASE - 2; p >= 0; --p) b = fma(b, x, M.base[o][p]);
  return b + M.mean[o] + M.stdv[o] * (double)y;
}

__device__ __forceinline__ int gate_bin(const MlpDev &M, double h) {
  const int bin = (int)((h - M.g0) * M.ginv);
  return bin < 0 ? 0 : (bin >= M.nbins ? M.nbins - 1 : bin);
}

__device__ __forceinline__ unsigned gate_mask(const MlpDev &M, double h) { return M.gate[gate_bin(M, h)]; }

// Whether the gate cleared h's bin for every output of kStepMask (the CTA's
// shared-memory copy of the gate, one bit per bin).
template <class S>
__device__ __forceinline__ bool gate_step(const S &s, const MlpDev &M, double h) {
  const int bin = gate_bin(M, h);
  return (s.gstep[bin >> 5] >> (bin & 31)) & 1u;
}

}  // namespace chapsim_mlp

// Host-side helpers (props.cu): build the canonical BF16 hi/lo weight tiles
// from the FP32 parameters.
#include <string.h>
namespace chapsim_mlp {
inline uint16_t bf16_rn(float f) {
  uint32_t u;
  memcpy(&u, &f, 4);
  if ((u & 0x7F800000u) == 0x7F800000u) return (uint16_t)(u >> 16);  // inf / nan kept
  u += 0x7FFFu + ((u >> 16) & 1u);
  return (uint16_t)(u >> 16);
}
inline float bf16_f(uint16_t b) {
  const uint32_t u = (uint32_t)b << 16;
  float f;
  memcpy(&f, &u, 4);
  return f;
}
// out: W2 hi (4096), W2 lo (4096), W3 hi (1024), W3 lo (1024) in tile order
inline void build_weight_tiles(const float *par, uint16_t *out) {
  uint16_t *w2h = out, *w2l = out + NH * NH, *w3h = out + 2 * NH * NH, *w3l = w3h + NOP * NH;
  memset(out, 0, sizeof(uint16_t) * (2 * NH * NH + 2 * NOP * NH));
  for (int n = 0; n < NH; ++n)
    for (int k = 0; k < NH; ++k) {
      const float w = par[O_W2 + n * NH + k];
      const uint16_t h = bf16_rn(w);
      const int e = tile_off(n, k) / 2;
      w2h[e] = h;
      w2l[e] = bf16_rn(w - bf16_f(h));
    }
  for (int n = 0; n < NO; ++n)
    for (int k = 0; k < NH; ++k) {
      const float w = par[O_W3 + n * NH + k];
      const uint16_t h = bf16_rn(w);
      const int e = tile_off(n, k) / 2;
      w3h[e] = h;
      w3l[e] = bf16_rn(w - bf16_f(h));
    }
}
}  // namespace chapsim_mlp
