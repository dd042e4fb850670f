// Fused dequant GEMM for FEW activation rows (batched decode steps, short prompts):
// y[m, n] = sum_k x[m, k] * w[n, k], f32 accumulation, one launch per product.
//
// With a few dozen rows a product is bound by how fast the checkpoint bytes stream in and by the latency of
// the chain of launches around it. The tcgen05 GEMM spends ~740 cycles of hand-overs per 128 x 64 chunk
// whatever the row count, reads 36-byte pieces of 128 rows per chunk (0.7 TB/s) and needs an activation pass
// before and a K-split reduction behind it. Here every warp streams 16-row tiles of raw blocks through a
// shared-memory ring of its own (tensor copies, one request per 256 weights of 16 rows), unpacks them into
// mma.sync A fragments in registers and multiplies them with all activation rows (NT groups of 8) held in
// shared memory. A lane quarter t owns whole quantisation blocks of its two rows (the contiguous words
// that the single-row kernels read), because the order of the K elements inside a product is free: the
// activations are laid out so that the matching eight values of a row are one 16-byte load.
//   * Weights become f16(exact dequantised value), as in the tcgen05 GEMM: the integer is made exact
//     (q | 0x6400 = 1024 + q, or 0x5400 = 64 + q for a nibble in place) and one rounding gives q * d (+ m);
//     Q4_K and Q6_K, whose scales are products, go through f32. bf16 / f16 weights enter as they are.
//   * Activations arrive as f16 rows in that order, scaled by a power of two per row (largest magnitude in
//     [2^12, 2^13)), written by the kernel that produces them or by the activation pass below; every CTA brings
//     its K share in with bulk copies. (Converting f32 rows in every CTA doubled the bytes that the L2 has to
//     hand to the SMs, which was what bounded the kernel, and put 1 to 9 us in front of the products.)
//     With bf16 / f16 weights they enter as two or three terms of that type, so nothing of an f32 row is lost.
//   * The first stage is unpacked while the kernel before still runs; only then are the activations awaited.
//   * K is split over the warps of a CTA (KW) and over the CTAs of a cluster (CK); the sums meet in shared
//     memory and through distributed shared memory, in a fixed order: no partial buffer, no second launch.
//   * The SwiGLU form gives a CTA matching tiles of the gate and the up matrix and writes silu(gate) * up.
// All waits are bounded; one that runs out sets the device error word.
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <array>
#include <map>

#include "gemv_core.cuh"
#include "ring.cuh"
#include "tensor_map.cuh"

namespace dyn {

namespace {

constexpr int SK_MAX_SMEM = 226 * 1024;
constexpr long long SK_SPINS = 1LL << 22;
constexpr int SK_UNIT = 256;  // K elements per unit

struct SkArgs {
  int64_t N;            // rows of the weight matrix (SwiGLU: of gate = of up)
  int K, M;
  int kstages;          // stages along K (K / (256 * KU), rounded up)
  int cstages;          // stages per CTA of a cluster
  int RW, KW, CK, nst;  // row warps, K warps, CTAs along K, ring stages per warp
  int swiglu;           // rows [N, 2N) of the matrix are the up projection
  const void* x;        // [TERMS][M, K] in fragment order
  const float* x_inv;   // [M]
  float* y;             // [M, N]
  const float* residual;
  int* error;
  // Q6_K
  const uint8_t* data;
  int64_t rb;
  int q6_mode;
  // MLX
  int aux_f16, sb, group32;
};

__device__ __forceinline__ uint32_t h2u(__half2 v) { return *reinterpret_cast<uint32_t*>(&v); }
__device__ __forceinline__ __half2 u2h(uint32_t v) { return *reinterpret_cast<__half2*>(&v); }

// ---- encodings -----------------------------------------------------------------------------------
// KU: 256-weight units per stage. LW: 32-bit words a lane keeps per row and unit. A lane has eight chunks of
// eight weights per row and unit; chunk c holds two runs of four K elements, run A at k_of(c, t) and run B
// RUNB further on; pairs() gives the f16 pairs (A0 A2) (A1 A3) (B0 B2) (B1 B3) when INTER == 1,
// (A0 A1) (A2 A3) (B0 B1) (B2 B3) when 0 and (A0 B0) (A1 B1) (A2 B2) (A3 B3) when 2.
template <int ENC>
struct Sk;

__device__ __forceinline__ uint32_t sk_h2(uint32_t half_bits) { return half_bits * 0x10001u; }
// (x & mask) | base as ONE instruction on registers (two immediates would make it two)
__device__ __forceinline__ __half2 sk_field(uint32_t x, uint32_t mask, uint32_t base) {
  uint32_t o;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(o) : "r"(x), "r"(mask), "r"(base));
  return *reinterpret_cast<__half2*>(&o);
}

template <>
struct Sk<E_Q4_0> {
  static constexpr int KU = 1, LW = 9, ROWB = 144, STAGE = 16 * ROWB, INTER = 1, RUNB = 16;
  __device__ static int k_of(int c, int t) { return (2 * t + (c >> 2)) * 32 + 4 * (c & 3); }
  __device__ static void load(const uint8_t* row, int t, uint32_t (&w)[LW]) {
    const uint32_t* p = reinterpret_cast<const uint32_t*>(row) + LW * t;
#pragma unroll
    for (int i = 0; i < LW; i++) w[i] = p[i];
  }
  __device__ static void pairs(const uint32_t (&w)[LW], int c, int, uint32_t (&o)[4]) {
    const int i = c & 3;
    const uint32_t x = c >= 4 ? w[5 + i] : __funnelshift_r(w[i], w[i + 1], 16);
    const __half2 d = u2h(c >= 4 ? __byte_perm(w[4], 0, 0x3232) : __byte_perm(w[0], 0, 0x1010));
    const uint32_t y = x >> 8;
    const __half2 c1032 = __floats2half2_rn(1032.f, 1032.f), c72 = __floats2half2_rn(72.f, 72.f);
    o[0] = h2u(__hmul2(__hsub2(sk_field(x, 0x000F000Fu, 0x64006400u), c1032), d));
    o[1] = h2u(__hmul2(__hsub2(sk_field(y, 0x000F000Fu, 0x64006400u), c1032), d));
    o[2] = h2u(__hmul2(__hsub2(sk_field(x, 0x00F000F0u, 0x54005400u), c72), d));
    o[3] = h2u(__hmul2(__hsub2(sk_field(y, 0x00F000F0u, 0x54005400u), c72), d));
  }
};

template <>
struct Sk<E_Q4_1> {
  static constexpr int KU = 1, LW = 10, ROWB = 160, STAGE = 16 * ROWB, INTER = 1, RUNB = 16;
  __device__ static int k_of(int c, int t) { return (2 * t + (c >> 2)) * 32 + 4 * (c & 3); }
  __device__ static void load(const uint8_t* row, int t, uint32_t (&w)[LW]) {
    const uint2* p = reinterpret_cast<const uint2*>(row) + 5 * t;
#pragma unroll
    for (int i = 0; i < 5; i++) {
      const uint2 v = p[i];
      w[2 * i] = v.x, w[2 * i + 1] = v.y;
    }
  }
  __device__ static void pairs(const uint32_t (&w)[LW], int c, int, uint32_t (&o)[4]) {
    const int e = c >> 2;
    const uint32_t x = w[5 * e + 1 + (c & 3)], y = x >> 8;
    const __half2 d = u2h(__byte_perm(w[5 * e], 0, 0x1010)), m = u2h(__byte_perm(w[5 * e], 0, 0x3232));
    const __half2 c1024 = __floats2half2_rn(1024.f, 1024.f), c64 = __floats2half2_rn(64.f, 64.f);
    o[0] = h2u(__hfma2(__hsub2(sk_field(x, 0x000F000Fu, 0x64006400u), c1024), d, m));
    o[1] = h2u(__hfma2(__hsub2(sk_field(y, 0x000F000Fu, 0x64006400u), c1024), d, m));
    o[2] = h2u(__hfma2(__hsub2(sk_field(x, 0x00F000F0u, 0x54005400u), c64), d, m));
    o[3] = h2u(__hfma2(__hsub2(sk_field(y, 0x00F000F0u, 0x54005400u), c64), d, m));
  }
};

template <>
struct Sk<E_Q8_0> {
  static constexpr int KU = 1, LW = 17, ROWB = 272, STAGE = 16 * ROWB, INTER = 0, RUNB = 4;
  __device__ static int k_of(int c, int t) { return (2 * t + (c >> 2)) * 32 + 8 * (c & 3); }
  __device__ static void load(const uint8_t* row, int t, uint32_t (&w)[LW]) {
    const uint32_t* p = reinterpret_cast<const uint32_t*>(row) + LW * t;
#pragma unroll
    for (int i = 0; i < LW; i++) w[i] = p[i];
  }
  __device__ static void pairs(const uint32_t (&w)[LW], int c, int, uint32_t (&o)[4]) {
    const __half2 d = u2h(c >= 4 ? __byte_perm(w[8], 0, 0x3232) : __byte_perm(w[0], 0, 0x1010));
    const __half2 c1152 = __floats2half2_rn(1152.f, 1152.f);
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int i = 2 * (c & 3) + h;
      const uint32_t x = (c >= 4 ? w[9 + i] : __funnelshift_r(w[i], w[i + 1], 16)) ^ 0x80808080u;
      o[2 * h] = h2u(__hmul2(__hsub2(u2h(__byte_perm(x, 0x64646464u, 0x4140)), c1152), d));
      o[2 * h + 1] = h2u(__hmul2(__hsub2(u2h(__byte_perm(x, 0x64646464u, 0x4342)), c1152), d));
    }
  }
};

template <>
struct Sk<E_Q4_K> {
  // words 0, 1: d * scale of sub-blocks 2t and 2t + 1, 2, 3: dmin * min (f32); 4 .. 11: the nibble bytes
  static constexpr int KU = 1, LW = 12, ROWB = 144, STAGE = 16 * ROWB, INTER = 1, RUNB = 32;
  __device__ static int k_of(int c, int t) { return 64 * t + 4 * c; }
  __device__ static void load(const uint8_t* row, int t, uint32_t (&w)[LW]) {
    const uint4 h = *reinterpret_cast<const uint4*>(row);
    const uint4 a = *reinterpret_cast<const uint4*>(row + 16 + 32 * t), b = *reinterpret_cast<const uint4*>(row + 32 + 32 * t);
    const uint32_t sw[3] = {h.y, h.z, h.w};
    auto sb = [&](int i) { return ((i >> 2) == 0 ? sw[0] : (i >> 2) == 1 ? sw[1] : sw[2]) >> (8 * (i & 3)) & 0xffu; };
    const __half2 dd = u2h(h.x);
    const float d = __low2float(dd), dm = __high2float(dd);
#pragma unroll
    for (int e = 0; e < 2; e++) {
      const int j = 2 * t + e;
      uint32_t sc, mn;
      if (j < 4) {
        sc = sb(j) & 63u, mn = sb(j + 4) & 63u;
      } else {
        sc = (sb(j + 4) & 15u) | ((sb(j - 4) >> 6) << 4);
        mn = (sb(j + 4) >> 4) | ((sb(j) >> 6) << 4);
      }
      w[e] = __float_as_uint(d * (float)sc), w[2 + e] = __float_as_uint(dm * (float)mn);
    }
    w[4] = a.x, w[5] = a.y, w[6] = a.z, w[7] = a.w, w[8] = b.x, w[9] = b.y, w[10] = b.z, w[11] = b.w;
  }
  __device__ static void pairs(const uint32_t (&w)[LW], int c, int, uint32_t (&o)[4]) {
    const uint32_t x = w[4 + c];
#pragma unroll
    for (int e = 0; e < 2; e++) {
      const uint32_t v = (x >> (4 * e)) & 0x0F0F0F0Fu;
      const float ds = __uint_as_float(w[e]), dm = __uint_as_float(w[2 + e]);
      float f[4];
#pragma unroll
      for (int i = 0; i < 4; i++)
        f[i] = __fsub_rn(__fmul_rn(ds, __uint_as_float(__byte_perm(v, 0x4B000000u, 0x7440 + i)) - 8388608.f), dm);
      o[2 * e] = h2u(__floats2half2_rn(f[0], f[2]));
      o[2 * e + 1] = h2u(__floats2half2_rn(f[1], f[3]));
    }
  }
};

template <>
struct Sk<E_Q6_K> {
  // quarter t = (p, s): for each half n 16 ql bytes (words 4n ..), for each half 16 qh bytes (words 8 + 4n ..),
  // then the f32 scales of sub-blocks (n, h): words 16 + 2n + h
  static constexpr int KU = 2, LW = 20, ROWB = 432, STAGE = 16 * ROWB, INTER = 0, RUNB = 64;
  __device__ static int k_of(int c, int t) { return (c >> 2) * 128 + 16 * t + 4 * (c & 3); }
  template <int MIS>
  __device__ static void ld16(const uint8_t* q, uint32_t* w) {
    const uint32_t* p = reinterpret_cast<const uint32_t*>(q - MIS);
    if (MIS == 0) {
#pragma unroll
      for (int i = 0; i < 4; i++) w[i] = p[i];
    } else {
      uint32_t r[5];
#pragma unroll
      for (int i = 0; i < 5; i++) r[i] = p[i];
#pragma unroll
      for (int i = 0; i < 4; i++) w[i] = __funnelshift_r(r[i], r[i + 1], 16);
    }
  }
  template <int MIS>
  __device__ static void load(const uint8_t* b, int t, uint32_t (&w)[LW]) {
    const float d = __half2float(*reinterpret_cast<const __half*>(b + 208));
#pragma unroll
    for (int n = 0; n < 2; n++) {
      ld16<MIS>(b + n * 64 + 16 * t, w + 4 * n);
      ld16<MIS>(b + 128 + n * 32 + 16 * (t & 1), w + 8 + 4 * n);
#pragma unroll
      for (int h = 0; h < 2; h++)
        w[16 + 2 * n + h] = __float_as_uint(d * (float)*reinterpret_cast<const int8_t*>(b + 192 + n * 8 + h * 4 + t));
    }
  }
  __device__ static void pairs(const uint32_t (&w)[LW], int c, int t, uint32_t (&o)[4]) {
    const uint32_t ql = w[c], qh = w[8 + c] >> (2 * (t >> 1));
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const uint32_t v = ((ql >> (4 * h)) & 0x0F0F0F0Fu) | (((qh >> (4 * h)) & 0x03030303u) << 4);
      const float s = __uint_as_float(w[16 + 2 * (c >> 2) + h]);
      float f[4];
#pragma unroll
      for (int i = 0; i < 4; i++) f[i] = __fmul_rn(__uint_as_float(__byte_perm(v, 0x4B000000u, 0x7440 + i)) - 8388640.f, s);
      o[2 * h] = h2u(__floats2half2_rn(f[0], f[1]));
      o[2 * h + 1] = h2u(__floats2half2_rn(f[2], f[3]));
    }
  }
};

template <>
struct Sk<E_MLX_U4> {
  // words 0 .. 7: blocks 2t and 2t + 1; 8, 9: their scales as f16 pairs, 10, 11: their biases
  static constexpr int KU = 2, LW = 12, ROWB = 128, STAGE = 2 * 16 * ROWB, INTER = 2, RUNB = 4;
  __device__ static int k_of(int c, int t) { return (2 * t + (c >> 2)) * 32 + 8 * (c & 3); }
  __device__ static void pairs(const uint32_t (&w)[LW], int c, int, uint32_t (&o)[4]) {
    const int e = c >> 2;
    const uint32_t x = w[c], y = x >> 8;
    const __half2 d = u2h(w[8 + e]), m = u2h(w[10 + e]);
    const __half2 c1024 = __floats2half2_rn(1024.f, 1024.f), c64 = __floats2half2_rn(64.f, 64.f);
    o[0] = h2u(__hfma2(__hsub2(sk_field(x, 0x000F000Fu, 0x64006400u), c1024), d, m));
    o[1] = h2u(__hfma2(__hsub2(sk_field(x, 0x00F000F0u, 0x54005400u), c64), d, m));
    o[2] = h2u(__hfma2(__hsub2(sk_field(y, 0x000F000Fu, 0x64006400u), c1024), d, m));
    o[3] = h2u(__hfma2(__hsub2(sk_field(y, 0x00F000F0u, 0x54005400u), c64), d, m));
  }
};

template <>
struct Sk<E_BF16> {
  // 512 bytes per row and unit in four 128-byte swizzled boxes; chunk c of quarter t = elements 32 c + 8 t ..
  static constexpr int KU = 1, LW = 32, ROWB = 512, STAGE = 16 * ROWB, INTER = 0, RUNB = 4;
  __device__ static int k_of(int c, int t) { return 32 * c + 8 * t; }
  __device__ static void pairs(const uint32_t (&w)[LW], int c, int, uint32_t (&o)[4]) {
#pragma unroll
    for (int i = 0; i < 4; i++) o[i] = w[4 * c + i];
  }
};
template <>
struct Sk<E_F16> : Sk<E_BF16> {};

__host__ __device__ constexpr bool sk_plain(int enc) { return enc == E_BF16 || enc == E_F16; }
// terms an activation is split into (bf16: 8 bits each, f16: 11)
__host__ __device__ constexpr int sk_terms(int enc, int nt) { return enc == E_BF16 ? (nt <= 2 ? 3 : 2) : enc == E_F16 ? 2 : 1; }

template <int ENC, int NT, int RT>
__global__ void __launch_bounds__(288, NT <= 2 ? 2 : 1)
gemm_skinny_kernel(const SkArgs a, const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap smap,
                   const __grid_constant__ CUtensorMap bmap) {
  using S = Sk<ENC>;
  constexpr int KU = S::KU, LW = S::LW, TERMS = sk_terms(ENC, NT);
  constexpr bool PLAIN = sk_plain(ENC);
  constexpr int AHEAD = RT == 1 && NT <= 2 && !PLAIN ? 4 : 1;  // chunks unpacked before their products (8 registers each)
  extern __shared__ __align__(1024) uint8_t sk_smem_raw[];
  __shared__ int s_abort;
  __shared__ uint64_t xbar;
  __shared__ float s_inv[NT * 8];
  uint8_t* smem = sk_smem_raw + ((1024u - (smem_u32(sk_smem_raw) & 1023u)) & 1023u);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = a.RW * a.KW;  // one more warp brings the activations
  const int g = lane >> 2, t = lane & 3;
  const int kw = warp % a.KW, rw = warp / a.KW;
  const int aux_stage = ENC == E_MLX_U4 ? 2 * 16 * a.sb : 0;
  const int nst = a.nst;
  // shared memory: [warp][stage][RT] weights | the same of scales and biases (MLX) | barriers | activations;
  // the sums of the epilogue reuse it from the start
  uint8_t* ring = smem + warp * nst * RT * S::STAGE;
  uint8_t* aring = smem + nwarps * nst * RT * S::STAGE + warp * nst * RT * aux_stage;
  uint8_t* after = smem + nwarps * nst * RT * (S::STAGE + aux_stage);
  uint64_t* bars = reinterpret_cast<uint64_t*>(after) + warp * nst;
  uint8_t* xs = after + (nwarps * nst * 8 + 127) / 128 * 128;
  if (tid == 0) {
    s_abort = 0;
    mbar_init(&xbar, 1);
  }
  if (lane == 0) {
    if (warp < nwarps)
      for (int i = 0; i < nst; i++) mbar_init(bars + i, 1);
    mbar_fence_init();
  }
  __syncwarp();

  // this CTA: row group blockIdx.x / CK, K share blockIdx.x % CK (the rank in its cluster)
  const int rank = a.CK > 1 ? (int)(blockIdx.x % (unsigned)a.CK) : 0;
  const int grp = (int)(a.CK > 1 ? blockIdx.x / (unsigned)a.CK : blockIdx.x);
  const int st_lo = rank * a.cstages, st_hi = min(a.kstages, st_lo + a.cstages);
  const int my = warp < nwarps && st_hi - st_lo > kw ? (st_hi - st_lo - kw + a.KW - 1) / a.KW : 0;  // st_lo + kw, + KW, ...
  // first weight row of this warp; SwiGLU: the lower half of the row warps takes gate, the upper half up
  const int N = (int)a.N, last_row = (a.swiglu ? 2 * N : N) - 1;
  const int hw = a.RW >> 1;
  const int row0 = !a.swiglu ? (grp * a.RW + rw) * (16 * RT)
                             : (grp * hw + (rw < hw ? rw : rw - hw)) * (16 * RT) + (rw < hw ? 0 : N);

  int c_left = my, c_stage = st_lo + kw, c_slot = 0;
  auto issue = [&]() {
    if (c_left <= 0) return;
    if (lane == 0 || (ENC == E_Q6_K && a.q6_mode == 0 && lane < 16)) {  // one lane asks for everything
      uint64_t* bar = bars + c_slot;
      if (lane == 0) mbar_expect_tx(bar, RT * (S::STAGE + aux_stage));
      if (ENC == E_Q6_K && a.q6_mode == 0) __syncwarp(0xffffu);
#pragma unroll
      for (int rt = 0; rt < RT; rt++) {
        uint8_t* dst = ring + (c_slot * RT + rt) * S::STAGE;
        const int row = row0 + 16 * rt;
        if constexpr (ENC == E_MLX_U4) {
          uint8_t* adst = aring + (c_slot * RT + rt) * aux_stage;
          tma_box_g2s(dst, &wmap, c_stage * 64, row, bar);
          tma_box_g2s(dst + 2048, &wmap, c_stage * 64 + 32, row, bar);
          tma_box_g2s(adst, &smap, c_stage * (a.sb / 4), row, bar);
          tma_box_g2s(adst + 16 * a.sb, &bmap, c_stage * (a.sb / 4), row, bar);
        } else if constexpr (ENC == E_Q6_K) {
          // a stage is 420 bytes of a row that start anywhere on the 4-byte grid: copy from the 16-byte boundary below
          const int64_t coff = (int64_t)c_stage * 420;
          if (a.q6_mode == 1) {
            tma_box_g2s(dst, &wmap, (int)((coff >> 4) << 2), row, bar);
          } else if (a.q6_mode == 2) {
            tma_box_g2s(dst, &wmap, (int)((coff >> 4) << 2), row >> 1, bar);
            tma_box_g2s(dst + 8 * S::ROWB, &wmap, (int)(((a.rb + coff) >> 4) << 2), row >> 1, bar);
          } else {
            const int r = row + lane > last_row ? last_row : row + lane;
            const uint8_t* src = a.data + (int64_t)r * a.rb + coff;
            src -= reinterpret_cast<uintptr_t>(src) & 15;
            bulk_g2s(dst + lane * S::ROWB, src, S::ROWB, bar);
          }
        } else if constexpr (PLAIN) {
#pragma unroll
          for (int q = 0; q < 4; q++) tma_box_g2s(dst + q * 2048, &wmap, c_stage * 128 + q * 32, row, bar);
        } else {
          tma_box_g2s(dst, &wmap, c_stage * (S::ROWB / 4), row, bar);
        }
      }
    }
    c_left--, c_stage += a.KW;
    if (++c_slot == nst) c_slot = 0;
  };
  for (int q = 0; q < nst; q++) issue();
  __syncthreads();  // xbar is initialised

  // the weights do not depend on the kernels before this one; everything else does
  const int pitch = a.cstages * KU * SK_UNIT * 2 + 64, plane = pitch * NT * 8;
  if (warp == nwarps) {
    // this CTA's K share of the activations, one bulk copy per row and term (columns n >= M of the products are
    // never stored, so those rows stay unwritten)
    pdl_wait_then_trigger();
    const int units = (st_hi - st_lo) * KU;
    if (lane == 0) mbar_expect_tx(&xbar, (unsigned)(TERMS * a.M * units * 512));
    __syncwarp();
    const uint8_t* src = reinterpret_cast<const uint8_t*>(a.x) + (size_t)st_lo * KU * SK_UNIT * 2;
    for (int i = lane; i < TERMS * a.M; i += 32) {
      const int k = i / a.M, n = i - k * a.M;
      bulk_g2s(xs + k * plane + n * pitch, src + (size_t)i * a.K * 2, units * 512, &xbar);
    }
    for (int n = lane; n < a.M; n += 32) s_inv[n] = __ldcg(a.x_inv + n);
  }

  // few row groups: several accumulators per group, so that consecutive mma do not wait for one another
  constexpr int CH = NT * RT == 1 ? 4 : NT * RT == 2 ? 2 : 1;
  float acc[RT][NT][4], accx[CH > 1 ? CH - 1 : 1][RT][NT][4];
#pragma unroll
  for (int rt = 0; rt < RT; rt++)
#pragma unroll
    for (int nt = 0; nt < NT; nt++) {
#pragma unroll
      for (int e = 0; e < 4; e++) {
        acc[rt][nt][e] = 0.f;
#pragma unroll
        for (int h = 0; h + 1 < CH; h++) accx[h][rt][nt][e] = 0.f;
      }
    }
  // Plain weights: an mma truncates where it adds to its accumulator (about 1.5e-8 of the sum each time, always toward
  // zero), so the sums start from zero with every unit and are added up with rounded adds, up to 16 rows with the lower
  // terms in accumulators of their own. Error against 64 bits of a 4096 x 4096 bf16 matrix, 16 f32 rows: 1.7e-6 with one
  // chain, now 1.4e-7 (row kernel in f32: 2.1e-7); 151936 x 1024, 16 rows 135 -> 145 us, 8 rows 82 as before. Quantised weights
  // are rounded to 2^-12, which hides this.
  constexpr bool APART = PLAIN && NT <= 2;
  float tot[PLAIN ? NT : 1][4], low[APART ? 2 : 1][APART ? NT : 1][4];
#pragma unroll
  for (int nt = 0; nt < (PLAIN ? NT : 1); nt++)
#pragma unroll
    for (int e = 0; e < 4; e++) tot[nt][e] = 0.f;
#pragma unroll
  for (int nt = 0; nt < (APART ? NT : 1); nt++)
#pragma unroll
    for (int e = 0; e < 4; e++) low[0][nt][e] = low[APART ? 1 : 0][nt][e] = 0.f;
  auto give_up = [&]() {
    if (!s_abort) {
      s_abort = 1;
      report_wait_expired(a.error, DEV_ERR_GEMV_RING);
    }
  };
  int slot = 0;
  unsigned parity = 0;
  const uint8_t* xu = xs + kw * KU * 512 + t * 16 + g * pitch;  // activations of the current stage
  for (int i = 0; i < my; i++) {
    if (!mbar_try_wait(bars + slot, parity) && !mbar_wait_bounded_sleepy(bars + slot, parity, SK_SPINS, &s_abort, 1000u)) {
      give_up();
      break;  // warp-uniform; the barriers below are still joined
    }
    bool ok = true;
#pragma unroll
    for (int ku = 0; ku < KU; ku++) {
      uint32_t w0[RT][PLAIN ? 1 : LW], w1[RT][PLAIN ? 1 : LW];
      const uint8_t* pb[RT];
      if constexpr (!PLAIN) {
#pragma unroll
        for (int rt = 0; rt < RT; rt++) {
          const uint8_t* base = ring + (slot * RT + rt) * S::STAGE;
          if constexpr (ENC == E_MLX_U4) {
            const uint8_t* ab = aring + (slot * RT + rt) * aux_stage;
#pragma unroll
            for (int h = 0; h < 2; h++) {
              const int piece = ((2 * t + h) ^ g) << 4;
              const uint4 v0 = *reinterpret_cast<const uint4*>(base + ku * 2048 + g * 128 + piece);
              const uint4 v1 = *reinterpret_cast<const uint4*>(base + ku * 2048 + 1024 + g * 128 + piece);
              w0[rt][4 * h] = v0.x, w0[rt][4 * h + 1] = v0.y, w0[rt][4 * h + 2] = v0.z, w0[rt][4 * h + 3] = v0.w;
              w1[rt][4 * h] = v1.x, w1[rt][4 * h + 1] = v1.y, w1[rt][4 * h + 2] = v1.z, w1[rt][4 * h + 3] = v1.w;
              const int si = a.group32 ? ku * 8 + 2 * t + h : ku * 4 + t;
              auto aux = [&](int off, int r) -> uint32_t {
                const uint32_t b = *reinterpret_cast<const uint16_t*>(ab + off + r * a.sb + 2 * si);
                return h2u(a.aux_f16 ? u2h(sk_h2(b)) : __float2half2_rn(__uint_as_float(b << 16)));
              };
              w0[rt][8 + h] = aux(0, g), w0[rt][10 + h] = aux(16 * a.sb, g);
              w1[rt][8 + h] = aux(0, g + 8), w1[rt][10 + h] = aux(16 * a.sb, g + 8);
            }
          } else if constexpr (ENC == E_Q6_K) {
            const int64_t coff = (int64_t)(st_lo + kw + i * a.KW) * 420;
            const int ra = row0 + 16 * rt + g, rb = ra + 8;
            const uint32_t o0 = (uint32_t)(reinterpret_cast<uintptr_t>(a.data) + (int64_t)(ra > last_row ? last_row : ra) * a.rb + coff) & 15u;
            const uint32_t o1 = (uint32_t)(reinterpret_cast<uintptr_t>(a.data) + (int64_t)(rb > last_row ? last_row : rb) * a.rb + coff) & 15u;
            const int s0 = a.q6_mode == 2 ? (g & 1) * 8 + (g >> 1) : g, s1 = a.q6_mode == 2 ? s0 + 4 : g + 8;
            const uint8_t *b0 = base + s0 * S::ROWB + o0, *b1 = base + s1 * S::ROWB + o1;
            if (ku == 0) S::template load<0>(b0, t, w0[rt]), S::template load<0>(b1, t, w1[rt]);
            else S::template load<2>(b0 + 210, t, w0[rt]), S::template load<2>(b1 + 210, t, w1[rt]);
          } else {
            S::load(base + g * S::ROWB, t, w0[rt]);
            S::load(base + (g + 8) * S::ROWB, t, w1[rt]);
          }
        }
        if (ku == KU - 1) {  // everything of the slot is in registers: refill it before the math
          __syncwarp();
          issue();
        }
      } else {
#pragma unroll
        for (int rt = 0; rt < RT; rt++) pb[rt] = ring + (slot * RT + rt) * S::STAGE + g * 128;
      }
      (void)pb;
      uint32_t p0[AHEAD][RT][4], p1[AHEAD][RT][4];
      auto unpack = [&](int c, uint32_t (&q0)[RT][4], uint32_t (&q1)[RT][4]) {
#pragma unroll
        for (int rt = 0; rt < RT; rt++) {
          if constexpr (PLAIN) {
            const uint8_t* q = pb[rt] + (c >> 1) * 2048 + ((((c & 1) * 4 + t) ^ g) << 4);
            const uint4 v0 = *reinterpret_cast<const uint4*>(q), v1 = *reinterpret_cast<const uint4*>(q + 1024);
            q0[rt][0] = v0.x, q0[rt][1] = v0.y, q0[rt][2] = v0.z, q0[rt][3] = v0.w;
            q1[rt][0] = v1.x, q1[rt][1] = v1.y, q1[rt][2] = v1.z, q1[rt][3] = v1.w;
          } else {
            S::pairs(w0[rt], c, t, q0[rt]);
            S::pairs(w1[rt], c, t, q1[rt]);
          }
        }
      };
#pragma unroll
      for (int c = 0; c < 8; c++) {
        if (c % AHEAD == 0) {
#pragma unroll
          for (int q = 0; q < AHEAD; q++) unpack(c + q, p0[q], p1[q]);
        }
        if (c == 0 && i == 0 && ku == 0 && !mbar_wait_bounded_sleepy(&xbar, 0, SK_SPINS, &s_abort, 1000u)) {
          give_up();
          ok = false;
          break;
        }
        const int pc = c % AHEAD;
#pragma unroll
        for (int k = 0; k < TERMS; k++) {
          const uint8_t* xc = xu + ku * 512 + c * 64 + k * plane;
#pragma unroll
          for (int nt = 0; nt < NT; nt++) {
            const uint4 b = *reinterpret_cast<const uint4*>(xc + nt * 8 * pitch);
#pragma unroll
            for (int rt = 0; rt < RT; rt++) {
              constexpr bool BF = ENC == E_BF16;
              const int h0 = CH == 4 ? 2 * (c & 1) : 0, h1 = CH == 4 ? h0 + 1 : CH == 2 ? 1 : 0;
              const bool second = APART && k > 0;
              float(&c0)[4] = second ? low[0][APART ? nt : 0] : h0 == 0 ? acc[rt][nt] : accx[h0 > 0 ? h0 - 1 : 0][rt][nt];
              float(&c1)[4] = second ? low[APART ? 1 : 0][APART ? nt : 0] : h1 == 0 ? acc[rt][nt] : accx[h1 > 0 ? h1 - 1 : 0][rt][nt];
              const uint32_t(&q0)[4] = p0[pc][rt], (&q1)[4] = p1[pc][rt];
              if constexpr (BF) {
                mma_bf16_16816(c0, q0[0], q1[0], q0[1], q1[1], b.x, b.y);
                mma_bf16_16816(c1, q0[2], q1[2], q0[3], q1[3], b.z, b.w);
              } else {
                mma_f16_16816(c0, q0[0], q1[0], q0[1], q1[1], b.x, b.y);
                mma_f16_16816(c1, q0[2], q1[2], q0[3], q1[3], b.z, b.w);
              }
            }
          }
        }
      }
      if constexpr (PLAIN) {
        __syncwarp();
        issue();
#pragma unroll
        for (int nt = 0; nt < NT; nt++)
#pragma unroll
          for (int e = 0; e < 4; e++) {
            float v = acc[0][nt][e];
#pragma unroll
            for (int h = 0; h + 1 < CH; h++) v += accx[h][0][nt][e], accx[h][0][nt][e] = 0.f;
            tot[nt][e] += v, acc[0][nt][e] = 0.f;
          }
      }
    }
    if (!ok) break;
    xu += a.KW * KU * 512;
    if (++slot == nst) slot = 0, parity ^= 1u;
  }
  if constexpr (PLAIN) {
#pragma unroll
    for (int nt = 0; nt < NT; nt++)
#pragma unroll
      for (int e = 0; e < 4; e++) acc[0][nt][e] = APART ? tot[nt][e] + (low[0][APART ? nt : 0][e] + low[APART ? 1 : 0][APART ? nt : 0][e]) : tot[nt][e];
  } else if constexpr (CH > 1) {
#pragma unroll
    for (int h = 0; h + 1 < CH; h++)
#pragma unroll
      for (int rt = 0; rt < RT; rt++)
#pragma unroll
        for (int nt = 0; nt < NT; nt++)
#pragma unroll
          for (int e = 0; e < 4; e++) acc[rt][nt][e] += accx[h][rt][nt][e];
  }
  pdl_wait();  // residual, inverse scales, and y may still be read by the kernels before

  // ---- epilogue: sums of the K warps, then of the cluster's CTAs, in ascending order -------------------
  if (a.KW == 1 && a.CK == 1 && !a.swiglu) {
    // a warp's sums are complete: eight consecutive weight rows of one activation row are a 32-byte sector
    if (warp >= nwarps) return;
#pragma unroll
    for (int nt = 0; nt < NT; nt++) {
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int m = nt * 8 + 2 * t + e;
        if (m >= a.M) continue;
        const float inv = __ldcg(a.x_inv + m);
#pragma unroll
        for (int rt = 0; rt < RT; rt++)
#pragma unroll
          for (int h = 0; h < 2; h++) {
            const int n = row0 + 16 * rt + 8 * h + g;
            if (n >= N) continue;
            const int64_t at = (int64_t)m * N + n;
            a.y[at] = acc[rt][nt][2 * h + e] * inv + (a.residual ? a.residual[at] : 0.f);
          }
      }
    }
    return;
  }
  // the first outputs of every thread and their residuals, while the other warps finish; a thread's outputs step
  // through (m, r) without divisions, Q at a time so that their loads overlap
  constexpr int Q = 4;
  const int rows = a.RW * 16 * RT, rp = NT * 8 + 1;
  const int64_t n_base = (int64_t)grp * (a.swiglu ? rows >> 1 : rows);
  const int step_m = blockDim.x / rows, step_r = blockDim.x - step_m * rows;
  int ms[Q], rs[Q], m = tid / rows, r = tid - m * rows;
  float res[Q];
  auto next_outputs = [&]() {
#pragma unroll
    for (int q = 0; q < Q; q++) {
      ms[q] = m, rs[q] = r;
      m += step_m, r += step_r;
      if (r >= rows) r -= rows, m++;
      res[q] = ms[q] < a.M && a.CK == 1 && a.residual && n_base + rs[q] < a.N ? a.residual[(int64_t)ms[q] * a.N + n_base + rs[q]] : 0.f;
    }
  };
  next_outputs();
  __syncthreads();  // ring and activations are no longer used (every copy issued has been waited for)
  float* red = reinterpret_cast<float*>(smem);                       // [KW][rows][NT * 8 + 1]
  float* part = red + ((size_t)a.KW * rows * rp + 31) / 32 * 32;      // [M][rows]: this CTA's share (CK > 1, SwiGLU)
  if (warp < nwarps)
#pragma unroll
  for (int rt = 0; rt < RT; rt++) {
    float* r0 = red + ((size_t)kw * rows + rw * 16 * RT + rt * 16 + g) * rp + 2 * t;
#pragma unroll
    for (int nt = 0; nt < NT; nt++) {
      r0[nt * 8] = acc[rt][nt][0], r0[nt * 8 + 1] = acc[rt][nt][1];
      r0[8 * rp + nt * 8] = acc[rt][nt][2], r0[8 * rp + nt * 8 + 1] = acc[rt][nt][3];
    }
  }
  __syncthreads();
  const int out_rows = a.swiglu ? rows >> 1 : rows;
  const int kstep = rows * rp, total = a.M * rows;
  auto finish = [&](int m, int r, float v, float up) {
    const int64_t n = n_base + r;
    if (n >= a.N) return;
    const int64_t at = (int64_t)m * a.N + n;
    if (a.swiglu) v = (v / (1.0f + expf(-v))) * up;
    else if (a.residual) v += a.residual[at];
    a.y[at] = v;
  };
  for (int i0 = tid; i0 < total; i0 += Q * blockDim.x) {
    if (i0 != tid) next_outputs();
    float v[Q];
#pragma unroll
    for (int q = 0; q < Q; q++) {
      const float* p = red + (ms[q] < a.M ? rs[q] * rp + ms[q] : 0);
      v[q] = p[0];
      for (int k = 1; k < a.KW; k++) v[q] += p[k * kstep];
    }
#pragma unroll
    for (int q = 0; q < Q; q++) {
      if (ms[q] >= a.M) continue;
      const float f = v[q] * s_inv[ms[q]];
      if (a.CK > 1 || a.swiglu)
        part[ms[q] * rows + rs[q]] = f;
      else if (n_base + rs[q] < a.N)
        a.y[(int64_t)ms[q] * a.N + n_base + rs[q]] = f + res[q];
    }
  }
  if (a.CK == 1) {
    if (!a.swiglu) return;
    __syncthreads();
    for (int i = tid; i < a.M * out_rows; i += blockDim.x) {
      const int m = i / out_rows, r = i - m * out_rows;
      finish(m, r, part[m * rows + r], part[m * rows + out_rows + r]);
    }
    return;
  }
  asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
  {
    const uint32_t base = smem_u32(part);
    uint32_t peer[8];
#pragma unroll
    for (int c = 0; c < 8; c++)
      asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer[c]) : "r"(base), "r"(c < a.CK ? c : 0));
    // four consecutive weight rows per thread: one 16-byte read per CTA of the cluster
    auto cluster_sum = [&](int i, float (&v)[4]) {
      float4 f[8];
#pragma unroll
      for (int c = 0; c < 8; c++)
        if (c < a.CK)
          asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                       : "=f"(f[c].x), "=f"(f[c].y), "=f"(f[c].z), "=f"(f[c].w)
                       : "r"(peer[c] + 4u * (uint32_t)i)
                       : "memory");
      v[0] = v[1] = v[2] = v[3] = 0.f;
#pragma unroll
      for (int c = 0; c < 8; c++)
        if (c < a.CK) v[0] += f[c].x, v[1] += f[c].y, v[2] += f[c].z, v[3] += f[c].w;
    };
    const int quads = out_rows >> 2;
    for (int i = tid + rank * blockDim.x; i < a.M * quads; i += blockDim.x * a.CK) {
      const int m = i / quads, r = (i - m * quads) * 4;
      float v[4], up[4] = {0.f, 0.f, 0.f, 0.f};
      cluster_sum(m * rows + r, v);
      if (a.swiglu) cluster_sum(m * rows + out_rows + r, up);
#pragma unroll
      for (int e = 0; e < 4; e++) finish(m, r + e, v[e], up[e]);
    }
  }
  // nobody leaves while its sums may still be read
  asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}

// ---- activation pass for many rows: rows -> f16 fragment order + inverse scales ------------------------
// One block per row; a thread takes runs of eight elements.
__global__ void __launch_bounds__(256)
sk_prepare_kernel(const void* x, int x_bf16, int K, int enc, int terms, int64_t plane, __half* out, float* inv_s) {
  __shared__ float red[8];
  const int64_t m = blockIdx.x;
  const int tid = threadIdx.x;
  constexpr int R = 4;  // runs in registers at a time: rows of up to 8192 elements are loaded once
  float v[R][8];
  pdl_wait_then_trigger();
  auto load = [&](int i0) {
#pragma unroll
    for (int i = 0; i < R; i++) {
      const int k = (tid + (i0 + i) * 256) * 8;
      if (k >= K) {
#pragma unroll
        for (int e = 0; e < 8; e++) v[i][e] = 0.f;
      } else if (x_bf16) {
        const uint4 q = __ldcg(reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(x) + m * K + k));
        const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int e = 0; e < 4; e++) v[i][2 * e] = __uint_as_float(w[e] << 16), v[i][2 * e + 1] = __uint_as_float(w[e] & 0xffff0000u);
      } else {
        const float4* p = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(x) + m * K + k);
        const float4 a = __ldcg(p), b = __ldcg(p + 1);
        v[i][0] = a.x, v[i][1] = a.y, v[i][2] = a.z, v[i][3] = a.w, v[i][4] = b.x, v[i][5] = b.y, v[i][6] = b.z, v[i][7] = b.w;
      }
    }
  };
  const int runs = (K / 8 + 255) / 256;
  float mx = 0.f;
  for (int i0 = 0; i0 < runs; i0 += R) {
    load(i0);
#pragma unroll
    for (int i = 0; i < R; i++)
#pragma unroll
      for (int e = 0; e < 8; e++) mx = fmaxf(mx, fabsf(v[i][e]));
  }
  mx = warp_max(mx);
  if ((tid & 31) == 0) red[tid >> 5] = mx;
  __syncthreads();
  mx = red[0];
#pragma unroll
  for (int i = 1; i < 8; i++) mx = fmaxf(mx, red[i]);
  float sc, inv;
  scale_for(mx, &sc, &inv);
  if (tid == 0) inv_s[m] = inv;
  for (int i0 = 0; i0 < runs; i0 += R) {
    if (runs > R) load(i0);
#pragma unroll
    for (int i = 0; i < R; i++) {
      const int k = (tid + (i0 + i) * 256) * 8;
      if (k >= K) continue;
      if (terms == 1) {
        sk_store_frag8(out + m * K, enc, k, v[i], sc);
        continue;
      }
      // plain weights: natural order, the value as a sum of `terms` values of the weights' type
#pragma unroll
      for (int e = 0; e < 8; e++) v[i][e] *= sc;
      for (int q = 0; q < terms; q++) {
        uint32_t o[4];
#pragma unroll
        for (int e = 0; e < 4; e++) {
          if (enc == E_BF16) {
            const __nv_bfloat162 h = __floats2bfloat162_rn(v[i][2 * e], v[i][2 * e + 1]);
            o[e] = *reinterpret_cast<const uint32_t*>(&h);
            v[i][2 * e] -= __low2float(h), v[i][2 * e + 1] -= __high2float(h);
          } else {
            const __half2 h = __floats2half2_rn(v[i][2 * e], v[i][2 * e + 1]);
            o[e] = h2u(h);
            v[i][2 * e] -= __low2float(h), v[i][2 * e + 1] -= __high2float(h);
          }
        }
        *reinterpret_cast<uint4*>(out + q * plane + m * K + k) = make_uint4(o[0], o[1], o[2], o[3]);
      }
    }
  }
}

// ---- plan ------------------------------------------------------------------------------------------
struct SkPlan {
  int NT, RT, RW, KW, CK, nst, kstages, cstages;
  int64_t groups;
  size_t smem;
};

int sk_ku(int enc) { return enc == E_MLX_U4 || enc == E_Q6_K ? 2 : 1; }
int sk_stage_bytes(const WRef& w) {
  switch (w.enc) {
    case E_Q4_1: return Sk<E_Q4_1>::STAGE;
    case E_Q8_0: return Sk<E_Q8_0>::STAGE;
    case E_Q6_K: return Sk<E_Q6_K>::STAGE;
    case E_MLX_U4: return Sk<E_MLX_U4>::STAGE + 2 * 16 * (w.group == 32 ? 32 : 16);
    case E_BF16:
    case E_F16: return Sk<E_BF16>::STAGE;
    default: return Sk<E_Q4_0>::STAGE;
  }
}

size_t sk_smem(const WRef& w, const SkPlan& p, int M) {
  const int warps = p.RW * p.KW, rows = p.RW * 16 * p.RT;
  const size_t ring = (size_t)warps * p.nst * p.RT * sk_stage_bytes(w) + ((size_t)warps * p.nst * 8 + 127) / 128 * 128;
  const size_t x = (size_t)sk_terms(w.enc, p.NT) * p.NT * 8 * ((size_t)p.cstages * sk_ku(w.enc) * SK_UNIT * 2 + 64);
  const size_t red = ((size_t)p.KW * rows * (p.NT * 8 + 1) + 31) / 32 * 32 * 4 + (size_t)M * rows * 4;
  return 1024 + std::max(ring + x, red);
}

bool sk_make_plan(const WRef& w, int64_t M, bool swiglu, SkPlan* best) {
  const int sms = std::max(1, sm_count());
  const int64_t N = swiglu ? w.rows / 2 : w.rows;
  const int ku = sk_ku(w.enc);
  SkPlan p;
  p.NT = M <= 8 ? 1 : M <= 16 ? 2 : M <= 32 ? 4 : 8;
  p.kstages = (int)((w.cols + ku * SK_UNIT - 1) / (ku * SK_UNIT));
  double best_cost = 1e30;
  for (p.RT = 1; p.RT <= (p.NT >= 4 && !sk_plain(w.enc) ? 2 : 1); p.RT++)
    for (p.CK = 1; p.CK <= 8; p.CK *= 2) {
      if (p.CK > p.kstages) break;
      p.cstages = (p.kstages + p.CK - 1) / p.CK;
      if ((int64_t)p.cstages * (p.CK - 1) >= p.kstages) continue;  // every CTA of a cluster has work
      for (p.KW = 1; p.KW <= 8; p.KW++) {
        if (p.KW > p.cstages) break;
        for (p.RW = swiglu ? 2 : 1; p.RW * p.KW <= 8; p.RW *= 2) {
          const int wst = (p.cstages + p.KW - 1) / p.KW;
          p.nst = std::min(wst, 2);
          p.smem = sk_smem(w, p, (int)M);
          if (p.smem > (size_t)SK_MAX_SMEM) continue;
          p.groups = (N + (swiglu ? 8 : 16) * p.RT * p.RW - 1) / ((swiglu ? 8 : 16) * p.RT * p.RW);
          const int64_t ctas = p.groups * p.CK;
          if (ctas > 0x7fffffff) continue;
          const int threads = (p.RW * p.KW + 1) * 32;
          const int occ = (int)std::max<int64_t>(1, std::min<int64_t>((int64_t)((227 * 1024) / (p.smem + 1024)), 1024 / std::max(threads, 32)));
          // Microseconds, fitted to measured plans of eleven shapes at 8 to 64 rows (within 20 %): per round of CTAs
          // the part of prologue and drain that its SM-mates do not cover (clusters of eight start late), the activations (about 45 bytes per
          // nanosecond reach an SM that shares them with all others), and the units of 16 x 256 weights, bound by
          // issue (few warps per SM hide less latency) or by one warp's own chain.
          const double rounds = (double)ctas / ((double)sms * occ);
          const double live = std::min<double>(occ, std::max(1.0, (double)ctas / sms));  // CTAs that share an SM
          const double heavy = sk_plain(w.enc) ? 0.5 * sk_terms(w.enc, p.NT) : w.enc == E_Q6_K || w.enc == E_Q4_K ? 1.6 : 1.0;
          const double unit = heavy * (p.RT == 2 ? 2.4 : 1.0) * (1.0 + 0.14 * (p.NT - 1)), warps_sm = live * p.RW * p.KW;
          const double units = (double)wst * ku;
          const double fixed = 0.3 + 2.4 / live + (p.CK > 1 ? 1.0 + p.CK : p.KW > 1 ? 0.8 : 0.0);
          const double x_us = (double)M * p.cstages * ku * SK_UNIT * 2.0 * sk_terms(w.enc, p.NT) * live / 45e3;
          const double w_us = std::max(units * 0.4 * unit, units * warps_sm * std::max(0.058 * unit * (1.0 + 4.0 / warps_sm),
                                                                                       p.RT * sk_stage_bytes(w) / (double)ku / 40e3));
          const double cost = (rounds <= 1.0 ? 1.0 : rounds + 0.35) * (fixed + x_us + w_us) +
                              (p.CK > 1 ? 1.5 + 0.5 * M * 16 * p.RT * p.RW / (double)(4 * p.CK * threads) : p.KW > 1 || swiglu ? 0.7 : 0.4);
          if (cost < best_cost) best_cost = cost, *best = p;
        }
      }
    }
  if (best_cost > 1e29) return false;
  return true;
}

// Plans are looked up, not searched, after the first product of a shape (a search costs the host several
// microseconds). Per thread; dropped when a program with very many shapes fills it.
bool sk_plan(const WRef& w, int64_t M, bool swiglu, SkPlan* p) {
  typedef std::array<int64_t, 4> Key;
  static thread_local std::map<Key, std::pair<bool, SkPlan>> plans;
  const Key key = {w.rows, w.cols, M, (int64_t)w.enc * 4 + (w.group == 32 ? 2 : 0) + (swiglu ? 1 : 0)};
  auto it = plans.find(key);
  if (it == plans.end()) {
    if (plans.size() >= 1024) plans.clear();
    SkPlan q;
    const bool ok = sk_make_plan(w, M, swiglu, &q);
    it = plans.emplace(key, std::make_pair(ok, q)).first;
  }
  *p = it->second.second;
  return it->second.first;
}

template <int ENC, int NT, int RT>
int sk_run(const SkArgs& a, const SkPlan& p, const CUtensorMap& wm, const CUtensorMap& sm, const CUtensorMap& bm, cudaStream_t s) {
  auto kernel = gemm_skinny_kernel<ENC, NT, RT>;
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), SK_MAX_SMEM)) return 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(p.groups * p.CK)), cfg.blockDim = dim3((p.RW * p.KW + 1) * 32);
  cfg.dynamicSmemBytes = p.smem, cfg.stream = s;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (pdl_enabled()) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (p.CK > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = (unsigned)p.CK, attr[n].val.clusterDim.y = 1, attr[n].val.clusterDim.z = 1;
    n++;
  }
  cfg.attrs = attr, cfg.numAttrs = n;
  DYN_CUDA(cudaLaunchKernelEx(&cfg, kernel, a, wm, sm, bm));
  count_launch();
  return 0;
}

template <int ENC>
int sk_run_enc(const SkArgs& a, const SkPlan& p, const CUtensorMap& wm, const CUtensorMap& sm, const CUtensorMap& bm, cudaStream_t s) {
  if (p.NT == 1) return sk_run<ENC, 1, 1>(a, p, wm, sm, bm, s);
  if (p.NT == 2) return sk_run<ENC, 2, 1>(a, p, wm, sm, bm, s);
  if constexpr (!sk_plain(ENC)) {
    if (p.RT == 2) return p.NT == 4 ? sk_run<ENC, 4, 2>(a, p, wm, sm, bm, s) : sk_run<ENC, 8, 2>(a, p, wm, sm, bm, s);
  }
  return p.NT == 4 ? sk_run<ENC, 4, 1>(a, p, wm, sm, bm, s) : sk_run<ENC, 8, 1>(a, p, wm, sm, bm, s);
}

}  // namespace

// Encodings, alignments and row counts the kernel reads. A 4-row product of f32 activations keeps its hi / lo
// kernels (they carry 22 bits of an activation); K a multiple of 256 (of 512 for MLX-U4 and Q6_K).
bool gemm_skinny_takes(const WRef& w, int64_t M) {
  if (M < 1 || M > 64 || w.rows < 1 || w.rows > (1LL << 30)) return false;
  {  // the activations of an eighth of K have to fit beside one warp's ring
    const int ku = sk_ku(w.enc), nt = M <= 8 ? 1 : M <= 16 ? 2 : M <= 32 ? 4 : 8;
    const int64_t stages = (w.cols + ku * SK_UNIT - 1) / (ku * SK_UNIT);
    if (sk_terms(w.enc, nt) * nt * 8 * ((stages + 7) / 8 * ku * SK_UNIT * 2 + 64) > 160 * 1024) return false;
  }
  const bool aligned = (reinterpret_cast<uintptr_t>(w.data) & 15) == 0;
  switch (w.enc) {
    case E_Q4_0:
    case E_Q4_1:
    case E_Q8_0:
    case E_Q4_K:
    case E_BF16:
    case E_F16: return aligned && w.cols >= 256 && w.cols % 256 == 0;
    case E_Q6_K: return aligned && w.cols >= 512 && w.cols % 512 == 0;
    case E_MLX_U4:
      return aligned && w.cols >= 512 && w.cols % 512 == 0 && (w.group == 64 || w.group == 32) &&
             (w.aux == E_BF16 || w.aux == E_F16) && w.scales && w.biases &&
             ((reinterpret_cast<uintptr_t>(w.scales) | reinterpret_cast<uintptr_t>(w.biases)) & 15) == 0;
    default: return false;
  }
}

// Where the kernel is ahead of the tcgen05 GEMMs. More rows of a large matrix are bound by the mma.sync rate and by the
// activations every CTA reads, from 17 rows where raw weights arrive in boxes, from 33 with the others.
// A product by itself: over 100 shapes of 512 x 512 to 57344 x 8192 at 17 to 64 rows a line at 8 M weights costs 4.0 %
// against the faster kernel of each shape, at 4 M 3.9, at 12 M 5.0, at 16 M 6.8 %; Q6_K at 33 to 64 rows 2.6, 2.7, 2.7 and
// 4.7 % (4096 x 4096, 48 rows, here / there: Q4_0 19 / 14 us, Q6_K 46 / 26 us). Plain weights keep more of an f32 row here
// than the GEMM's one f16 term, so they stay as long as they can.
// In a chain of layers, where norm, residual and SwiGLU ride on the products, the line is higher: eight layers of
// 2048 x 3072 ([gate; up] 12 M) take 0.50 against 0.65 ms at 24 rows, Q6_K 0.80 against 0.86 at 40 (Q4_0 0.78 against 0.72
// there); eight layers of the 8B shape (100 M) 1.99 against 1.51 ms.
bool gemm_skinny_prefers(const WRef& w, int64_t M, bool chain) {
  if (!gemm_skinny_takes(w, M)) return false;
  const int64_t line = (chain || sk_plain(w.enc) ? 16LL : 8LL) << 20;
  return M <= (gemm_stream_takes(w) ? 16 : 32) || w.rows * w.cols <= line;
}

// y[M, N] = x w^T + residual, or with `swiglu` (the matrix is [gate; up], N = rows / 2) silu(x gate^T) * (x up^T).
// x: rows in fragment order (gemm_skinny_terms of them per activation row, [terms][M, K]), x_inv their inverse
// scales. *handled = false when the product does not qualify.
int launch_gemm_skinny(const WRef& w, const __half* x, const float* x_inv, int64_t M, float* y,
                       const float* residual, bool swiglu, cudaStream_t s, bool* handled) {
  *handled = false;
  if (!gemm_skinny_takes(w, M) || (swiglu && w.rows % 32)) return 0;
  SkPlan p;
  if (!sk_plan(w, M, swiglu, &p)) return 0;
  if (swiglu && (w.rows / 2) % (16 * p.RT)) return 0;
  SkArgs a{};
  a.N = swiglu ? w.rows / 2 : w.rows, a.K = (int)w.cols, a.M = (int)M;
  a.kstages = p.kstages, a.cstages = p.cstages;
  a.RW = p.RW, a.KW = p.KW, a.CK = p.CK, a.nst = p.nst;
  a.swiglu = swiglu ? 1 : 0;
  a.x = x, a.x_inv = x_inv, a.y = y, a.residual = residual;
  a.error = device_error_word();
  if (!a.error) return 1;
  a.data = w.data, a.rb = w.enc == E_MLX_U4 ? w.cols / 2 : w.row_bytes();
  CUtensorMap wm, sm, bm;
  memset(&wm, 0, sizeof wm);
  switch (w.enc) {
    case E_MLX_U4: {
      a.aux_f16 = w.aux == E_F16 ? 1 : 0, a.sb = w.group == 32 ? 32 : 16, a.group32 = w.group == 32 ? 1 : 0;
      const size_t aux_row = (size_t)(w.cols / w.group) * 2;
      if (make_row_box_map(w.data, (size_t)w.cols / 2, w.rows, 32, 16, &wm, true) ||
          make_row_box_map(w.scales, aux_row, w.rows, a.sb / 4, 16, &sm) ||
          make_row_box_map(w.biases, aux_row, w.rows, a.sb / 4, 16, &bm))
        return 1;
      break;
    }
    case E_Q6_K:
      if (a.rb % 16 == 0) {
        if (make_row_box_map(w.data, (size_t)a.rb, w.rows, Sk<E_Q6_K>::ROWB / 4, 16, &wm)) return 1;
        a.q6_mode = 1;
      } else if (a.rb % 8 == 0 && w.rows % 2 == 0) {
        if (make_row_box_map(w.data, (size_t)a.rb * 2, w.rows / 2, Sk<E_Q6_K>::ROWB / 4, 8, &wm)) return 1;
        a.q6_mode = 2;
      }
      break;
    case E_BF16:
    case E_F16:
      if (make_row_box_map(w.data, (size_t)w.row_bytes(), w.rows, 32, 16, &wm, true)) return 1;
      break;
    default: {
      const int words = w.enc == E_Q4_1 ? 40 : w.enc == E_Q8_0 ? 68 : 36;
      if (make_row_box_map(w.data, (size_t)w.row_bytes(), w.rows, words, 16, &wm)) return 1;
    }
  }
  if (w.enc != E_MLX_U4) sm = wm, bm = wm;
  int rc = 1;
  switch (w.enc) {
    case E_Q4_0: rc = sk_run_enc<E_Q4_0>(a, p, wm, sm, bm, s); break;
    case E_Q4_1: rc = sk_run_enc<E_Q4_1>(a, p, wm, sm, bm, s); break;
    case E_Q8_0: rc = sk_run_enc<E_Q8_0>(a, p, wm, sm, bm, s); break;
    case E_Q6_K: rc = sk_run_enc<E_Q6_K>(a, p, wm, sm, bm, s); break;
    case E_Q4_K: rc = sk_run_enc<E_Q4_K>(a, p, wm, sm, bm, s); break;
    case E_MLX_U4: rc = sk_run_enc<E_MLX_U4>(a, p, wm, sm, bm, s); break;
    case E_BF16: rc = sk_run_enc<E_BF16>(a, p, wm, sm, bm, s); break;
    case E_F16: rc = sk_run_enc<E_F16>(a, p, wm, sm, bm, s); break;
    default: break;
  }
  if (rc) return 1;
  DYN_CUDA(cudaGetLastError());
  *handled = true;
  return 0;
}

int gemm_skinny_terms(const WRef& w, int64_t M) { return sk_terms(w.enc, M <= 8 ? 1 : M <= 16 ? 2 : M <= 32 ? 4 : 8); }

int launch_skinny_prepare(const WRef& w, const void* x, int x_type, int64_t M, __half* out, float* inv_s, cudaStream_t s, bool natural) {
  DYN_CUDA(launch_pdl(sk_prepare_kernel, dim3((unsigned)M), dim3(256), 0, s, x, x_type == E_BF16 ? 1 : 0, (int)w.cols,
                      natural ? SK_NATURAL : w.enc, natural ? 1 : gemm_skinny_terms(w, M), M * w.cols, out, inv_s));
  count_launch();
  return 0;
}

// A product of plain rows (f32 or bf16): activation pass, then the GEMM.
int launch_linear_skinny(const WRef& w, const void* x, int x_type, int64_t M, float* y, const float* residual, cudaStream_t s,
                         bool* handled) {
  *handled = false;
  const bool cluster = gemm_cluster_prefers(w, M, false);
  const size_t x_rows = cluster ? (size_t)gemm_cluster_rows(M) : (size_t)gemm_skinny_terms(w, M) * M;
  const size_t xb = (x_rows * w.cols * 2 + 255) / 256 * 256, bytes = xb + (size_t)M * 4;
  uint8_t* ws = reinterpret_cast<uint8_t*>(thread_scratch(bytes));
  const bool pooled = ws == nullptr;
  if (pooled) {
    if (keep_scratch_pool_cached()) return 1;
    DYN_CUDA(cudaMallocAsync(reinterpret_cast<void**>(&ws), bytes, s));
  }
  float* inv = reinterpret_cast<float*>(ws + xb);
  int rc = launch_skinny_prepare(w, x, x_type, M, reinterpret_cast<__half*>(ws), inv, s, cluster);
  if (!rc && cluster) {
    rc = launch_gemm_cluster(w, reinterpret_cast<const __half*>(ws), inv, M, y, residual, false, s);
    *handled = true;
  } else if (!rc) rc = launch_gemm_skinny(w, reinterpret_cast<const __half*>(ws), inv, M, y, residual, false, s, handled);
  const cudaError_t fe = pooled ? cudaFreeAsync(ws, s) : cudaSuccess;
  if (rc) return 1;
  if (fe != cudaSuccess) return cuda_fail(fe, "cudaFreeAsync", __FILE__, __LINE__);
  return 0;
}

}  // namespace dyn
