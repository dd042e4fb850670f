// Fused dequant product for 1 to 8 activation rows that keeps every bit of the weights and 22 bits of the
// activations (single-row decode steps, batches of up to four): y[m, n] = sum_k x[m, k] * w[n, k].
//
// mma.sync.m16n8k16 has 8 output columns, and the product of one row needs two (its values enter as an f16 pair
// hi + lo). The other columns keep FOUR quantisation blocks apart: lane quarter t feeds the A operand with the
// raw integers of its own blocks (an integer in the low mantissa bits of an f16 is the subnormal q * 2^-24:
// exact, one logic instruction per two weights), and the B operand holds the activations of quarter t's blocks
// only in columns 2t (hi) and 2t + 1 (lo), zeros elsewhere. A lane's accumulators are then (its two rows) x (its own
// block), and block scale, zero point and minimum are applied to them in f32, with the blocks' activation sums
// (sum x (q d + m) = d sum x q + m sum x). More rows repeat the mma with other B registers; the unpacking is shared.
//
// Where the forms before this one split K over CTAs, left the sums in global memory and added them in a second
// launch, here a CTA's warps split K among themselves (KW) and meet in shared memory; only rows too wide for an
// SM's shared memory are split over a cluster. RMSNorm of the input can be part of the staging (the sum of
// squares is taken over the whole row by every CTA, the product is linear in 1 / rms, which is applied at the
// end), the residual or the SwiGLU part of the epilogue. Each warp streams its 16-row tiles through a ring of its
// own, one tensor copy per stage, and asks for the first stages before the kernel in front has finished.
// All waits are bounded; one that runs out sets the device error word.
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <cmath>
#include <array>
#include <map>

#include "gemv_core.cuh"
#include "ring.cuh"
#include "tensor_map.cuh"

namespace dyn {

namespace {

constexpr int GR_MAX_SMEM = 226 * 1024;
constexpr long long GR_SPINS = 1LL << 22;
constexpr int GR_UNIT = 256;  // K elements per unit

struct GrArgs {
  int64_t N;            // rows of the weight matrix (SwiGLU: of gate = of up)
  int K, M;
  int kstages, cstages; // stages along K; per CTA of a cluster
  int RW, KW, CK, nst;
  int swiglu;           // rows [N, 2N) of the matrix are the up projection
  int x_bf16;
  const void* x;        // [M, K]
  const void* norm_w;   // RMSNorm weights of the input rows, or NULL
  int norm_type;
  float eps;
  float* y;             // [M, N]
  const float* residual;
  int* error;
  const uint8_t* data;  // Q6_K
  int64_t rb;
  int q6_mode;
  int aux_f16, sb, group32;  // MLX
};

// Per encoding. KU: units per stage; LW: words a lane keeps per row and unit; NG: scale groups of a lane per unit.
// A lane has eight chunks of eight weights per row and unit: run A (four elements at k_of) and run B (RUNB further).
// raw() gives the four half2 of a chunk with the integers in place, in the order pair() defines for the activations:
// INTER 1: (A0 A2) (A1 A3) (B0 B2) (B1 B3); 0: (A0 A1) (A2 A3) (B0 B1) (B2 B3); 2: (A0 B0) (A1 B1) (A2 B2) (A3 B3).
// SH: bit j set = pair j holds 16 q, so its activations enter divided by 16. The first two pairs of chunk c belong
// to scale group ga(c), the last two to gb(c). apply(): acc += scale * c + offset * sum for group i of a row.
template <int ENC>
struct Gr;

template <>
struct Gr<E_Q4_0> {
  static constexpr int KU = 1, LW = 9, NG = 2, ROWB = 144, STAGE = 16 * ROWB, INTER = 1, RUNB = 16, SH = 0xC;
  __device__ static constexpr int ga(int c) { return c >> 2; }
  __device__ static constexpr int gb(int c) { return c >> 2; }
  __device__ static int k_of(int c, int t) { return (2 * t + (c >> 2)) * 32 + 4 * (c & 3); }
  __device__ static void load(const uint8_t* row, int t, uint32_t (&w)[LW]) {
    const uint32_t* p = reinterpret_cast<const uint32_t*>(row) + LW * t;
#pragma unroll
    for (int i = 0; i < LW; i++) w[i] = p[i];
  }
  __device__ static void raw(const uint32_t (&w)[LW], int c, int, uint32_t (&o)[4]) {
    const int i = c & 3;
    const uint32_t x = c >= 4 ? w[5 + i] : __funnelshift_r(w[i], w[i + 1], 16), y = x >> 8;
    o[0] = x & 0x000F000Fu, o[1] = y & 0x000F000Fu, o[2] = x & 0x00F000F0u, o[3] = y & 0x00F000F0u;
  }
  __device__ static float apply(const uint32_t (&w)[LW], int i, float c, float sum, float acc) {
    const __half2 h = *reinterpret_cast<const __half2*>(&w[i ? 4 : 0]);
    return fmaf(i ? __high2float(h) : __low2float(h), fmaf(-8.0f, sum, c), acc);
  }
};

template <>
struct Gr<E_Q4_1> {
  static constexpr int KU = 1, LW = 10, NG = 2, ROWB = 160, STAGE = 16 * ROWB, INTER = 1, RUNB = 16, SH = 0xC;
  __device__ static constexpr int ga(int c) { return c >> 2; }
  __device__ static constexpr int gb(int c) { return c >> 2; }
  __device__ static int k_of(int c, int t) { return (2 * t + (c >> 2)) * 32 + 4 * (c & 3); }
  __device__ static void load(const uint8_t* row, int t, uint32_t (&w)[LW]) {
    const uint2* p = reinterpret_cast<const uint2*>(row) + 5 * t;
#pragma unroll
    for (int i = 0; i < 5; i++) {
      const uint2 v = p[i];
      w[2 * i] = v.x, w[2 * i + 1] = v.y;
    }
  }
  __device__ static void raw(const uint32_t (&w)[LW], int c, int, uint32_t (&o)[4]) {
    const uint32_t x = w[5 * (c >> 2) + 1 + (c & 3)], y = x >> 8;
    o[0] = x & 0x000F000Fu, o[1] = y & 0x000F000Fu, o[2] = x & 0x00F000F0u, o[3] = y & 0x00F000F0u;
  }
  __device__ static float apply(const uint32_t (&w)[LW], int i, float c, float sum, float acc) {
    const __half2 h = *reinterpret_cast<const __half2*>(&w[5 * i]);
    return fmaf(__low2float(h), c, fmaf(__high2float(h), sum, acc));
  }
};

template <>
struct Gr<E_Q8_0> {
  static constexpr int KU = 1, LW = 17, NG = 2, ROWB = 272, STAGE = 16 * ROWB, INTER = 0, RUNB = 4, SH = 0;
  __device__ static constexpr int ga(int c) { return c >> 2; }
  __device__ static constexpr int gb(int c) { return c >> 2; }
  __device__ static int k_of(int c, int t) { return (2 * t + (c >> 2)) * 32 + 8 * (c & 3); }
  __device__ static void load(const uint8_t* row, int t, uint32_t (&w)[LW]) {
    const uint32_t* p = reinterpret_cast<const uint32_t*>(row) + LW * t;
#pragma unroll
    for (int i = 0; i < LW; i++) w[i] = p[i];
  }
  __device__ static void raw(const uint32_t (&w)[LW], int c, int, uint32_t (&o)[4]) {
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int i = 2 * (c & 3) + h;
      const uint32_t x = (c >= 4 ? w[9 + i] : __funnelshift_r(w[i], w[i + 1], 16)) ^ 0x80808080u;  // int8 -> biased byte
      o[2 * h] = __byte_perm(x, 0, 0x4140), o[2 * h + 1] = __byte_perm(x, 0, 0x4342);
    }
  }
  __device__ static float apply(const uint32_t (&w)[LW], int i, float c, float sum, float acc) {
    const __half2 h = *reinterpret_cast<const __half2*>(&w[i ? 8 : 0]);
    return fmaf(i ? __high2float(h) : __low2float(h), fmaf(-128.0f, sum, c), acc);
  }
};

template <>
struct Gr<E_Q4_K> {
  // words 0, 1: d * scale of sub-blocks 2t and 2t + 1, 2, 3: dmin * min (f32); 4 .. 11: the nibble bytes
  static constexpr int KU = 1, LW = 12, NG = 2, ROWB = 144, STAGE = 16 * ROWB, INTER = 1, RUNB = 32, SH = 0xC;
  __device__ static constexpr int ga(int) { return 0; }
  __device__ static constexpr int gb(int) { return 1; }
  __device__ static int k_of(int c, int t) { return 64 * t + 4 * c; }
  __device__ static void load(const uint8_t* row, int t, uint32_t (&w)[LW]) {
    const uint4 h = *reinterpret_cast<const uint4*>(row);
    const uint4 a = *reinterpret_cast<const uint4*>(row + 16 + 32 * t), b = *reinterpret_cast<const uint4*>(row + 32 + 32 * t);
    auto sb = [&](int i) { return ((i >> 2) == 0 ? h.y : (i >> 2) == 1 ? h.z : h.w) >> (8 * (i & 3)) & 0xffu; };
    const __half2 dd = *reinterpret_cast<const __half2*>(&h.x);
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
      w[e] = __float_as_uint(__low2float(dd) * (float)sc), w[2 + e] = __float_as_uint(__high2float(dd) * (float)mn);
    }
    w[4] = a.x, w[5] = a.y, w[6] = a.z, w[7] = a.w, w[8] = b.x, w[9] = b.y, w[10] = b.z, w[11] = b.w;
  }
  __device__ static void raw(const uint32_t (&w)[LW], int c, int, uint32_t (&o)[4]) {
    const uint32_t x = w[4 + c], y = x >> 8;
    o[0] = x & 0x000F000Fu, o[1] = y & 0x000F000Fu, o[2] = x & 0x00F000F0u, o[3] = y & 0x00F000F0u;
  }
  __device__ static float apply(const uint32_t (&w)[LW], int i, float c, float sum, float acc) {
    return fmaf(__uint_as_float(w[i]), c, fmaf(-__uint_as_float(w[2 + i]), sum, acc));
  }
};

template <>
struct Gr<E_Q6_K> {
  // quarter t = (p, s): for each half n 16 ql bytes (words 4n ..), for each half 16 qh bytes (words 8 + 4n ..),
  // then the f32 scales of sub-blocks (n, h): words 16 + 2n + h
  static constexpr int KU = 2, LW = 20, NG = 4, ROWB = 432, STAGE = 16 * ROWB, INTER = 0, RUNB = 64, SH = 0;
  __device__ static constexpr int ga(int c) { return (c >> 2) * 2; }
  __device__ static constexpr int gb(int c) { return (c >> 2) * 2 + 1; }
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
  __device__ static void raw(const uint32_t (&w)[LW], int c, int t, uint32_t (&o)[4]) {
    const uint32_t ql = w[c], qh = w[8 + c] >> (2 * (t >> 1));
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const uint32_t v = ((ql >> (4 * h)) & 0x0F0F0F0Fu) | (((qh >> (4 * h)) & 0x03030303u) << 4);
      o[2 * h] = __byte_perm(v, 0, 0x4140), o[2 * h + 1] = __byte_perm(v, 0, 0x4342);
    }
  }
  __device__ static float apply(const uint32_t (&w)[LW], int i, float c, float sum, float acc) {
    return fmaf(__uint_as_float(w[16 + i]), fmaf(-32.0f, sum, c), acc);
  }
};

template <>
struct Gr<E_MLX_U4> {
  // words 0 .. 7: blocks 2t and 2t + 1; 8, 9: their scales, 10, 11: their biases (f32)
  static constexpr int KU = 2, LW = 12, NG = 2, ROWB = 128, STAGE = 2 * 16 * ROWB, INTER = 2, RUNB = 4, SH = 0xA;
  __device__ static constexpr int ga(int c) { return c >> 2; }
  __device__ static constexpr int gb(int c) { return c >> 2; }
  __device__ static int k_of(int c, int t) { return (2 * t + (c >> 2)) * 32 + 8 * (c & 3); }
  __device__ static void raw(const uint32_t (&w)[LW], int c, int, uint32_t (&o)[4]) {
    const uint32_t x = w[c], y = x >> 8;
    o[0] = x & 0x000F000Fu, o[1] = x & 0x00F000F0u, o[2] = y & 0x000F000Fu, o[3] = y & 0x00F000F0u;
  }
  __device__ static float apply(const uint32_t (&w)[LW], int i, float c, float sum, float acc) {
    return fmaf(__uint_as_float(w[8 + i]), c, fmaf(__uint_as_float(w[10 + i]), sum, acc));
  }
};

__device__ __forceinline__ float4 gr_bf16x4(uint2 v) {
  return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16),
                     __uint_as_float(v.y & 0xffff0000u));
}

template <int ENC, int NM>
__global__ void __launch_bounds__(256, NM <= 4 ? 2 : 1)
gemv_rows_kernel(const GrArgs a, const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap smap,
                 const __grid_constant__ CUtensorMap bmap) {
  using S = Gr<ENC>;
  constexpr int KU = S::KU, LW = S::LW, NG = S::NG;
  extern __shared__ __align__(1024) uint8_t gr_smem_raw[];
  __shared__ int s_abort;
  __shared__ float s_max[NM][8], s_ss[NM][8];
  uint8_t* smem = gr_smem_raw + ((1024u - (smem_u32(gr_smem_raw) & 1023u)) & 1023u);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int kw = warp % a.KW, rw = warp / a.KW;
  const int aux_stage = ENC == E_MLX_U4 ? 2 * 16 * a.sb : 0;
  const int nst = a.nst;
  // shared memory: [warp][stage] weights | the same of scales and biases (MLX) | barriers | activations [row][hi, lo] |
  // block sums; the K warps' sums of the epilogue reuse it from the start
  uint8_t* ring = smem + warp * nst * S::STAGE;
  uint8_t* aring = smem + nwarps * nst * S::STAGE + warp * nst * aux_stage;
  uint8_t* after = smem + nwarps * nst * (S::STAGE + aux_stage);
  uint64_t* bars = reinterpret_cast<uint64_t*>(after) + warp * nst;
  uint8_t* xs = after + (nwarps * nst * 8 + 127) / 128 * 128;
  if (tid == 0) s_abort = 0;
  if (lane == 0) {
    for (int i = 0; i < nst; i++) mbar_init(bars + i, 1);
    mbar_fence_init();
  }
  __syncwarp();

  // this CTA: row group blockIdx.x / CK, K share blockIdx.x % CK (the rank in its cluster)
  const int rank = a.CK > 1 ? (int)(blockIdx.x % (unsigned)a.CK) : 0;
  const int grp = (int)(a.CK > 1 ? blockIdx.x / (unsigned)a.CK : blockIdx.x);
  const int st_lo = rank * a.cstages, st_hi = min(a.kstages, st_lo + a.cstages);
  const int my = st_hi - st_lo > kw ? (st_hi - st_lo - kw + a.KW - 1) / a.KW : 0;  // stages st_lo + kw, + KW, ...
  // first weight row of this warp; SwiGLU: the lower half of the row warps takes gate, the upper half up
  const int N = (int)a.N, last_row = (a.swiglu ? 2 * N : N) - 1, hw = a.RW >> 1;
  const int row0 = !a.swiglu ? (grp * a.RW + rw) * 16 : (grp * hw + (rw < hw ? rw : rw - hw)) * 16 + (rw < hw ? 0 : N);

  int c_left = my, c_stage = st_lo + kw, c_slot = 0;
  auto issue = [&]() {
    if (c_left <= 0) return;
    if (lane == 0 || (ENC == E_Q6_K && a.q6_mode == 0 && lane < 16)) {  // one lane asks for everything
      uint64_t* bar = bars + c_slot;
      uint8_t* dst = ring + c_slot * S::STAGE;
      if (lane == 0) mbar_expect_tx(bar, S::STAGE + aux_stage);
      if (ENC == E_Q6_K && a.q6_mode == 0) __syncwarp(0xffffu);
      if constexpr (ENC == E_MLX_U4) {
        uint8_t* adst = aring + c_slot * aux_stage;
        tma_box_g2s(dst, &wmap, c_stage * 64, row0, bar);
        tma_box_g2s(dst + 2048, &wmap, c_stage * 64 + 32, row0, bar);
        tma_box_g2s(adst, &smap, c_stage * (a.sb / 4), row0, bar);
        tma_box_g2s(adst + 16 * a.sb, &bmap, c_stage * (a.sb / 4), row0, bar);
      } else if constexpr (ENC == E_Q6_K) {
        // a stage is 420 bytes of a row that start anywhere on the 4-byte grid: copy from the 16-byte boundary below
        const int64_t coff = (int64_t)c_stage * 420;
        if (a.q6_mode == 1) {
          tma_box_g2s(dst, &wmap, (int)((coff >> 4) << 2), row0, bar);
        } else if (a.q6_mode == 2) {  // rows of 8 mod 16 bytes: the matrix as row pairs, even rows first in shared memory
          tma_box_g2s(dst, &wmap, (int)((coff >> 4) << 2), row0 >> 1, bar);
          tma_box_g2s(dst + 8 * S::ROWB, &wmap, (int)(((a.rb + coff) >> 4) << 2), row0 >> 1, bar);
        } else {
          const int r = row0 + lane > last_row ? last_row : row0 + lane;
          const uint8_t* src = a.data + (int64_t)r * a.rb + coff;
          src -= reinterpret_cast<uintptr_t>(src) & 15;
          bulk_g2s(dst + lane * S::ROWB, src, S::ROWB, bar);
        }
      } else {
        tma_box_g2s(dst, &wmap, c_stage * (S::ROWB / 4), row0, bar);
      }
    }
    c_left--, c_stage += a.KW;
    if (++c_slot == nst) c_slot = 0;
  };
  for (int q = 0; q < nst; q++) issue();

  // the weights do not depend on the kernels before this one; everything else does
  pdl_wait_then_trigger();

  // ---- activations: largest magnitude (and sum of squares) of every row, then hi / lo fragments of the K share ----
  const int units = (st_hi - st_lo) * KU, u_lo = st_lo * KU, all_units = a.K / GR_UNIT;
  const int pitch = a.cstages * KU * 512 + 64;  // of a plane: hi and lo of a row fall into different banks
  const uint8_t* zeros = xs + NM * 2 * pitch;  // KU * 512 bytes: what the lanes that feed zero columns read
  float* sx = reinterpret_cast<float*>(xs + NM * 2 * pitch + KU * 512);  // [row][unit][quarter][group]
  const int c8 = lane >> 2, ka = S::k_of(c8, t);  // a lane takes chunk c8 of quarter t of a unit
  constexpr int R = NM == 1 ? 4 : 1;              // units kept in registers between the passes
  float4 va[R], vb[R];
  auto load_unit = [&](int m, int u, float4& A, float4& B) {  // unit u of row m, norm weights applied
    const int64_t at = (int64_t)m * a.K + (int64_t)u * GR_UNIT + ka;
    if (a.x_bf16) {
      const uint16_t* p = reinterpret_cast<const uint16_t*>(a.x) + at;
      const uint2 ra = __ldcg(reinterpret_cast<const uint2*>(p)), rb = __ldcg(reinterpret_cast<const uint2*>(p + S::RUNB));
      A = gr_bf16x4(ra), B = gr_bf16x4(rb);
    } else {
      const float* p = reinterpret_cast<const float*>(a.x) + at;
      A = __ldcg(reinterpret_cast<const float4*>(p)), B = __ldcg(reinterpret_cast<const float4*>(p + S::RUNB));
    }
  };
  auto norm_unit = [&](int u, float4& A, float4& B) {
    const int k = u * GR_UNIT + ka;
    const uint8_t* nw = reinterpret_cast<const uint8_t*>(a.norm_w);
    float wa[4], wb[4];
    if (a.norm_type == E_F32) {
      const float4 p = *reinterpret_cast<const float4*>(nw + 4 * k), q = *reinterpret_cast<const float4*>(nw + 4 * (k + S::RUNB));
      wa[0] = p.x, wa[1] = p.y, wa[2] = p.z, wa[3] = p.w, wb[0] = q.x, wb[1] = q.y, wb[2] = q.z, wb[3] = q.w;
    } else {
#pragma unroll
      for (int e = 0; e < 4; e++) wa[e] = aux_load(nw, a.norm_type, k + e), wb[e] = aux_load(nw, a.norm_type, k + S::RUNB + e);
    }
    A = make_float4(A.x * wa[0], A.y * wa[1], A.z * wa[2], A.w * wa[3]);
    B = make_float4(B.x * wb[0], B.y * wb[1], B.z * wb[2], B.w * wb[3]);
  };
  auto sq = [](const float4& A) { return fmaf(A.x, A.x, A.y * A.y) + fmaf(A.z, A.z, A.w * A.w); };
  auto mx4 = [](const float4& A) { return fmaxf(fmaxf(fabsf(A.x), fabsf(A.y)), fmaxf(fabsf(A.z), fabsf(A.w))); };
  const bool keep = NM == 1 && a.CK == 1 && all_units <= R * nwarps;
#pragma unroll
  for (int m = 0; m < NM; m++) {
    if (m >= a.M) break;
    float mx = 0.f, ss = 0.f;
    for (int u0 = warp; u0 < all_units; u0 += R * nwarps) {
#pragma unroll
      for (int i = 0; i < R; i++) {
        va[i] = vb[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (u0 + i * nwarps < all_units) load_unit(m, u0 + i * nwarps, va[i], vb[i]);
      }
#pragma unroll
      for (int i = 0; i < R; i++) {
        if (a.norm_w && u0 + i * nwarps < all_units) {
          ss += sq(va[i]) + sq(vb[i]);
          norm_unit(u0 + i * nwarps, va[i], vb[i]);
        }
        mx = fmaxf(mx, fmaxf(mx4(va[i]), mx4(vb[i])));
      }
    }
    mx = warp_max(mx);
    if (a.norm_w) ss = warp_sum(ss);
    if (lane == 0) s_max[m][warp] = mx, s_ss[m][warp] = ss;
  }
  __syncthreads();
  // what turns accumulator units back into the product
  auto row_scale = [&](int m, float* sc) -> float {
    float mx = 0.f, ss = 0.f;
    for (int i = 0; i < nwarps; i++) mx = fmaxf(mx, s_max[m][i]), ss += s_ss[m][i];
    float inv;
    scale_for(mx, sc, &inv);
    inv *= GV_2P24;
    return a.norm_w ? inv * (1.0f / sqrtf(ss / (float)a.K + a.eps)) : inv;
  };
  for (int i = tid; i < KU * 32; i += blockDim.x) *reinterpret_cast<uint4*>(xs + NM * 2 * pitch + i * 16) = make_uint4(0, 0, 0, 0);
#pragma unroll
  for (int m = 0; m < NM; m++) {
    if (m >= a.M) break;
    float sc;
    row_scale(m, &sc);
    for (int u0 = warp; u0 < units; u0 += R * nwarps) {
#pragma unroll
      for (int i = 0; i < R; i++) {
        const int u = u0 + i * nwarps;
        if (u >= units) break;
        if (!keep) {
          load_unit(m, u_lo + u, va[i], vb[i]);
          if (a.norm_w) norm_unit(u_lo + u, va[i], vb[i]);
        }
        const float A[4] = {va[i].x * sc, va[i].y * sc, va[i].z * sc, va[i].w * sc};
        const float B[4] = {vb[i].x * sc, vb[i].y * sc, vb[i].z * sc, vb[i].w * sc};
        // block sums (of what is multiplied by the integers, in accumulator units)
        float sa = GV_2M24 * ((A[0] + A[1]) + (A[2] + A[3])), sb = GV_2M24 * ((B[0] + B[1]) + (B[2] + B[3]));
        if (NG == 2 && S::ga(0) == S::gb(0)) sa += sb;
        sa += __shfl_xor_sync(0xffffffffu, sa, 4);
        sa += __shfl_xor_sync(0xffffffffu, sa, 8);
        if (ENC == E_Q4_K) sa += __shfl_xor_sync(0xffffffffu, sa, 16);
        if (NG == 4 || ENC == E_Q4_K) {
          sb += __shfl_xor_sync(0xffffffffu, sb, 4);
          sb += __shfl_xor_sync(0xffffffffu, sb, 8);
          if (ENC == E_Q4_K) sb += __shfl_xor_sync(0xffffffffu, sb, 16);
        }
        if ((c8 & 3) == 0) {
          float* dst = sx + ((m * units + u) * 4 + t) * NG;
          dst[S::ga(c8)] = sa;
          if (NG == 4 || ENC == E_Q4_K) dst[S::gb(c8)] = sb;
        }
        float v[8];
        if (S::INTER == 1) {
          v[0] = A[0], v[1] = A[2], v[2] = A[1], v[3] = A[3], v[4] = B[0], v[5] = B[2], v[6] = B[1], v[7] = B[3];
        } else if (S::INTER == 0) {
          v[0] = A[0], v[1] = A[1], v[2] = A[2], v[3] = A[3], v[4] = B[0], v[5] = B[1], v[6] = B[2], v[7] = B[3];
        } else {
          v[0] = A[0], v[1] = B[0], v[2] = A[1], v[3] = B[1], v[4] = A[2], v[5] = B[2], v[6] = A[3], v[7] = B[3];
        }
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const float f = (S::SH >> j) & 1 ? 0.0625f : 1.0f;
          const float p = v[2 * j] * f, q = v[2 * j + 1] * f;
          const __half2 h = __floats2half2_rn(p, q);
          const __half2 l = __floats2half2_rn(p - __low2float(h), q - __high2float(h));
          hi[j] = *reinterpret_cast<const uint32_t*>(&h), lo[j] = *reinterpret_cast<const uint32_t*>(&l);
        }
        uint8_t* dst = xs + m * 2 * pitch + u * 512 + lane * 16;
        *reinterpret_cast<uint4*>(dst) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        *reinterpret_cast<uint4*>(dst + pitch) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
      }
    }
  }
  __syncthreads();

  // ---- main loop: only the lanes with g >> 1 == t feed non-zero B columns (hi for even g, lo for odd g) ------------
  const bool active = (g >> 1) == t;
  float acc[NM][2];
#pragma unroll
  for (int m = 0; m < NM; m++) acc[m][0] = acc[m][1] = 0.f;
  int slot = 0;
  unsigned parity = 0;
  int u = kw * KU;  // unit within the share
  for (int i = 0; i < my; i++, u += a.KW * KU) {
    if (!mbar_try_wait(bars + slot, parity) && !mbar_wait_bounded_sleepy(bars + slot, parity, GR_SPINS, &s_abort, 1000u)) {
      if (!s_abort) {
        s_abort = 1;
        report_wait_expired(a.error, DEV_ERR_GEMV_RING);
      }
      break;  // warp-uniform; the barriers below are still joined
    }
    const uint8_t* base = ring + slot * S::STAGE;
#pragma unroll
    for (int ku = 0; ku < KU; ku++) {
      uint32_t w0[LW], w1[LW];
      if constexpr (ENC == E_MLX_U4) {
        const uint8_t* ab = aring + slot * aux_stage;
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int piece = ((2 * t + h) ^ g) << 4;
          const uint4 v0 = *reinterpret_cast<const uint4*>(base + ku * 2048 + g * 128 + piece);
          const uint4 v1 = *reinterpret_cast<const uint4*>(base + ku * 2048 + 1024 + g * 128 + piece);
          w0[4 * h] = v0.x, w0[4 * h + 1] = v0.y, w0[4 * h + 2] = v0.z, w0[4 * h + 3] = v0.w;
          w1[4 * h] = v1.x, w1[4 * h + 1] = v1.y, w1[4 * h + 2] = v1.z, w1[4 * h + 3] = v1.w;
          const int si = a.group32 ? ku * 8 + 2 * t + h : ku * 4 + t;
          auto aux = [&](int off, int r) -> uint32_t {
            const uint32_t b = *reinterpret_cast<const uint16_t*>(ab + off + r * a.sb + 2 * si);
            return a.aux_f16 ? __float_as_uint(f16_bits_to_f32(b)) : b << 16;
          };
          w0[8 + h] = aux(0, g), w0[10 + h] = aux(16 * a.sb, g);
          w1[8 + h] = aux(0, g + 8), w1[10 + h] = aux(16 * a.sb, g + 8);
        }
      } else if constexpr (ENC == E_Q6_K) {
        const int64_t coff = (int64_t)(st_lo + kw + i * a.KW) * 420;
        const int ra = row0 + g, rb = ra + 8;
        const uint32_t o0 = (uint32_t)(reinterpret_cast<uintptr_t>(a.data) + (int64_t)(ra > last_row ? last_row : ra) * a.rb + coff) & 15u;
        const uint32_t o1 = (uint32_t)(reinterpret_cast<uintptr_t>(a.data) + (int64_t)(rb > last_row ? last_row : rb) * a.rb + coff) & 15u;
        const int s0 = a.q6_mode == 2 ? (g & 1) * 8 + (g >> 1) : g, s1 = a.q6_mode == 2 ? s0 + 4 : g + 8;
        const uint8_t *b0 = base + s0 * S::ROWB + o0, *b1 = base + s1 * S::ROWB + o1;
        if (ku == 0) S::template load<0>(b0, t, w0), S::template load<0>(b1, t, w1);
        else S::template load<2>(b0 + 210, t, w0), S::template load<2>(b1 + 210, t, w1);
      } else {
        S::load(base + g * S::ROWB, t, w0);
        S::load(base + (g + 8) * S::ROWB, t, w1);
      }
      if (ku == KU - 1) {  // everything of the slot is in registers: refill it before the math
        __syncwarp();
        issue();
      }
      const uint8_t* xb = active ? xs + (g & 1) * pitch + (u + ku) * 512 + t * 16 : zeros;
      const int row_step = active ? 2 * pitch : 0;
      const float* sb = sx + ((u + ku) * 4 + t) * NG;
      float ca[NM][4], cb[NM][4];
#pragma unroll
      for (int c = 0; c < 8; c++) {
        const bool fresh = c == 0 || (c == 4 && ENC != E_Q4_K);
        if (fresh) {
#pragma unroll
          for (int m = 0; m < NM; m++)
#pragma unroll
            for (int e = 0; e < 4; e++) ca[m][e] = cb[m][e] = 0.f;
        }
        uint32_t p0[4], p1[4];
        S::raw(w0, c, t, p0);
        S::raw(w1, c, t, p1);
#pragma unroll
        for (int m = 0; m < NM; m++) {
          const uint4 b = *reinterpret_cast<const uint4*>(xb + m * row_step + c * 64);
          mma_f16_16816(ca[m], p0[0], p1[0], p0[1], p1[1], b.x, b.y);
          mma_f16_16816(cb[m], p0[2], p1[2], p0[3], p1[3], b.z, b.w);
        }
        if (c == 7 || (c == 3 && ENC != E_Q4_K)) {
#pragma unroll
          for (int m = 0; m < NM; m++) {
            const float* sm = sb + m * units * 4 * NG;
            const int ia = S::ga(c), ib = S::gb(c);
            if (ia == ib) {
              acc[m][0] = S::apply(w0, ia, (ca[m][0] + ca[m][1]) + (cb[m][0] + cb[m][1]), sm[ia], acc[m][0]);
              acc[m][1] = S::apply(w1, ia, (ca[m][2] + ca[m][3]) + (cb[m][2] + cb[m][3]), sm[ia], acc[m][1]);
            } else {
              acc[m][0] = S::apply(w0, ia, ca[m][0] + ca[m][1], sm[ia], acc[m][0]);
              acc[m][1] = S::apply(w1, ia, ca[m][2] + ca[m][3], sm[ia], acc[m][1]);
              acc[m][0] = S::apply(w0, ib, cb[m][0] + cb[m][1], sm[ib], acc[m][0]);
              acc[m][1] = S::apply(w1, ib, cb[m][2] + cb[m][3], sm[ib], acc[m][1]);
            }
          }
        }
      }
    }
    if (++slot == nst) slot = 0, parity ^= 1u;
  }

  // ---- epilogue: the four quarters of a row hold disjoint blocks; then the K warps, then the cluster, in order -----
#pragma unroll
  for (int m = 0; m < NM; m++)
#pragma unroll
    for (int h = 0; h < 2; h++) {
      acc[m][h] += __shfl_xor_sync(0xffffffffu, acc[m][h], 1);
      acc[m][h] += __shfl_xor_sync(0xffffffffu, acc[m][h], 2);
    }
  float fac[NM];
#pragma unroll
  for (int m = 0; m < NM; m++) {
    float sc;
    fac[m] = m < a.M ? row_scale(m, &sc) : 0.f;
  }
  if (a.KW == 1 && a.CK == 1 && !a.swiglu) {
#pragma unroll
    for (int m = 0; m < NM; m++) {
      if (m >= a.M || (m & 3) != t) continue;  // lane quarter m mod 4 stores row m
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int n = row0 + 8 * h + g;
        if (n < N) a.y[(int64_t)m * N + n] = acc[m][h] * fac[m] + (a.residual ? a.residual[(int64_t)m * N + n] : 0.f);
      }
    }
    return;
  }
  const int rows = a.RW * 16, out_rows = a.swiglu ? rows >> 1 : rows;
  const int64_t n_base = (int64_t)grp * out_rows;
  __syncthreads();  // rings and activations are no longer used (every copy issued has been waited for)
  float* red = reinterpret_cast<float*>(smem);       // [KW][NM][rows]
  float* part = red + a.KW * NM * rows;              // [NM][rows]: this CTA's sums (CK > 1)
#pragma unroll
  for (int m = 0; m < NM; m++)
    if ((m & 3) == t) {
      red[(kw * NM + m) * rows + rw * 16 + g] = acc[m][0] * fac[m];
      red[(kw * NM + m) * rows + rw * 16 + 8 + g] = acc[m][1] * fac[m];
    }
  __syncthreads();
  auto local_sum = [&](int m, int r) -> float {
    float v = red[m * rows + r];
    for (int k = 1; k < a.KW; k++) v += red[(k * NM + m) * rows + r];
    return v;
  };
  auto finish = [&](int m, int r, float v, float up) {
    const int64_t n = n_base + r;
    if (n >= a.N) return;
    const int64_t at = (int64_t)m * a.N + n;
    if (a.swiglu) v = (v / (1.0f + expf(-v))) * up;
    else if (a.residual) v += a.residual[at];
    a.y[at] = v;
  };
  if (a.CK == 1) {
    for (int i = tid; i < a.M * out_rows; i += blockDim.x) {
      const int m = NM == 1 ? 0 : i / out_rows, r = i - m * out_rows;
      finish(m, r, local_sum(m, r), a.swiglu ? local_sum(m, out_rows + r) : 0.f);
    }
    return;
  }
  for (int i = tid; i < a.M * rows; i += blockDim.x) {
    const int m = NM == 1 ? 0 : i / rows, r = i - m * rows;
    part[i] = local_sum(m, r);
  }
  asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
  {
    const uint32_t pb = smem_u32(part);
    auto cluster_sum = [&](int i) -> float {
      float f[8], v = 0.f;
#pragma unroll
      for (int c = 0; c < 8; c++)
        if (c < a.CK) {
          uint32_t ra;
          asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(pb + 4u * (uint32_t)i), "r"(c));
          asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(f[c]) : "r"(ra) : "memory");
        }
#pragma unroll
      for (int c = 0; c < 8; c++)
        if (c < a.CK) v += f[c];
      return v;
    };
    for (int i = tid + rank * blockDim.x; i < a.M * out_rows; i += blockDim.x * a.CK) {
      const int m = NM == 1 ? 0 : i / out_rows, r = i - m * out_rows;
      finish(m, r, cluster_sum(m * rows + r), a.swiglu ? cluster_sum(m * rows + out_rows + r) : 0.f);
    }
  }
  // nobody leaves while its sums may still be read
  asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}

// ---- plan ------------------------------------------------------------------------------------------
struct GrPlan {
  int NM, RW, KW, CK, nst, kstages, cstages;
  int64_t groups;
  size_t smem;
  int per_sm;  // CTAs that share an SM
};

int gr_ku(int enc) { return enc == E_MLX_U4 || enc == E_Q6_K ? 2 : 1; }
int gr_ng(int enc) { return enc == E_Q6_K ? 4 : 2; }
int gr_stage_bytes(const WRef& w) {
  switch (w.enc) {
    case E_Q4_1: return Gr<E_Q4_1>::STAGE;
    case E_Q8_0: return Gr<E_Q8_0>::STAGE;
    case E_Q6_K: return Gr<E_Q6_K>::STAGE;
    case E_MLX_U4: return Gr<E_MLX_U4>::STAGE + 2 * 16 * (w.group == 32 ? 32 : 16);
    default: return Gr<E_Q4_0>::STAGE;
  }
}

size_t gr_smem(const WRef& w, const GrPlan& p) {
  const int warps = p.RW * p.KW, rows = p.RW * 16;
  const size_t ring = (size_t)warps * p.nst * gr_stage_bytes(w) + ((size_t)warps * p.nst * 8 + 127) / 128 * 128;
  const size_t units = (size_t)p.cstages * gr_ku(w.enc);
  const size_t x = (size_t)p.NM * 2 * (units * 512 + 64) + (size_t)gr_ku(w.enc) * 512 + (size_t)p.NM * units * 4 * gr_ng(w.enc) * 4;
  const size_t red = ((size_t)p.KW + 1) * p.NM * rows * 4;
  return 1024 + std::max(ring + x, red);
}

template <int ENC>
const void* gr_kernel_of(int nm) {
  switch (nm) {
    case 1: return reinterpret_cast<const void*>(gemv_rows_kernel<ENC, 1>);
    case 2: return reinterpret_cast<const void*>(gemv_rows_kernel<ENC, 2>);
    case 4: return reinterpret_cast<const void*>(gemv_rows_kernel<ENC, 4>);
    default: return reinterpret_cast<const void*>(gemv_rows_kernel<ENC, 8>);
  }
}
const void* gr_kernel(int enc, int nm) {
  switch (enc) {
    case E_Q4_1: return gr_kernel_of<E_Q4_1>(nm);
    case E_Q8_0: return gr_kernel_of<E_Q8_0>(nm);
    case E_Q6_K: return gr_kernel_of<E_Q6_K>(nm);
    case E_Q4_K: return gr_kernel_of<E_Q4_K>(nm);
    case E_MLX_U4: return gr_kernel_of<E_MLX_U4>(nm);
    default: return gr_kernel_of<E_Q4_0>(nm);
  }
}

// The split of the work, from sweeps of all plans over eleven shapes at 1 to 4 rows: eight warps per CTA (four where
// the stages are large), of which as many as divide K evenly share a tile; one 16-row tile per CTA up to 384 CTAs,
// more tiles beyond, so that the activations are not arranged more often than it takes to fill the GPU; a cluster
// only to let two CTAs fit an SM.
bool gr_make_plan(const WRef& w, int64_t M, bool swiglu, GrPlan* best) {
  const int64_t N = swiglu ? w.rows / 2 : w.rows;
  const int ku = gr_ku(w.enc), max_warps = w.enc == E_Q6_K ? 4 : 8;
  const int64_t tiles = (w.rows + 15) / 16;
  GrPlan p;
  p.NM = M <= 1 ? 1 : M <= 2 ? 2 : M <= 4 ? 4 : 8;
  p.kstages = (int)((w.cols + ku * GR_UNIT - 1) / (ku * GR_UNIT));
  bool found = false;
  for (const size_t limit : {(size_t)110 * 1024, (size_t)GR_MAX_SMEM}) {
    for (p.CK = 1; p.CK <= 8 && !found; p.CK *= 2) {
      if (p.CK > p.kstages) break;
      p.cstages = (p.kstages + p.CK - 1) / p.CK;
      if ((int64_t)p.cstages * (p.CK - 1) >= p.kstages) continue;  // every CTA of a cluster has work
      p.RW = swiglu ? 2 : 1;
      while (p.RW < max_warps && tiles * p.CK / p.RW >= 384) p.RW *= 2;
      int waste = 1 << 30;
      for (int kw = std::min(max_warps / p.RW, p.cstages); kw >= 1 && kw * 2 > std::min(max_warps / p.RW, p.cstages); kw--) {
        const int left = (p.cstages + kw - 1) / kw * kw - p.cstages;
        if (left < waste) waste = left, p.KW = kw;
      }
      while (p.RW * p.KW * 2 <= max_warps && tiles * p.CK / (2 * p.RW) >= 96) p.RW *= 2;
      p.nst = std::min((p.cstages + p.KW - 1) / p.KW, 2);
      p.smem = gr_smem(w, p);
      found = p.smem <= limit;
      if (found) *best = p;
    }
    if (found) break;
  }
  if (!found) return false;
  const void* kernel = gr_kernel(w.enc, best->NM);
  if (ensure_dynamic_smem(kernel, GR_MAX_SMEM)) return false;
  // Blocks of twice the rows and half the K warps where the blocks do not fit the SMs well. Measured on 2560 to 9216 rows x 512 to 8192
  // (and 5120 x 13824) of five encodings, weights out of L2 and out of HBM; us with the plan above / with twice the rows.
  //   More blocks than places: a second round of a few blocks costs as much as a full one (5120 x 4096 Q4_0, 320 blocks for 296
  //     places, one row 10.0 / 6.8, four rows 26.7 / 18.9), up to twelve stages per warp (5120 x 13824 Q8_0, four rows 56 / 60).
  //   Two blocks on some SMs: eight warps get through a tile's K faster alone than beside a second block.
  //     Two and more rows: up to eight stages per warp (4096 x 4096 four rows 15.7 / 14.5). Q4_K, whose decoding needs the warps, with two
  //       rows only while that makes two tiles per block (4096 x 4096 9.9 / 9.6, 6144 x 4096 12.2 / 12.7).
  //     One row: up to two stages per warp (3072 x 2048 Q4_0 4.3 / 4.0, 6144 x 1024 4.4 / 4.1; 6144 x 4096 with eight 7.0 / 7.4,
  //       Q8_0 8.0 / 8.6); up to four where that makes two tiles per block and leaves few SMs without one (4096 x 4096 Q4_0 5.8 / 5.6,
  //       3584 x 4096 Q8_0 7 % slower) or the encoding is MLX-U4 (4096 x 4096 5.9 / 5.1, 3584 x 4096 4 to 8 % faster); Q4_K never
  //       (4096 x 4096 6.2 / 6.5).
  const int tile_rows = swiglu ? 8 : 16;
  const int64_t sms = std::max(1, sm_count());
  auto alone = [&](int64_t ctas) {  // a block on its own rather than two
    const int stages = (2 * best->cstages + best->KW - 1) / best->KW;  // of a warp with twice the rows
    const bool pairs = best->RW == 1;                                  // two tiles per block then
    if (best->KW < 4 || ctas <= sms) return false;
    if (best->NM >= 2) return stages <= 8 && (best->NM > 2 || pairs || w.enc != E_Q4_K);
    if (w.enc == E_Q4_K) return false;
    return stages <= 2 || (stages <= 4 && pairs && (w.enc == E_MLX_U4 || 10 * ctas >= 17 * sms));
  };
  auto tail = [&](int64_t ctas) {  // a second round of a few blocks
    const int64_t places = best->per_sm * sms;
    return best->KW >= 2 && ctas > places && 10 * ctas <= 13 * places && 2 * best->cstages <= 12 * best->KW;
  };
  for (int i = 0;; i++) {
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&best->per_sm, kernel, best->RW * best->KW * 32, best->smem) != cudaSuccess || best->per_sm < 1)
      best->per_sm = 1;
    best->groups = (N + tile_rows * best->RW - 1) / (tile_rows * best->RW);
    const int64_t ctas = best->groups * best->CK;
    if (best->RW * best->KW != 8 || !(tail(ctas) || (i == 0 && alone(ctas)))) break;
    GrPlan q = *best;
    q.RW *= 2, q.KW /= 2;
    q.nst = std::min((q.cstages + q.KW - 1) / q.KW, 2);
    q.smem = gr_smem(w, q);
    if (q.smem > (size_t)GR_MAX_SMEM || (q.smem > (size_t)110 * 1024 && best->smem <= (size_t)110 * 1024)) break;
    *best = q;
  }
  if (best->groups * best->CK > 0x7fffffff) return false;
  return true;
}

// Plans are looked up, not searched, after the first product of a shape. Per thread; dropped when a program with
// very many shapes fills it.
bool gr_plan(const WRef& w, int64_t M, bool swiglu, GrPlan* p) {
  typedef std::array<int64_t, 4> Key;
  static thread_local std::map<Key, std::pair<bool, GrPlan>> plans;
  const Key key = {w.rows, w.cols, M, (int64_t)w.enc * 4 + (w.group == 32 ? 2 : 0) + (swiglu ? 1 : 0)};
  auto it = plans.find(key);
  if (it == plans.end()) {
    if (plans.size() >= 1024) plans.clear();
    GrPlan q;
    const bool ok = gr_make_plan(w, M, swiglu, &q);
    it = plans.emplace(key, std::make_pair(ok, q)).first;
  }
  *p = it->second.second;
  return it->second.first;
}

template <int ENC, int NM>
int gr_run(const GrArgs& a, const GrPlan& p, const CUtensorMap& wm, const CUtensorMap& sm, const CUtensorMap& bm, cudaStream_t s) {
  auto kernel = gemv_rows_kernel<ENC, NM>;
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), GR_MAX_SMEM)) return 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(p.groups * p.CK)), cfg.blockDim = dim3(p.RW * p.KW * 32);
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
int gr_run_enc(const GrArgs& a, const GrPlan& p, const CUtensorMap& wm, const CUtensorMap& sm, const CUtensorMap& bm, cudaStream_t s) {
  switch (p.NM) {
    case 1: return gr_run<ENC, 1>(a, p, wm, sm, bm, s);
    case 2: return gr_run<ENC, 2>(a, p, wm, sm, bm, s);
    case 4: return gr_run<ENC, 4>(a, p, wm, sm, bm, s);
    default: return gr_run<ENC, 8>(a, p, wm, sm, bm, s);
  }
}

}  // namespace

// Encodings, alignments and row counts the kernel reads: K a multiple of 256 (of 512 for MLX-U4 and Q6_K), rows
// whose hi / lo fragments fit shared memory, split over a cluster of eight at most.
bool gemv_rows_takes(const WRef& w, int64_t M) {
  if (M < 1 || M > 8 || w.rows < 1 || w.rows > (1LL << 30)) return false;
  const int64_t nm = M <= 1 ? 1 : M <= 2 ? 2 : M <= 4 ? 4 : 8;
  if (nm * ((w.cols + 8 * 512 - 1) / (8 * 512)) * (2048 + 128) > 160 * 1024) return false;
  const bool aligned = (reinterpret_cast<uintptr_t>(w.data) & 15) == 0;
  switch (w.enc) {
    case E_Q4_0:
    case E_Q4_1:
    case E_Q8_0:
    case E_Q4_K: return aligned && w.cols >= 256 && w.cols % 256 == 0;
    case E_Q6_K: return aligned && w.cols >= 512 && w.cols % 512 == 0;
    case E_MLX_U4:
      return aligned && w.cols >= 512 && w.cols % 512 == 0 && (w.group == 64 || w.group == 32) &&
             (w.aux == E_BF16 || w.aux == E_F16) && w.scales && w.biases &&
             ((reinterpret_cast<uintptr_t>(w.scales) | reinterpret_cast<uintptr_t>(w.biases)) & 15) == 0;
    default: return false;
  }
}

// Where this kernel is ahead of those that split K over CTAs and add the sums in a second launch (they keep one CTA per SM
// alive over all its tiles). Both sides measured on 100 shapes of 512 x 512 to 57344 x 8192 per encoding, us here / there.
// What decides is the plan, not the size: CTAs that do not fit the SMs at once leave a second round, and one that is
// nearly empty costs as much as a full one. 5120 x 13824 Q4_0 has 320 CTAs for 296 places: 26 / 17 (4096 x 14336, 256
// CTAs: 14.5 / 14.7); with eight tiles per CTA there are so many that it does not show (40745 x 1536: 14 / 15).
//   One row: vocabulary-sized matrices are done before a prologue has paid off (151936 x 1024 Q4_0 27 / 23, Q6_K 40 / 35;
//     between 65536 and 128256 rows the two are within 10 % either way); with rows of 16384 and more the others have to fall
//     back for Q8_0 and Q6_K (8192 x 28672 52 / 117 and 70 / 174; Q4_0 5120 x 25600 39 / 25); wide rows need more than a
//     CTA per SM (1288 x 12800 Q4_0 13 / 10). Q6_K, four warps per CTA, needs the SMs filled by one round from 4096 wide on
//     (4096 x 14336 21 / 23, 12288 x 4096 21 / 17, 2560 x 9728 17 / 15). MLX-U4 has the slower kernel on the other side.
//   Two rows: nearly always (12288 x 4096 Q4_0 15 / 38).
//   Three and four: the others are bound by arithmetic, so all but large matrices (24576 x 4096 Q4_0 43 / 39); Q8_0 also
//     those, unless clusters of four are left with short shares (27648 x 5120 80 / 69, 10240 x 5120 39 / 53); Q4_K, whose
//     other side is the row kernel, the large ones (24576 x 4096 45 / 87, 1024 x 1024 9 / 7, 5120 x 5120 with its second
//     round 42 / 29).
//   Five to eight bf16 rows, which the other kernel multiplies as one term: small matrices only (3072 x 1024 Q4_0 14 / 25,
//     4096 x 4096 40 / 38), Q4_K none (1024 x 1024 14 / 9).
//   Q6_K rows that are not multiples of 8 bytes (K an odd multiple of 512) come in a copy per row here; the row kernel on
//     the other side is ahead on few rows (2560 x 2560, four rows 20 / 12, eight bf16 rows 48 / 18).
// `fused`: the norm in front rides on this kernel, which saves a launch (3 us): below 32 MB of weights that is worth more
// than the differences above (a step of four 14B-sized layers 374 -> 338 us with this rule, of Q6_K 606 -> 507).
bool gemv_rows_prefers(const WRef& w, int64_t M, bool fused) {
  GrPlan p;
  if (!gemv_rows_takes(w, M) || !gr_plan(w, M, false, &p)) return false;
  const bool six = w.enc == E_Q6_K, odd = six && w.row_bytes() % 8, wide = w.cols >= 16384;
  const int64_t units = ((w.rows + 15) / 16) * (w.cols / GR_UNIT);
  const double places = (double)p.per_sm * std::max(1, sm_count()), rounds = p.groups * p.CK / places;
  const bool tail = rounds > 1 && rounds < 0.7 * std::ceil(rounds) && p.RW < (six ? 4 : 8);
  const bool chain = fused && !wide && w.total_bytes() < ((int64_t)32 << 20);
  if (M == 1) {
    if (w.rows >= 100000) return false;
    if (chain) return true;
    if (wide) return six || (w.enc == E_Q8_0 && !tail);
    if (six && w.cols >= 4096) return rounds >= 0.55 && rounds <= 1;
    if (tail && !(w.enc == E_MLX_U4 && w.cols <= 6144)) return false;
    return w.cols <= 12288 || p.groups * p.CK > sm_count();
  }
  if (wide) return false;
  if (M == 2) return chain || !odd || w.rows > 5200;
  if (M <= 4) {
    if (chain && (six || w.enc == E_Q8_0)) return true;
    if (odd) return w.cols < 2048 && w.rows >= 18000;
    if (six) return units < 65536;
    if (w.enc == E_Q8_0) return units < 32768 || p.CK < 4 || p.cstages > 5;
    if (w.enc == E_Q4_K) return chain || ((w.rows >= 8000 || w.cols >= 2048) && !(tail && units < 8192));
    return units < 16384 && !(p.per_sm == 1 && rounds > 1);
  }
  if (w.enc == E_Q4_K) return false;
  if (odd) return w.cols < 2048 && w.rows >= 18000 && M < 8;
  return units < (six ? 8192 : 1024);
}

// y[M, N] = x w^T + residual, or with `swiglu` (the matrix is [gate; up], N = rows / 2) silu(x gate^T) * (x up^T);
// with norm_w, x is RMSNorm(x) * norm_w. *handled = false when the product does not qualify.
int launch_gemv_rows(const WRef& w, const void* x, int x_type, int64_t M, const void* norm_w, int norm_type, float eps, float* y,
                     const float* residual, bool swiglu, cudaStream_t s, bool* handled) {
  *handled = false;
  if (!gemv_rows_takes(w, M) || (swiglu && w.rows % 32) || (reinterpret_cast<uintptr_t>(x) & 15)) return 0;
  GrPlan p;
  if (!gr_plan(w, M, swiglu, &p)) return 0;
  GrArgs a{};
  a.N = swiglu ? w.rows / 2 : w.rows, a.K = (int)w.cols, a.M = (int)M;
  a.kstages = p.kstages, a.cstages = p.cstages;
  a.RW = p.RW, a.KW = p.KW, a.CK = p.CK, a.nst = p.nst;
  a.swiglu = swiglu ? 1 : 0;
  a.x = x, a.x_bf16 = x_type == E_BF16 ? 1 : 0, a.norm_w = norm_w, a.norm_type = norm_type, a.eps = eps;
  a.y = y, a.residual = residual;
  a.error = device_error_word();
  if (!a.error) return 1;
  a.data = w.data, a.rb = w.row_bytes();
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
        if (make_row_box_map(w.data, (size_t)a.rb, w.rows, Gr<E_Q6_K>::ROWB / 4, 16, &wm)) return 1;
        a.q6_mode = 1;
      } else if (a.rb % 8 == 0 && w.rows % 2 == 0) {
        if (make_row_box_map(w.data, (size_t)a.rb * 2, w.rows / 2, Gr<E_Q6_K>::ROWB / 4, 8, &wm)) return 1;
        a.q6_mode = 2;
      }
      break;
    default: {
      const int words = w.enc == E_Q4_1 ? 40 : w.enc == E_Q8_0 ? 68 : 36;
      if (make_row_box_map(w.data, (size_t)w.row_bytes(), w.rows, words, 16, &wm)) return 1;
    }
  }
  if (w.enc != E_MLX_U4) sm = wm, bm = wm;
  int rc = 1;
  switch (w.enc) {
    case E_Q4_0: rc = gr_run_enc<E_Q4_0>(a, p, wm, sm, bm, s); break;
    case E_Q4_1: rc = gr_run_enc<E_Q4_1>(a, p, wm, sm, bm, s); break;
    case E_Q8_0: rc = gr_run_enc<E_Q8_0>(a, p, wm, sm, bm, s); break;
    case E_Q6_K: rc = gr_run_enc<E_Q6_K>(a, p, wm, sm, bm, s); break;
    case E_Q4_K: rc = gr_run_enc<E_Q4_K>(a, p, wm, sm, bm, s); break;
    case E_MLX_U4: rc = gr_run_enc<E_MLX_U4>(a, p, wm, sm, bm, s); break;
    default: break;
  }
  if (rc) return 1;
  DYN_CUDA(cudaGetLastError());
  *handled = true;
  return 0;
}

}  // namespace dyn
