// Causal GQA attention for prefill chunks: many query rows of ONE sequence at consecutive
// positions against an f32, bf16 or f16 KV cache, on the 5th-generation tensor cores.
//
// Same mathematics as the per-row kernel (kernels.rs:310-458: s = (q.k) * 1/sqrt(d), keys beyond the
// row's position masked, online max / sum merge, out / sum at the end), restructured the usual
// flash-attention way. One CTA = 128 consecutive rows of one query head = the 128 lanes of tensor memory:
//   * Q lies in tensor memory as (hi, lo) pairs (128 columns). 64-key tiles of K and V arrive as tensor copies.
//   * Two streams of eight warps take the tiles in turn, each with its own running (max, sum, out), so that one's softmax runs under
//     the other's MMAs. Two threads share a row: each has half of a tile's keys and half of the output's dims. A ninth warp per stream
//     (warps 16 and 17) asks for its tiles and issues its MMAs, a tenth (18 and 19) looks for values that are not finite. Per tile: S (64
//     columns) = Qhi Khi, a second accumulator for the terms with a lo part; a thread reads its half of the row twice (maximum, then
//     weights) and leaves P as (hi, lo) pairs in place of S; U (128 columns) = P V, with V's tile as an operand that is
//     contiguous along N; a thread folds its half of U into 64 f32 sums. The second score accumulator uses U's columns, so a
//     stream needs 192, and 512 hold everything.
//   * Keys are also dealt over the CTAs of a cluster where there are few (head, row block) pairs (16 heads x 512 rows: 64); all streams'
//     states meet through shared memory at the end and are merged in a fixed order.
//   * From 32 rows on. Against the kernels for fewer (attention_decode.cu, f32 caches the slices of kernels_misc.cu), us here / there with
//     16 heads: bf16 16 rows at 0 6.1 / 5.3, 32 at 0 6.2 / 10.3, 32 at 1000 17.4 / 30.1; f32 32 at 0 9.7 / 7.1, 48 at 0 10.0 / 9.7,
//     32 at 200 11.8 / 19.3. (Calls of 17 to 31 rows behind a context would gain by a lower line.)
// On mma.sync (16 rows per warp, 64 per CTA) the MMAs alone kept an SM busy four times as long: 512 rows of 16 heads at 1536, f32
// cache, 92 us.
//
// The cache entries are used in their stored type (exact); the f32 operands Q and P enter as hi + lo pairs of that type. f16
// operands: query rows are scaled by a power of two, weights by 2^14.
// f32 caches: a first pass turns the sequence's keys and values into (hi, lo) pairs of f16, every 64-key
// tile of a head scaled by a power of two of its own (no overflow, nothing lost to subnormals), so a pair
// holds the entry to 2^-24 of its magnitude. The products take three MMAs (hi hi, lo hi, hi lo; what is dropped is 2^-24 of a
// term). The tile scales are exact: the keys' multiply the scores, the values' a tile's share of the output.
// Weight 0 times an entry that is not finite would reach rows that do not see its key. On 2-byte caches a warp per stream, idle
// otherwise, looks through the values of the tiles on the diagonal while their scores are made, puts zeros in such places and
// marks the keys; where there are any, the idle warps add the entry itself to the states of the rows that see its key. (Code for
// it in the softmax warps, in their loop or behind it, costs the loop registers: 2 to 7 % of a call.)
// Every tile's products start from zero and join the running output by a rounded fma, because a tensor-core accumulation
// truncates.
#include <algorithm>

#include "common.cuh"
#include "tensor_map.cuh"
#include "umma.cuh"

namespace dyn {

namespace {

constexpr int FA_D = 128;           // head dim handled by this kernel
constexpr int FA_BR = 128;          // query rows per CTA
constexpr int FA_SPLIT_TILE = 64;   // keys per tile = per scale of the (hi, lo) form
constexpr int FA_BOX = 64 * 128;    // bytes of a tensor copy: 64 keys x 64 two-byte elements
constexpr int FA_WORKERS = 576;     // two streams of eight softmax warps, one issuing warp each
constexpr int FA_THREADS = 640;     // whole warpgroups: registers are dealt out per group
// 640 threads start with 96 registers each = 61440; 512 x 112 + 128 x 32 = 61440
constexpr int FA_SOFTMAX_REGS = 112, FA_ISSUE_REGS = 32;
static_assert(512 * FA_SOFTMAX_REGS + 128 * FA_ISSUE_REGS <= FA_THREADS * 96, "the groups' shares come out of the launch's registers");
constexpr int fa_items(int kv) { return kv == E_F32 ? 3 : 6; }             // K or V tiles a stream keeps in shared memory
constexpr int fa_item_bytes(int kv) { return (kv == E_F32 ? 4 : 2) * FA_BOX; }
constexpr int FA_Q_BYTES = 32768;   // half of the query rows' dims in f32, in the last places of a stream's tiles
constexpr int FA_PITCH = FA_D + 4;  // floats per row of a stream's final state
constexpr int FA_SMEM = 2 * 3 * 4 * FA_BOX + 1024;
static_assert(2 * FA_BR * FA_PITCH * 4 <= FA_SMEM - 1024, "the streams' final states reuse the tiles' memory");

// (hi, lo) packed pairs of two f32 values. The packing conversions matter: scalar ones share the unit of the exponentials.
template <bool BF>
__device__ __forceinline__ void fa_split2(float x, float y, uint32_t* hi, uint32_t* lo) {
  if constexpr (BF) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y), l = __floats2bfloat162_rn(x - __low2float(h), y - __high2float(h));
    *hi = *reinterpret_cast<const uint32_t*>(&h), *lo = *reinterpret_cast<const uint32_t*>(&l);
  } else {
    const __half2 h = __floats2half2_rn(x, y), l = __floats2half2_rn(x - __low2float(h), y - __high2float(h));
    *hi = *reinterpret_cast<const uint32_t*>(&h), *lo = *reinterpret_cast<const uint32_t*>(&l);
  }
}

// Power of two that puts `mx` into [2^12, 2^13), and its inverse; magnitudes below 2^-41 share one scale.
__device__ __forceinline__ void fa_pow2_scale(float mx, float* sc, float* inv) {
  int e = 0;  // mx = [0.5, 1) * 2^e
  if (mx > 0.f && mx <= 3.40282347e38f) e = max((int)(__float_as_uint(mx) >> 23) - 126, -40);
  *sc = __uint_as_float((uint32_t)(127 + 13 - e) << 23);
  *inv = __uint_as_float((uint32_t)(127 - 13 + e) << 23);
}

// (a, b) = (a, b) * f + (x, y) * s, two values per instruction; s is a power of two.
__device__ __forceinline__ void fa_fold2(float& a, float& b, float f, float x, float y, float s) {
  asm("{\n\t.reg .b64 o, g, u, t;\n\t"
      "mov.b64 o, {%0, %1};\n\tmov.b64 g, {%2, %2};\n\tmov.b64 u, {%3, %4};\n\tmov.b64 t, {%5, %5};\n\t"
      "mul.rn.f32x2 u, u, t;\n\tfma.rn.f32x2 o, o, g, u;\n\tmov.b64 {%0, %1}, o;\n\t}"
      : "+f"(a), "+f"(b)
      : "f"(f), "f"(x), "f"(y), "f"(s));
}

// f32 cache -> f16 pairs: out[plane][kv head][key][hi 128 | lo 128], inv[plane][kv head][tile]; plane 0 = keys,
// 1 = values. One block per (tile of 64 keys, kv head, plane); 64 bytes in flight per thread and load step.
// Entries that are not finite have no part in the scale. Among the values they become zeros and the key is marked in
// `lost`: weight 0 times such an entry would reach the rows that do not see the key. (A key's own reach its scores only.)
__global__ void __launch_bounds__(256)
fa_split_kernel(const float* kc, const float* vc, int64_t nkv, int64_t cap, int64_t seq,
                int64_t nkeys, __half* out, float* inv, unsigned* lost) {
  __shared__ float red[8];
  __shared__ unsigned s_lost[2];
  const int64_t tile = blockIdx.x, kvh = blockIdx.y, plane = blockIdx.z;
  const float* src = (plane ? vc : kc) + ((seq * nkv + kvh) * cap + tile * FA_SPLIT_TILE) * FA_D;
  const int left = (int)min((int64_t)FA_SPLIT_TILE, nkeys - tile * FA_SPLIT_TILE) * (FA_D / 4);  // float4s
  float4 v[8];
  float mx = 0.f;
  pdl_wait_then_trigger();
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const int i = threadIdx.x + 256 * k;
    v[k] = i < left ? __ldcg(reinterpret_cast<const float4*>(src) + i) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  if (threadIdx.x < 2) s_lost[threadIdx.x] = 0;
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 8; k++) {
    float m = fmaxf(fmaxf(fabsf(v[k].x), fabsf(v[k].y)), fmaxf(fabsf(v[k].z), fabsf(v[k].w)));
    const float sum = fabsf(v[k].x * 0.f + v[k].y * 0.f) + fabsf(v[k].z * 0.f + v[k].w * 0.f);  // 0 unless one is not finite
    if (sum != 0.f) {
      float* e = reinterpret_cast<float*>(&v[k]);
      m = 0.f;
#pragma unroll
      for (int i = 0; i < 4; i++) {
        if (fabsf(e[i]) <= 3.40282347e38f) m = fmaxf(m, fabsf(e[i]));
        else if (plane) e[i] = 0.f;
      }
      const int key = (threadIdx.x + 256 * k) / (FA_D / 4);
      atomicOr(&s_lost[key >> 5], 1u << (key & 31));
    }
    mx = fmaxf(mx, m);
  }
  mx = warp_max(mx);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
  __syncthreads();
  mx = red[0];
#pragma unroll
  for (int i = 1; i < 8; i++) mx = fmaxf(mx, red[i]);
  float sc, is;
  fa_pow2_scale(mx, &sc, &is);
  if (threadIdx.x == 0) inv[(plane * nkv + kvh) * (cap / FA_SPLIT_TILE) + tile] = is;
  if (plane && threadIdx.x < 2) lost[kvh * (cap / 32) + 2 * tile + threadIdx.x] = s_lost[threadIdx.x];
  __half* dst = out + ((plane * nkv + kvh) * cap + tile * FA_SPLIT_TILE) * (2 * FA_D);
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const int i = threadIdx.x + 256 * k;
    if (i >= left) continue;
    uint2 hi, lo;
    fa_split2<false>(v[k].x * sc, v[k].y * sc, &hi.x, &lo.x);
    fa_split2<false>(v[k].z * sc, v[k].w * sc, &hi.y, &lo.y);
    __half* row = dst + (i / (FA_D / 4)) * (2 * FA_D) + (i % (FA_D / 4)) * 4;
    *reinterpret_cast<uint2*>(row) = hi;
    *reinterpret_cast<uint2*>(row + FA_D) = lo;
  }
}

struct FaArgs {
  const float* q;     // [rows, nh, d]
  int64_t krow, vrow; // row of the tensor maps at which the sequence's keys (values) of kv head 0 start
  const float* kinv;  // f32 caches: inverse tile scales [kv head][cap / 64]
  const float* vinv;
  const unsigned* vlost;  // f32 caches: a bit per key whose values are not all finite [kv head][cap / 32]
  const uint16_t* vals;   // 2-byte caches: the sequence's values of kv head 0
  float* ctx;         // [rows, nh * d]
  int* error;
  int64_t rows, nh, nkv, cap, base_pos;
  int64_t ldq;        // floats between consecutive rows of q
};

// kind::f16 descriptor: M = 128, N = n, f32 accumulation; BF: bf16 operands; mn: B contiguous along N.
__device__ __forceinline__ uint32_t fa_idesc(int n, bool bf, bool mn) {
  return umma_idesc(n) | (bf ? (1u << 7) | (1u << 10) : 0u) | (mn ? 1u << 16 : 0u);
}
// B operand contiguous along N, 128-byte swizzle: 64 elements of N per 128-byte row, a row per K element; LBO = the next 64 of N (the
// next box), SBO = the next eight of K.
__device__ __forceinline__ uint64_t fa_desc_mn(uint32_t smem_addr) {
  return (uint64_t)((smem_addr >> 4) & 0x3fff) | ((uint64_t)(FA_BOX >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void tmem_st8(uint32_t addr, const uint32_t (&v)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]),
               "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}

// Bit 15 of each half that is not finite, of two f16 or bf16 entries.
template <bool BF>
__device__ __forceinline__ uint32_t fa_not_finite2(uint32_t w) {
  return BF ? ((w & 0x7f807f80u) + 0x00800080u) & 0x80008000u : ((w & 0x7c007c00u) + 0x04000400u) & 0x80008000u;
}
// c plus two entries times zero: not a number once one of them was not finite.
template <bool BF>
__device__ __forceinline__ uint32_t fa_fma0(uint32_t w, uint32_t c) {
  uint32_t r;
  if constexpr (BF) asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(w), "r"(0u), "r"(c));
  else asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(w), "r"(0u), "r"(c));
  return r;
}
// Adds what is not finite of two entries to their sums.
template <bool BF>
__device__ __forceinline__ void fa_add_not_finite2(float* o, uint32_t w) {
  const uint32_t m = fa_not_finite2<BF>(w);
  if (m & 0x8000u) o[0] += BF ? __uint_as_float(w << 16) : f16_bits_to_f32(w & 0xffffu);
  if (m & 0x80000000u) o[1] += BF ? __uint_as_float(w & 0xffff0000u) : f16_bits_to_f32(w >> 16);
}

// NS CTAs share the keys of a row block (a template: each count's merge, and the loop in front of it, in as few registers as it needs).
template <int KV, int NS>
__global__ void __launch_bounds__(FA_THREADS, 1)
attention_prefill_kernel(const FaArgs a, const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap kmap,
                         const __grid_constant__ CUtensorMap vmap) {
  constexpr bool SPLIT = KV == E_F32, BF = KV == E_BF16;
  constexpr bool SCALED = !BF;                      // f16 terms: the query rows and the weights need scales
  constexpr float PMUL = SCALED ? 16384.0f : 1.0f;  // the weights' (the sum carries it too)
  constexpr int R = fa_items(KV), ITEM = fa_item_bytes(KV);
  // parts of a tile's keys that are folded into the output one by one: with f32 caches the tensor cores' truncation is the largest
  // error (4 large terms in a chain: 1.7 times that of 2 for values of one sign)
  constexpr int FOLDS = SPLIT ? 2 : 1;
  constexpr uint32_t Q_COL = 384;                   // hi in 64 columns, lo in 64; stream i: S at 192 i, U at 192 i + 64
  constexpr float LOWEST = -3.40282347e38f;
  extern __shared__ __align__(1024) uint8_t fa_smem[];
  __shared__ uint64_t item_full[2][6], q_full[2], s_full[2], p_full[2], u_full[2], u_free[2], started;
  __shared__ uint32_t tmem_base_s;
  __shared__ int s_abort;
  __shared__ float s_x[4][FA_BR];         // largest magnitude of a quarter of the dims
  __shared__ float s_mx[2][2][2][FA_BR];  // [tile parity][stream][half of the keys]: a row's maximum
  __shared__ float s_m[2][FA_BR], s_l[2][2][FA_BR];
  __shared__ uint4 s_lost4[2];            // 2-byte caches: a bit per key whose values are not all finite, of the tiles from diag0 on
  unsigned* const s_lost = reinterpret_cast<unsigned*>(s_lost4);
  uint8_t* const smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(fa_smem) + 1023) & ~uintptr_t(1023));
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int rank = (int)(blockIdx.x % (unsigned)NS);
  const int64_t h = blockIdx.x / (unsigned)NS, rb = gridDim.y - 1 - blockIdx.y;  // the longest row blocks start first
  const int64_t kvh = h / (a.nh / a.nkv);
  // keys 0 .. last position of the CTA's rows, in tiles of 64; in turn to the first streams of the NS CTAs of a cluster,
  // then to the second ones: with two to eight tiles, streams of one CTA get in each other's way (96 rows at 0 on an f16 cache, two tiles: 11.3 us
  // in one CTA, 9.0 in two; 128 at 5, three: 14.6 in one, 9.9 in four)
  const int64_t row_lo = rb * FA_BR, row_hi = min(row_lo + FA_BR, a.rows) - 1;
  const int last = (int)(a.base_pos + row_hi), ntiles = last / FA_SPLIT_TILE + 1;
  const int stream = warp < 16 ? warp >> 3 : warp & 1;
  const int first = rank + NS * stream, step = 2 * NS, mine = first < ntiles ? (ntiles - first + step - 1) / step : 0;
  const int diag0 = (int)(a.base_pos + row_lo + 1) / FA_SPLIT_TILE;  // the first of up to three tiles whose keys not all rows see

  if (tid == 0) {
    s_abort = 0;
    if constexpr (!SPLIT) s_lost4[0] = s_lost4[1] = make_uint4(0, 0, 0, 0);
    for (int i = 0; i < 2; i++) {
      for (int j = 0; j < 6; j++) mbar_init(&item_full[i][j], 1);
      mbar_init(q_full + i, 1), mbar_init(s_full + i, 1), mbar_init(p_full + i, SPLIT ? 8 : 9), mbar_init(u_full + i, 1), mbar_init(u_free + i, 8);
    }
    mbar_init(&started, 1);
    mbar_fence_init();
  }
  if (warp == 17 && lane < 3) {  // (their first use is 0.1 us shorter for it)
    const CUtensorMap* const m = lane == 0 ? &qmap : lane == 1 ? &kmap : &vmap;
    asm volatile("prefetch.tensormap [%0];" ::"l"(m) : "memory");
  }
  // Tensor memory is taken before this block lets the next kernel start, so that kernel cannot take it first and then wait for this one.
  if (warp == 16) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base_s, s_col = tmem + 192u * stream, u_col = s_col + 64u;
  pdl_wait();
  if (tid == 0) pdl_trigger();

  uint8_t* const items = smem + stream * (R * ITEM);
  float o[FA_D / 2];  // the running output of this thread's row and half of the dims
  float m_run = LOWEST, l_run = 0.f;

  // every thread's part of the ends of the loops: copies and products in flight land before shared memory is used again
  auto drained = [&] {
    if (s_abort) {
      const long long t0 = clock64();
      while (clock64() - t0 < (1LL << 22)) {
      }
    }
    __syncwarp();
    __syncthreads();  // nobody reads the tiles any more
  };
  auto cluster_sync = [] {
    if constexpr (NS > 1) asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
    else __syncthreads();
  };
  auto any_lost = [&] {  // the same for the whole CTA, behind drained()
    const uint4 u = s_lost4[0], v = s_lost4[1];
    return (u.x | u.y | u.z | u.w | v.x | v.y) != 0;
  };
  // row of this thread, and its half of a tile's keys and of the output's dims
  const int row = (warp & 3) * 32 + lane, part = (warp >> 2) & 1;

  if (warp < 16) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(FA_SOFTMAX_REGS));
    const uint32_t tlane = (uint32_t)((warp & 3) * 32) << 16;
    const int pos = (int)(a.base_pos + min(row_lo + row, a.rows - 1));
    // ---- Q: four threads share a row, 32 dims each
    float scale = 1.0f / sqrtf((float)FA_D);
    {
      if (!mbar_wait_bounded(q_full + stream, 0, TG_SPINS, &s_abort) && !s_abort) s_abort = 5;
      const uint8_t* q = items + R * ITEM - FA_Q_BYTES + part * (FA_Q_BYTES / 2) + row * 128;
      float4 x[8];
#pragma unroll
      for (int i = 0; i < 8; i++) x[i] = *reinterpret_cast<const float4*>(q + ((i ^ (row & 7)) << 4));
      float sc = 1.0f;
      if constexpr (SCALED) {
        float mx = 0.f;
#pragma unroll
        for (int i = 0; i < 8; i++) mx = fmaxf(mx, fmaxf(fmaxf(fabsf(x[i].x), fabsf(x[i].y)), fmaxf(fabsf(x[i].z), fabsf(x[i].w))));
        s_x[2 * stream + part][row] = mx;
        asm volatile("bar.sync 1, 512;" ::: "memory");
        mx = fmaxf(fmaxf(s_x[0][row], s_x[1][row]), fmaxf(s_x[2][row], s_x[3][row]));
        float inv;
        fa_pow2_scale(mx, &sc, &inv);
        scale *= inv;
      }
#pragma unroll
      for (int i = 0; i < 8; i += 4) {
        uint32_t hi[8], lo[8];
#pragma unroll
        for (int j = 0; j < 4; j++) {
          fa_split2<BF>(x[i + j].x * sc, x[i + j].y * sc, &hi[2 * j], &lo[2 * j]);
          fa_split2<BF>(x[i + j].z * sc, x[i + j].w * sc, &hi[2 * j + 1], &lo[2 * j + 1]);
        }
        const uint32_t at = tmem + tlane + Q_COL + 32u * stream + 16u * part + 2u * i;
        tmem_st8(at, hi);
        tmem_st8(at + 64u, lo);
      }
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    tc_fence_before();
    asm volatile("bar.sync 2, %0;" ::"n"(FA_WORKERS) : "memory");  // Q is complete, and its place in shared memory free
#pragma unroll
    for (int d = 0; d < FA_D / 2; d++) o[d] = 0.f;
    float nki = 1.f, nvi = 1.f;
    unsigned nl0 = 0, nl1 = 0;
    auto tile_info = [&](int i) {  // of the stream's tile i, a tile ahead
      if constexpr (SPLIT) {
        const int t = first + i * step;
        nki = __ldcg(a.kinv + kvh * (a.cap / FA_SPLIT_TILE) + t), nvi = __ldcg(a.vinv + kvh * (a.cap / FA_SPLIT_TILE) + t);
        nl0 = __ldcg(a.vlost + kvh * (a.cap / 32) + 2 * t), nl1 = __ldcg(a.vlost + kvh * (a.cap / 32) + 2 * t + 1);
      }
    };
    if (mine) tile_info(0);
    int item = 1;  // of the tile's values
    unsigned iphase = 0;
#pragma unroll 1
    for (int i = 0; i < mine; i++) {
      const int key0 = (first + i * step) * FA_SPLIT_TILE;
      const float ks = scale * nki, vi = SPLIT ? nvi * (1.0f / PMUL) : 1.0f;
      const unsigned lost0 = nl0, lost1 = nl1;
      if (i + 1 < mine) tile_info(i + 1);
      const int lim = pos - key0;  // keys 0 .. lim of the tile are seen
      const bool masked = key0 + FA_SPLIT_TILE - 1 > a.base_pos + row_lo + (warp & 3) * 32;
      // a failed wait is not left with a break: every warp keeps the same sequence of barriers (and the next waits return at
      // once, because they look at s_abort)
      if (!mbar_wait_bounded(s_full + stream, i & 1, TG_SPINS, &s_abort) && !s_abort) s_abort = 1;
      tc_fence_after();
      float mx = LOWEST;
#pragma unroll 1
      for (int c = 2 * part; c < 2 * part + 2; c++) {
        uint32_t x[16], y[16];
        tmem_ld16(s_col + tlane + 16u * c, x);
        tmem_ld16(u_col + tlane + 16u * c, y);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (masked) {
#pragma unroll
          for (int e = 0; e < 16; e++)
            if (16 * c + e <= lim) mx = fmaxf(mx, __fmul_rn(__uint_as_float(x[e]) + __uint_as_float(y[e]), ks));
        } else {
          float m1 = LOWEST;
#pragma unroll
          for (int e = 0; e < 16; e += 2) {
            mx = fmaxf(mx, __fmul_rn(__uint_as_float(x[e]) + __uint_as_float(y[e]), ks));
            m1 = fmaxf(m1, __fmul_rn(__uint_as_float(x[e + 1]) + __uint_as_float(y[e + 1]), ks));
          }
          mx = fmaxf(mx, m1);
        }
      }
      s_mx[i & 1][stream][part][row] = mx;
      asm volatile("bar.sync %0, 256;" ::"r"(3 + stream) : "memory");
      mx = fmaxf(mx, s_mx[i & 1][stream][part ^ 1][row]);
      const float mn = fmaxf(m_run, mx), f = expf(m_run - mn);
      m_run = mn, l_run *= f;
#pragma unroll 1
      for (int c = 2 * part; c < 2 * part + 2; c++) {
        uint32_t x[16], y[16];
        tmem_ld16(s_col + tlane + 16u * c, x);
        tmem_ld16(u_col + tlane + 16u * c, y);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        uint32_t hi[8], lo[8];
        float sum = 0.f;
#pragma unroll
        for (int e = 0; e < 16; e++) x[e] = __float_as_uint(expf(__fmul_rn(__uint_as_float(x[e]) + __uint_as_float(y[e]), ks) - m_run) * PMUL);
        if (masked) {  // exactly 0
#pragma unroll
          for (int e = 0; e < 16; e++)
            if (16 * c + e > lim) x[e] = 0;
        }
#pragma unroll
        for (int e = 0; e < 8; e++) {
          const float p0 = __uint_as_float(x[2 * e]), p1 = __uint_as_float(x[2 * e + 1]);
          sum += p0 + p1;
          fa_split2<BF>(p0, p1, &hi[e], &lo[e]);
        }
        l_run += sum;
        tmem_st8(s_col + tlane + 16u * c, hi);
        tmem_st8(s_col + tlane + 16u * c + 8u, lo);
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      if (SPLIT && key0 + FA_SPLIT_TILE - 1 > last) {
        // values past the last row may hold anything, and their weight 0 must stay 0: zeros
        if (!mbar_wait_bounded(&item_full[stream][item], iphase, TG_SPINS, &s_abort) && !s_abort) s_abort = 2;
        const int dead = last + 1 - key0;
        for (int e = tid & 255; e < (FA_SPLIT_TILE - dead) * 8 * (ITEM / FA_BOX); e += 256)
          *reinterpret_cast<uint4*>(items + item * ITEM + (e / ((FA_SPLIT_TILE - dead) * 8)) * FA_BOX + dead * 128 + e % ((FA_SPLIT_TILE - dead) * 8) * 16) = make_uint4(0, 0, 0, 0);
        fence_async_smem();
      }
      item += 2;
      if (item >= R) item -= R, iphase ^= 1u;
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full + stream);
#pragma unroll 1
      for (int q = 0; q < FOLDS; q++) {
        if (!mbar_wait_bounded(u_full + stream, (FOLDS * i + q) & 1, TG_SPINS, &s_abort) && !s_abort) s_abort = 3;
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < 4; c += 2) {
          uint32_t u[2][16];
          tmem_ld16(u_col + tlane + 64u * part + 16u * c, u[0]);
          tmem_ld16(u_col + tlane + 64u * part + 16u * c + 16u, u[1]);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int e = 0; e < 32; e += 2)
            fa_fold2(o[16 * c + e], o[16 * c + e + 1], q ? 1.0f : f, __uint_as_float(u[e >> 4][e & 15]), __uint_as_float(u[e >> 4][(e & 15) + 1]), vi);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(u_free + stream);
      }
      if (SPLIT && (lost0 | lost1)) {  // their pairs are zeros: rows that see one of them get no number, earlier rows are not touched
        const int key = lost0 ? __ffs(lost0) - 1 : 31 + __ffs(lost1);
        if (key <= lim) {
#pragma unroll
          for (int d = 0; d < FA_D / 2; d++) o[d] = __int_as_float(0x7fffffff);
        }
      }
    }
    drained();
    // ---- the streams' states: [stream][row][pitch]
    float* const state = reinterpret_cast<float*>(smem);
    if (mine && row_lo + (row & ~31) < a.rows) {  // (what is read below)
      float* const p = state + (stream * FA_BR + row) * FA_PITCH + part * (FA_D / 2);
#pragma unroll
      for (int d = 0; d < FA_D / 2; d += 4) *reinterpret_cast<float4*>(p + d) = make_float4(o[d], o[d + 1], o[d + 2], o[d + 3]);
      s_m[stream][row] = m_run, s_l[stream][part][row] = l_run;
    }
    __syncwarp();
    if (!SPLIT && any_lost()) __syncthreads();  // the other warps correct the states
    cluster_sync();
    {
      constexpr int NP = 2 * NS;
      const int np = min(NP, ntiles);  // parts that had tiles
      uint32_t base[NS];  // of the CTAs' shared memory; what is read there lies at the same offsets as here
#pragma unroll
      for (int c = 0; NS > 1 && c < NS; c++) asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(base[c]) : "r"(smem_u32(smem)), "r"(c));
      const uint32_t at_m = smem_u32(&s_m[0][0]) - smem_u32(smem), at_l = smem_u32(&s_l[0][0][0]) - smem_u32(smem);
      // a warp's rows, two at a time; lane = four dims
#pragma unroll 1
      for (int r0 = rank * 16 + warp; r0 < FA_BR && row_lo + r0 < a.rows; r0 += 32 * NS) {
        float4 acc[2];
        float l[2];
#pragma unroll
        for (int q = 0; q < 2; q++) {
          const int r = min(r0 + 16 * NS * q, FA_BR - 1);
          float mv[NP], l0[NP], l1[NP], M = LOWEST;
          float4 v[NP];
#pragma unroll
          for (int p = 0; p < NP; p++) {  // part p: stream p / NS of CTA p mod NS
            if (p >= np) break;
            if constexpr (NS == 1) {
              mv[p] = s_m[p][r], l0[p] = s_l[p][0][r], l1[p] = s_l[p][1][r];
              v[p] = *reinterpret_cast<const float4*>(state + (p * FA_BR + r) * FA_PITCH + 4 * lane);
              continue;
            }
            const uint32_t b = base[p % NS], st = p / NS, sr = st * FA_BR + r;
            asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(mv[p]) : "r"(b + at_m + 4u * sr) : "memory");
            asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(l0[p]) : "r"(b + at_l + 4u * (2u * FA_BR * st + r)) : "memory");
            asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(l1[p]) : "r"(b + at_l + 4u * (2u * FA_BR * st + FA_BR + r)) : "memory");
            asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                         : "=f"(v[p].x), "=f"(v[p].y), "=f"(v[p].z), "=f"(v[p].w)
                         : "r"(b + 4u * (sr * FA_PITCH + 4 * lane))
                         : "memory");
          }
#pragma unroll
          for (int p = 0; p < NP; p++)
            if (p < np) M = fmaxf(M, mv[p]);
          acc[q] = make_float4(0.f, 0.f, 0.f, 0.f), l[q] = 0.f;
#pragma unroll
          for (int p = 0; p < NP; p++) {
            if (p >= np) break;
            const float w = expf(mv[p] - M);  // a part whose keys the row does not see has sum 0 and contributes nothing
            acc[q].x = fmaf(v[p].x, w, acc[q].x), acc[q].y = fmaf(v[p].y, w, acc[q].y);
            acc[q].z = fmaf(v[p].z, w, acc[q].z), acc[q].w = fmaf(v[p].w, w, acc[q].w);
            l[q] = fmaf(l0[p] + l1[p], w, l[q]);
          }
        }
#pragma unroll
        for (int q = 0; q < 2; q++) {
          const int r = r0 + 16 * NS * q;
          if (r >= FA_BR || row_lo + r >= a.rows) break;
          const float i0 = (SPLIT ? PMUL : 1.0f) / l[q];  // pairs: o left the weights' scale with each tile
          *reinterpret_cast<float4*>(a.ctx + (row_lo + r) * a.nh * FA_D + h * FA_D + 4 * lane) =
              make_float4(acc[q].x * i0, acc[q].y * i0, acc[q].z * i0, acc[q].w * i0);
        }
      }
    }
    __syncwarp();
    if constexpr (NS > 1) cluster_sync();  // nobody leaves while its state may still be read
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(FA_ISSUE_REGS));
    if (warp < 18) {
    // ---- the stream's tiles and MMAs. The items K0 V0 K1 V1 .. go round R places; a place is free when the MMAs that read it are
    // done, which the softmax warps' arrivals imply: P(i) written = S(i) done, U(i) read = P V of i done. The warp walks along
    // together, so that addresses stay in uniform registers; one lane asks and issues.
    int put = 0, put_at = 0, get_at = 0;
    unsigned gphase = 0;
    auto ask = [&]() {  // the next item
      if (put < 2 * mine && elect_one()) {
        const bool values = put & 1;
        const int key0 = (first + (put >> 1) * step) * FA_SPLIT_TILE;
        const int y = (int)((values ? a.vrow : a.krow) + kvh * a.cap + key0);
        uint64_t* bar = &item_full[stream][put_at];
        uint8_t* dst = items + put_at * ITEM;
        mbar_expect_tx(bar, ITEM);
        for (int b = 0; b < ITEM / FA_BOX; b++) tma_box_g2s(dst + b * FA_BOX, values ? &vmap : &kmap, 32 * b, y, bar);
      }
      __syncwarp();
      put++;
      if (++put_at == R) put_at = 0;
    };
    if (elect_one()) {
      mbar_expect_tx(q_full + stream, FA_Q_BYTES);
      for (int b = 0; b < 2; b++)
        tma_box_g2s(items + R * ITEM - FA_Q_BYTES + b * (FA_Q_BYTES / 2), &qmap, (int)(h * FA_D) + stream * 64 + 32 * b, (int)row_lo, q_full + stream);
    }
    __syncwarp();
    for (int i = 0; i < R - FA_Q_BYTES / ITEM; i++) ask();
    asm volatile("bar.sync 2, %0;" ::"n"(FA_WORKERS) : "memory");
    for (int i = 0; i < FA_Q_BYTES / ITEM; i++) ask();
    tc_fence_after();
    const uint32_t q_hi = tmem + Q_COL, q_lo = q_hi + 64u;
    const uint32_t id_s = fa_idesc(FA_SPLIT_TILE, BF, false), id_u = fa_idesc(FA_D, BF, true);
    const uint64_t k_desc0 = umma_desc(smem_u32(items)), v_desc0 = fa_desc_mn(smem_u32(items));
    // the second stream starts half a tile later, so that the one's MMAs run under the other's softmax (in step, they would
    // wait for the same units). The barrier has this one phase: a warp that comes late finds it done whatever has gone on since.
    bool ok = !(stream && mine > 2) || mbar_wait_bounded(&started, 0, TG_SPINS, &s_abort);
#pragma unroll 1
    for (int i = 0; i < mine && ok; i++) {
      ok = mbar_wait_bounded(&item_full[stream][get_at], gphase, TG_SPINS, &s_abort) &&
           (i == 0 || mbar_wait_bounded(u_free + stream, (FOLDS * i - 1) & 1, TG_SPINS, &s_abort));
      if (!ok) break;
      tc_fence_after();
      const uint64_t k_hi = k_desc0 + (uint64_t)(get_at * (ITEM >> 4)), k_lo = k_hi + (2 * FA_BOX >> 4);
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < 8; k++) {  // sixteen dims at a time: boxes of 64 dims, 32 bytes in a row
          const uint64_t at = (uint64_t)((k >> 2) * (FA_BOX >> 4) + 2 * (k & 3));
          umma_f16_ts(u_col, q_lo + 8u * k, k_hi + at, id_s, k ? 1u : 0u);
          if constexpr (SPLIT) umma_f16_ts(u_col, q_hi + 8u * k, k_lo + at, id_s, 1u);
        }
        // the large terms in two chains of four, one of them on top of the small ones
#pragma unroll
        for (int k = 0; k < 8; k++)
          umma_f16_ts(k < 4 ? s_col : u_col, q_hi + 8u * k, k_hi + (uint64_t)((k >> 2) * (FA_BOX >> 4) + 2 * (k & 3)), id_s, k ? 1u : 0u);
        umma_commit(s_full + stream);
        if (!stream && i == 0) umma_commit(&started);
      }
      __syncwarp();
      if (i) ask();  // in place of the values of tile i - 1
      if (++get_at == R) get_at = 0, gphase ^= 1u;
      ok = mbar_wait_bounded(&item_full[stream][get_at], gphase, TG_SPINS, &s_abort) &&
           mbar_wait_bounded(p_full + stream, i & 1, TG_SPINS, &s_abort);
      if (!ok) break;
      tc_fence_after();
      const uint64_t v_hi = v_desc0 + (uint64_t)(get_at * (ITEM >> 4)), v_lo = v_hi + (2 * FA_BOX >> 4);
#pragma unroll
      for (int q = 0; q < FOLDS; q++) {
        if (q && ok) ok = mbar_wait_bounded(u_free + stream, (FOLDS * i + q - 1) & 1, TG_SPINS, &s_abort);
        if (!ok) break;
        tc_fence_after();
        if (elect_one()) {
          constexpr int KS = 4 / FOLDS;  // sixteen keys at a time; the small terms first
#pragma unroll
          for (int k = q * KS; k < (q + 1) * KS; k++) {
            const uint32_t p_hi = s_col + 16u * k, p_lo = p_hi + 8u;
            const uint64_t at = (uint64_t)(k * (2048 >> 4));
            umma_f16_ts(u_col, p_lo, v_hi + at, id_u, k > q * KS ? 1u : 0u);
            if constexpr (SPLIT) umma_f16_ts(u_col, p_hi, v_lo + at, id_u, 1u);
          }
#pragma unroll
          for (int k = q * KS; k < (q + 1) * KS; k++) umma_f16_ts(u_col, s_col + 16u * k, v_hi + (uint64_t)(k * (2048 >> 4)), id_u, 1u);
          umma_commit(u_full + stream);
        }
        __syncwarp();
      }
      ask();  // in place of the keys
      if (++get_at == R) get_at = 0, gphase ^= 1u;
    }
    if (!ok && !s_abort) s_abort = 4;
    __syncwarp();
    } else if constexpr (!SPLIT) {
      // ---- 2-byte caches: looks through the values of tiles whose keys not all rows see, while the scores are made. Weight 0 times an
      // entry that is not finite would reach the rows that do not see its key: the entry becomes a zero and the key is marked.
      // (Keys past the last row may hold anything; no row sees them.)
      int item = 1;
      unsigned iphase = 0;
#pragma unroll 1
      for (int i = 0; i < mine; i++) {
        // (this warp's arrival belongs to this tile's phase)
        if (i && !mbar_wait_bounded(p_full + stream, (i - 1) & 1, TG_SPINS, &s_abort) && !s_abort) s_abort = 6;
        const int at = first + i * step - diag0;
        if (at >= 0) {
          if (!mbar_wait_bounded(&item_full[stream][item], iphase, TG_SPINS, &s_abort) && !s_abort) s_abort = 2;
          uint4* const p = reinterpret_cast<uint4*>(items + item * ITEM) + lane;
          uint32_t acc[4] = {0, 0, 0, 0};  // sums of entries times zero
#pragma unroll 4
          for (int j = 0; j < ITEM / 512; j++) {
            const uint4 v = p[32 * j];
            acc[0] = fa_fma0<BF>(v.x, acc[0]), acc[1] = fa_fma0<BF>(v.y, acc[1]), acc[2] = fa_fma0<BF>(v.z, acc[2]), acc[3] = fa_fma0<BF>(v.w, acc[3]);
          }
          if (fa_not_finite2<BF>(acc[0]) | fa_not_finite2<BF>(acc[1]) | fa_not_finite2<BF>(acc[2]) | fa_not_finite2<BF>(acc[3])) {
#pragma unroll 1
            for (int j = 0; j < ITEM / 128; j++) {  // four bytes of key (4 (j / 4) + lane / 8) mod 64
              uint32_t* const w = reinterpret_cast<uint32_t*>(p + 32 * (j >> 2)) + (j & 3);
              const uint32_t m = fa_not_finite2<BF>(*w);
              if (!m) continue;
              *w &= ~((m >> 15) * 0xffffu);
              const int key = (4 * (j >> 2) + (lane >> 3)) & (FA_SPLIT_TILE - 1);
              atomicOr(s_lost + 2 * at + (key >> 5), 1u << (key & 31));
            }
          }
          fence_async_smem();
        }
        item += 2;
        if (item >= R) item -= R, iphase ^= 1u;
        __syncwarp();
        if (lane == 0) mbar_arrive(p_full + stream);
      }
    }
    // (the softmax warps' ends are theirs alone: these warps have given their registers away)
    drained();
    if (!SPLIT && any_lost()) {
      // zeros took the places of what is not finite: a thread adds it to its row's states, for the keys that the row sees. (Here, because the same in
      // the softmax warps costs their loop registers: 2 to 3 % of a call.)
      __syncthreads();
      const int r = tid - 512;
      for (int64_t t = rank; t < ntiles && row_lo + r < a.rows; t += NS)
        for (int q = 0; q < 2 && t >= diag0; q++)
          for (unsigned m = s_lost[2 * (t - diag0) + q]; m; m &= m - 1) {
            const int64_t key = t * FA_SPLIT_TILE + 32 * q + __ffs(m) - 1;
            if (key > a.base_pos + row_lo + r) break;
            const uint32_t* const w = reinterpret_cast<const uint32_t*>(a.vals + (kvh * a.cap + key) * FA_D);
            float* const p = reinterpret_cast<float*>(smem) + ((t / NS & 1) * FA_BR + r) * FA_PITCH;
#pragma unroll 1
            for (int d = 0; d < FA_D; d += 2) fa_add_not_finite2<BF>(p + d, __ldcg(w + d / 2));
          }
    }
    __syncwarp();  // (the rows' loops differ in length)
    cluster_sync();
    if constexpr (NS > 1) cluster_sync();
  }
  tc_fence_after();
  if (warp == 16) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  if (tid == 0 && s_abort) report_wait_expired(a.error, DEV_ERR_GEMM_PIPE);
}

template <int KV, int NS>
int fa_launch(const FaArgs& f, const CUtensorMap& qmap, const CUtensorMap& kmap, const CUtensorMap& vmap, cudaStream_t s) {
  auto kernel = attention_prefill_kernel<KV, NS>;
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), FA_SMEM)) return 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(f.nh * NS), (unsigned)((f.rows + FA_BR - 1) / FA_BR)), cfg.blockDim = dim3(FA_THREADS);
  cfg.dynamicSmemBytes = FA_SMEM, cfg.stream = s;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (pdl_enabled()) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (NS > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = NS, attr[n].val.clusterDim.y = 1, attr[n].val.clusterDim.z = 1;
    n++;
  }
  cfg.attrs = attr, cfg.numAttrs = n;
  DYN_CUDA(cudaLaunchKernelEx(&cfg, kernel, f, qmap, kmap, vmap));
  return 0;
}

}  // namespace

// Scratch of the f16 pairs of an f32 cache: the pairs, the inverse tile scales, a bit per key.
size_t attention_prefill_scratch_bytes(const AttnArgs& a) {
  if (a.kv_type != E_F32) return 0;
  return (size_t)(2 * a.nkv * a.cap) * (2 * FA_D) * 2 + (size_t)(2 * a.nkv * (a.cap / FA_SPLIT_TILE)) * 4 + (size_t)(a.nkv * (a.cap / 32)) * 4;
}

// Tensor-core attention for `a.rows` query rows of sequence `seq` at positions base_pos + row.
// *handled = false when the shape does not qualify (head dim != 128, few rows).
int launch_attention_prefill(const AttnArgs& a, int64_t base_pos, int64_t seq, cudaStream_t s, bool* handled) {
  *handled = false;
  if (a.d != FA_D || a.rows < 32 || (a.kv_type != E_BF16 && a.kv_type != E_F16 && a.kv_type != E_F32)) return 0;
  if (a.nkv <= 0 || a.nh % a.nkv || a.cap % FA_SPLIT_TILE) return 0;
  if (((reinterpret_cast<uintptr_t>(a.q) | reinterpret_cast<uintptr_t>(a.ctx) | reinterpret_cast<uintptr_t>(a.kcache) |
        reinterpret_cast<uintptr_t>(a.vcache)) & 15) || a.ldq % 4 || 2 * a.nkv * a.cap > 0x7fffffff)
    return 0;
  FaArgs f{};
  f.q = a.q, f.ctx = a.ctx, f.error = device_error_word();
  if (!f.error) return 1;
  f.rows = a.rows, f.nh = a.nh, f.nkv = a.nkv, f.cap = a.cap, f.base_pos = base_pos;
  f.ldq = a.ldq ? a.ldq : a.nh * FA_D;
  // The keys go to as many CTAs as the SMs hold besides one another, while there is a tile for each of half of them
  const int64_t pairs = a.nh * ((a.rows + FA_BR - 1) / FA_BR), tiles = (base_pos + a.rows + FA_SPLIT_TILE - 1) / FA_SPLIT_TILE;
  int splits = 1;
  while (splits < 4 && 2 * splits * pairs <= sm_count() && splits < tiles) splits *= 2;
  struct Pooled {  // given back however the call ends
    void* ptr = nullptr;
    cudaStream_t s;
    cudaError_t give_back() {
      void* const p = ptr;
      ptr = nullptr;
      return p ? cudaFreeAsync(p, s) : cudaSuccess;
    }
    ~Pooled() { give_back(); }
  } pooled{nullptr, s};
  CUtensorMap qmap, kmap, vmap;
  if (make_row_box_map(reinterpret_cast<const uint8_t*>(a.q), (size_t)f.ldq * 4, a.rows, 32, FA_BR, &qmap, true)) return 1;
  if (a.kv_type == E_F32) {
    const size_t bytes = attention_prefill_scratch_bytes(a);
    void* ws = a.pair_ws && a.pair_ws_bytes >= bytes ? a.pair_ws : nullptr;
    if (!ws) {
      if (keep_scratch_pool_cached()) return 1;
      DYN_CUDA(cudaMallocAsync(&pooled.ptr, bytes, s));
      ws = pooled.ptr;
    }
    __half* const out = reinterpret_cast<__half*>(ws);
    const size_t plane = (size_t)a.nkv * a.cap * 2 * FA_D;
    float* const inv = reinterpret_cast<float*>(out + 2 * plane);
    unsigned* const lost = reinterpret_cast<unsigned*>(inv + 2 * a.nkv * (a.cap / FA_SPLIT_TILE));
    const int64_t nkeys = base_pos + a.rows;
    DYN_CUDA(launch_pdl(fa_split_kernel, dim3((unsigned)((nkeys + FA_SPLIT_TILE - 1) / FA_SPLIT_TILE), (unsigned)a.nkv, 2), dim3(256), 0, s,
                        reinterpret_cast<const float*>(a.kcache), reinterpret_cast<const float*>(a.vcache), a.nkv, a.cap, seq, nkeys, out, inv,
                        lost));
    count_launch();
    f.kinv = inv, f.vinv = inv + a.nkv * (a.cap / FA_SPLIT_TILE), f.vlost = lost;
    if (make_row_box_map(reinterpret_cast<const uint8_t*>(out), 4 * FA_D, 2 * a.nkv * a.cap, 32, FA_SPLIT_TILE, &kmap, true)) return 1;
    vmap = kmap;
    f.krow = 0, f.vrow = a.nkv * a.cap;
  } else {
    const int64_t at = seq * a.nkv * a.cap;  // row of the sequence's first plane
    f.vals = reinterpret_cast<const uint16_t*>(a.vcache) + at * FA_D;
    if (make_row_box_map(reinterpret_cast<const uint8_t*>(a.kcache) + at * (2 * FA_D), 2 * FA_D, a.nkv * a.cap, 32, FA_SPLIT_TILE, &kmap, true) ||
        make_row_box_map(reinterpret_cast<const uint8_t*>(a.vcache) + at * (2 * FA_D), 2 * FA_D, a.nkv * a.cap, 32, FA_SPLIT_TILE, &vmap, true))
      return 1;
  }
  auto launch = [&](auto n1, auto n2, auto n4) { return (splits == 1 ? n1 : splits == 2 ? n2 : n4)(f, qmap, kmap, vmap, s); };
  const int rc = a.kv_type == E_F32    ? launch(fa_launch<E_F32, 1>, fa_launch<E_F32, 2>, fa_launch<E_F32, 4>)
                 : a.kv_type == E_BF16 ? launch(fa_launch<E_BF16, 1>, fa_launch<E_BF16, 2>, fa_launch<E_BF16, 4>)
                                       : launch(fa_launch<E_F16, 1>, fa_launch<E_F16, 2>, fa_launch<E_F16, 4>);
  const cudaError_t fe = pooled.give_back();
  if (rc) return 1;
  if (fe != cudaSuccess) return cuda_fail(fe, "cudaFreeAsync", __FILE__, __LINE__);
  count_launch();
  DYN_CUDA(cudaGetLastError());
  *handled = true;
  return 0;
}

}  // namespace dyn
