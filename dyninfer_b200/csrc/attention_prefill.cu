// Causal GQA attention for prefill chunks: many query rows of ONE sequence at consecutive
// positions against an f32, bf16 or f16 KV cache, on the tensor cores.
//
// Same mathematics as the per-row kernel (kernels.rs:310-458: s = (q.k) * 1/sqrt(d), keys beyond the
// row's position masked, online max / sum merge, out / sum at the end), restructured the usual
// flash-attention way: one CTA = one query head x 64 consecutive rows. The 64-key blocks stream through
// shared memory with cp.async, the next group of blocks in flight while the current one is used.
// Two shapes of CTA: when the grid is no larger than the GPU (a 512-row chunk of a 16-head model: 128
// CTAs), eight warps -- warp w takes the 16 rows of group w mod 4 and, of every PAIR of blocks, block
// w / 4, so two blocks are worked on at once and the two halves' running (max, sum, out) are merged at
// the end (four K + V tiles resident, one CTA per SM); for larger grids four warps and one block at a
// time (two tiles resident, two CTAs per SM). S = Q K^T and O += P V run on mma.sync.m16n8k16 with f32
// accumulators. The cache entries are used
// in their stored type (exact); the f32 operands Q and P enter as hi + lo pairs of that type
// (two mma per tile), so the products carry ~16 significant bits of Q / P and the result stays
// within ~1e-4 of the f32 evaluation.
//
// f32 caches: a first pass turns the sequence's keys and values into (hi, lo) pairs of f16, every 64-key
// tile of a head scaled by a power of two of its own (no overflow, nothing lost to subnormals), so a pair
// holds the entry to 2^-24 of its magnitude; the query rows are scaled and split the same way. The
// products take three mma per tile (hi hi, lo hi, hi lo; what is dropped is 2^-24 of a term). The tile
// scales are exact: the keys' multiply the scores, the values' a step's share of the output. Tiles are
// twice as wide, so a step takes 32 keys. One-row-per-block evaluation of the same chunk (what f32 caches
// used before) read every key once per query row: 0.6B, 2048-token prompt 102 -> 25 ms.
// An mma truncates where it adds to its accumulator (about 1.5e-8 of the sum each time, always toward
// zero). With f16 pairs the scores are therefore added up in chains of four, the products with a lo term
// apart, and the P V of a step starts from zero and joins the running output by a rounded fma. Error against
// 64 bits, 256 rows at 7936, mma adding up everything / now / per-row kernel in f32: normal values 1.5e-5 /
// 3.9e-7 / 8.9e-7, values of one sign 3.2e-5 / 2.0e-7 / 4.7e-7. Cost: 512 rows of 16 heads at 1536
// 125.5 -> 129.8 us.
#include <algorithm>

#include "common.cuh"

namespace dyn {

namespace {

constexpr int FA_D = 128;      // head dim handled by this kernel
constexpr int FA_BR = 64;      // query rows per CTA
constexpr int FA_PITCH = FA_D + 8;  // elements per shared-memory row (272 bytes: conflict-free fragment loads)
constexpr int FA_SPLIT_TILE = 64;   // keys per scale of the (hi, lo) form
constexpr int fa_keys(int kv) { return kv == E_F32 ? 32 : 64; }       // keys per step
constexpr int fa_planes(int kv) { return kv == E_F32 ? 2 : 1; }       // (hi, lo) or the entries themselves
constexpr int fa_tile(int kv) { return fa_keys(kv) * FA_PITCH * fa_planes(kv); }  // elements of one K (or V) tile
constexpr int fa_threads(int halves) { return 128 * halves; }
constexpr int fa_smem_bytes(int kv, int halves) { return 2 * halves * 2 * fa_tile(kv) * 2; }  // buffers x blocks of a group x (K, V) x 2 bytes

__device__ __forceinline__ void fa_cp16(void* dst, const void* src, bool live) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const int n = live ? 16 : 0;  // 0 source bytes: the 16 destination bytes are zero-filled
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}

template <int KV>
struct Mma;
template <>
struct Mma<E_BF16> {
  using T = __nv_bfloat16;
  __device__ static __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  }
  // (hi, lo) packed pairs of two f32 values
  __device__ static __forceinline__ void split2(float x, float y, uint32_t* hi, uint32_t* lo) {
    const __nv_bfloat16 hx = __float2bfloat16_rn(x), hy = __float2bfloat16_rn(y);
    const __nv_bfloat16 lx = __float2bfloat16_rn(x - __bfloat162float(hx));
    const __nv_bfloat16 ly = __float2bfloat16_rn(y - __bfloat162float(hy));
    *hi = (uint32_t)__bfloat16_as_ushort(hx) | ((uint32_t)__bfloat16_as_ushort(hy) << 16);
    *lo = (uint32_t)__bfloat16_as_ushort(lx) | ((uint32_t)__bfloat16_as_ushort(ly) << 16);
  }
};
template <>
struct Mma<E_F16> {
  using T = __half;
  __device__ static __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  }
  __device__ static __forceinline__ void split2(float x, float y, uint32_t* hi, uint32_t* lo) {
    const __half hx = __float2half_rn(x), hy = __float2half_rn(y);
    const __half lx = __float2half_rn(x - __half2float(hx)), ly = __float2half_rn(y - __half2float(hy));
    *hi = (uint32_t)__half_as_ushort(hx) | ((uint32_t)__half_as_ushort(hy) << 16);
    *lo = (uint32_t)__half_as_ushort(lx) | ((uint32_t)__half_as_ushort(ly) << 16);
  }
};

template <>
struct Mma<E_F32> : Mma<E_F16> {};  // operands are f16 pairs

// Power of two that puts `mx` into [2^12, 2^13), and its inverse; magnitudes below 2^-41 share one scale.
__device__ __forceinline__ void fa_pow2_scale(float mx, float* sc, float* inv) {
  int e = 0;
  if (mx > 0.f && mx <= 3.40282347e38f) frexpf(mx, &e);
  e = max(e, -40);
  *sc = ldexpf(1.0f, 13 - e);
  *inv = ldexpf(1.0f, e - 13);
}

__device__ __forceinline__ void fa_ldsm4(uint32_t& a, uint32_t& b, uint32_t& c, uint32_t& d, uint32_t at) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(a), "=r"(b), "=r"(c), "=r"(d) : "r"(at));
}
__device__ __forceinline__ void fa_ldsm4t(uint32_t& a, uint32_t& b, uint32_t& c, uint32_t& d, uint32_t at) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(a), "=r"(b), "=r"(c), "=r"(d) : "r"(at));
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
fa_split_kernel(const float* __restrict__ kc, const float* __restrict__ vc, int64_t nkv, int64_t cap, int64_t seq,
                int64_t nkeys, __half* __restrict__ out, float* __restrict__ inv, unsigned* __restrict__ lost) {
  __shared__ float red[8];
  __shared__ unsigned s_lost[2];
  const int64_t tile = blockIdx.x, kvh = blockIdx.y, plane = blockIdx.z;
  const float* src = (plane ? vc : kc) + ((seq * nkv + kvh) * cap + tile * FA_SPLIT_TILE) * FA_D;
  const int left = (int)min((int64_t)FA_SPLIT_TILE, nkeys - tile * FA_SPLIT_TILE) * (FA_D / 4);  // float4s
  float4 v[8];
  float mx = 0.f;
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const int i = threadIdx.x + 256 * k;
    v[k] = i < left ? reinterpret_cast<const float4*>(src)[i] : make_float4(0.f, 0.f, 0.f, 0.f);
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
    Mma<E_F16>::split2(v[k].x * sc, v[k].y * sc, &hi.x, &lo.x);
    Mma<E_F16>::split2(v[k].z * sc, v[k].w * sc, &hi.y, &lo.y);
    __half* row = dst + (i / (FA_D / 4)) * (2 * FA_D) + (i % (FA_D / 4)) * 4;
    *reinterpret_cast<uint2*>(row) = hi;
    *reinterpret_cast<uint2*>(row + FA_D) = lo;
  }
}

struct FaArgs {
  const float* q;     // [rows, nh, d]
  const void* kcache; // plane of (seq, kv head): [cap, d]; f32 caches: the f16 pairs, [kv head][cap][hi d | lo d]
  const void* vcache;
  const float* kinv;  // f32 caches: inverse tile scales [kv head][cap / 64]
  const float* vinv;
  const unsigned* vlost;  // f32 caches: a bit per key whose values are not all finite [kv head][cap / 32]
  float* ctx;         // [rows, nh * d]
  int64_t rows, nh, nkv, cap, base_pos, seq;
  int64_t ldq;        // floats between consecutive rows of q
};

template <int KV, int HALVES>
__global__ void __launch_bounds__(fa_threads(HALVES)) attention_prefill_kernel(const FaArgs a) {
  constexpr int FA_THREADS = fa_threads(HALVES);
  constexpr bool SPLIT = KV == E_F32;
  constexpr bool SCALED = KV != E_BF16;                // f16 terms: the query rows and the weights need scales
  constexpr float PMUL = SCALED ? 16384.0f : 1.0f;     // the weights' (the sum carries it too)
  constexpr int FA_BC = fa_keys(KV), FA_TILE = fa_tile(KV), NP = fa_planes(KV), NT = FA_BC / 8;
  constexpr int LO = FA_BC * FA_PITCH;  // the lo half of a tile
  using M = Mma<KV>;
  using T = typename M::T;
  extern __shared__ __align__(16) uint8_t fa_smem[];
  T* const tiles = reinterpret_cast<T*>(fa_smem);  // [buffer][block of the pair][K, V][hi, lo][FA_BC][FA_PITCH]
  const int tid = threadIdx.x, lane = tid & 31, warp8 = tid >> 5;
  const int warp = warp8 & 3, half = warp8 >> 2;   // row group; which block of a group
  const int g = lane >> 2, t = lane & 3;
  const int64_t h = blockIdx.x, rb = gridDim.y - 1 - blockIdx.y;  // the longest row blocks start first
  const int64_t kvh = h / (a.nh / a.nkv);
  const int64_t plane = (SPLIT ? kvh : a.seq * a.nkv + kvh) * a.cap * (FA_D * NP);
  const T* kplane = reinterpret_cast<const T*>(a.kcache) + plane;
  const T* vplane = reinterpret_cast<const T*>(a.vcache) + plane;
  const float* kinv = SPLIT ? a.kinv + kvh * (a.cap / FA_SPLIT_TILE) : nullptr;
  const float* vinv = SPLIT ? a.vinv + kvh * (a.cap / FA_SPLIT_TILE) : nullptr;
  const unsigned* vlost = SPLIT ? a.vlost + kvh * (a.cap / 32) : nullptr;
  const int64_t row_lo = rb * FA_BR + warp * 16;   // this warp's first query row
  const int64_t r0 = row_lo + g, r1 = r0 + 8;      // the lane's two rows
  const int64_t r0c = r0 < a.rows ? r0 : a.rows - 1, r1c = r1 < a.rows ? r1 : a.rows - 1;
  const int64_t pos0 = a.base_pos + r0, pos1 = a.base_pos + r1;
  const float scale = 1.0f / sqrtf((float)FA_D);

  // Q fragments (hi, lo) for the 8 k-steps over the head dim
  uint32_t qh[8][4], ql[8][4];
  float scale0 = scale, scale1 = scale;  // per query row: 1 / sqrt(d), with f16 pairs times the row's inverse scale
  {
    const float* q0 = a.q + r0c * a.ldq + h * FA_D;
    const float* q1 = a.q + r1c * a.ldq + h * FA_D;
    float s0 = 1.f, s1 = 1.f;
    if constexpr (SCALED) {
      float x0 = 0.f, x1 = 0.f;
#pragma unroll
      for (int kk = 0; kk < 16; kk++) {
        const float2 a0 = *reinterpret_cast<const float2*>(q0 + 8 * kk + 2 * t);
        const float2 a1 = *reinterpret_cast<const float2*>(q1 + 8 * kk + 2 * t);
        x0 = fmaxf(x0, fmaxf(fabsf(a0.x), fabsf(a0.y)));
        x1 = fmaxf(x1, fmaxf(fabsf(a1.x), fabsf(a1.y)));
      }
      x0 = fmaxf(x0, __shfl_xor_sync(0xffffffffu, x0, 1));
      x0 = fmaxf(x0, __shfl_xor_sync(0xffffffffu, x0, 2));
      x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, 1));
      x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, 2));
      float i0, i1;
      fa_pow2_scale(x0, &s0, &i0);
      fa_pow2_scale(x1, &s1, &i1);
      scale0 *= i0, scale1 *= i1;
    }
#pragma unroll
    for (int kk = 0; kk < 8; kk++) {
      const float2 a0 = *reinterpret_cast<const float2*>(q0 + 16 * kk + 2 * t);
      const float2 a1 = *reinterpret_cast<const float2*>(q1 + 16 * kk + 2 * t);
      const float2 a2 = *reinterpret_cast<const float2*>(q0 + 16 * kk + 8 + 2 * t);
      const float2 a3 = *reinterpret_cast<const float2*>(q1 + 16 * kk + 8 + 2 * t);
      M::split2(a0.x * s0, a0.y * s0, &qh[kk][0], &ql[kk][0]);
      M::split2(a1.x * s1, a1.y * s1, &qh[kk][1], &ql[kk][1]);
      M::split2(a2.x * s0, a2.y * s0, &qh[kk][2], &ql[kk][2]);
      M::split2(a3.x * s1, a3.y * s1, &qh[kk][3], &ql[kk][3]);
    }
  }
  float o[16][4];
#pragma unroll
  for (int dt = 0; dt < 16; dt++) o[dt][0] = o[dt][1] = o[dt][2] = o[dt][3] = 0.f;
  float m0 = -3.40282347e38f, m1 = -3.40282347e38f, l0 = 0.f, l1 = 0.f;

  // keys 0 .. last position of the CTA's rows
  int64_t cta_last = a.base_pos + rb * FA_BR + FA_BR - 1;
  if (cta_last > a.base_pos + a.rows - 1) cta_last = a.base_pos + a.rows - 1;
  const int64_t warp_last = a.base_pos + (row_lo + 15 < a.rows ? row_lo + 15 : a.rows - 1);
  const int64_t nkb = cta_last / FA_BC + 1, npairs = (nkb + HALVES - 1) / HALVES;
  // HALVES blocks x (K, V) x keys of a step x 16 (pairs: 32) pieces of 16 bytes per group, coalesced; rows past the last written
  // position may hold anything: they are masked, but 0 * NaN must not happen, so they arrive as zeros
  auto load_pair = [&](int64_t pr) {
    T* dst = tiles + (pr & 1) * 2 * HALVES * FA_TILE;
    constexpr int PC = NP * FA_D / 8;  // pieces per key
    for (int i = tid; i < HALVES * FA_BC * PC; i += FA_THREADS) {
      const int blk = i / (FA_BC * PC), key = (i / PC) % FA_BC, c = i % PC;
      const int64_t gk = (HALVES * pr + blk) * FA_BC + key;  // < cap for every written key
      const bool written = gk <= cta_last;
      const int64_t src = (written ? gk : 0) * (FA_D * NP) + c * 8;
      const int at = (c / (FA_D / 8)) * LO + key * FA_PITCH + (c % (FA_D / 8)) * 8;
      fa_cp16(dst + (blk * 2) * FA_TILE + at, kplane + src, written);
      fa_cp16(dst + (blk * 2 + 1) * FA_TILE + at, vplane + src, written);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  load_pair(0);
  for (int64_t pr = 0; pr < npairs; pr++) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();  // pair pr has arrived for everyone, and nobody still reads the buffer the next pair goes to
    if (pr + 1 < npairs) load_pair(pr + 1);
    const int64_t kb = HALVES * pr + half;
    if (kb >= nkb) continue;
    const T(*ks)[FA_PITCH] = reinterpret_cast<const T(*)[FA_PITCH]>(tiles + ((pr & 1) * 2 * HALVES + half * 2) * FA_TILE);
    const T(*vs)[FA_PITCH] = reinterpret_cast<const T(*)[FA_PITCH]>(tiles + ((pr & 1) * 2 * HALVES + half * 2 + 1) * FA_TILE);
    if (kb * FA_BC > warp_last) continue;  // every key of the block lies after this warp's rows
    float ks0 = scale0, ks1 = scale1, vi = 1.0f;
    unsigned lost = 0;  // keys of the step whose values are not finite
    if constexpr (SPLIT) {
      const int64_t tile = kb * FA_BC / FA_SPLIT_TILE;
      const float ki = __ldg(kinv + tile);
      vi = __ldg(vinv + tile) * (1.0f / PMUL);
      lost = __ldg(vlost + 2 * tile + (kb & 1));
      ks0 *= ki, ks1 *= ki;
    }
    // ---- S = Q K^T for 16 rows x the keys of the step. All key groups of a k-step in turn, so that consecutive MMAs do not
    // wait for one another; one ldmatrix brings the fragments of two groups
    float s[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; nt++) s[nt][0] = s[nt][1] = s[nt][2] = s[nt][3] = 0.f;
    const uint32_t ka = (uint32_t)__cvta_generic_to_shared(&ks[(lane & 7) + 8 * (lane >> 4)][8 * ((lane >> 3) & 1)]);
    if constexpr (SPLIT) {
#pragma unroll
      for (int n0 = 0; n0 < NT; n0 += 2) {
        float x[2][2][4], lo[2][2][4];  // group, chain
#pragma unroll
        for (int n = 0; n < 2; n++)
#pragma unroll
          for (int h = 0; h < 2; h++)
#pragma unroll
            for (int e = 0; e < 4; e++) x[n][h][e] = lo[n][h][e] = 0.f;
#pragma unroll
        for (int kk = 0; kk < 8; kk++) {
          uint32_t b[2][2], c[2][2];
          const uint32_t at = ka + (uint32_t)((n0 * 8 * FA_PITCH + 16 * kk) * 2);
          fa_ldsm4(b[0][0], b[0][1], b[1][0], b[1][1], at);
          fa_ldsm4(c[0][0], c[0][1], c[1][0], c[1][1], at + LO * 2);
#pragma unroll
          for (int n = 0; n < 2; n++) M::mma(x[n][kk & 1], qh[kk], b[n][0], b[n][1]);
#pragma unroll
          for (int n = 0; n < 2; n++) M::mma(lo[n][0], ql[kk], b[n][0], b[n][1]);
#pragma unroll
          for (int n = 0; n < 2; n++) M::mma(lo[n][1], qh[kk], c[n][0], c[n][1]);
        }
#pragma unroll
        for (int n = 0; n < 2; n++)
#pragma unroll
          for (int e = 0; e < 4; e++) s[n0 + n][e] = (x[n][0][e] + x[n][1][e]) + (lo[n][0][e] + lo[n][1][e]);
      }
    } else {
      constexpr int GR = NT < 4 ? NT : 4;  // groups at a time
#pragma unroll
      for (int n0 = 0; n0 < NT; n0 += GR)
#pragma unroll
        for (int kk = 0; kk < 8; kk++) {
          uint32_t b[GR][2];
#pragma unroll
          for (int n = 0; n < GR; n += 2)
            fa_ldsm4(b[n][0], b[n][1], b[n + 1][0], b[n + 1][1], ka + (uint32_t)(((n0 + n) * 8 * FA_PITCH + 16 * kk) * 2));
#pragma unroll
          for (int n = 0; n < GR; n++) M::mma(s[n0 + n], qh[kk], b[n][0], b[n][1]);
#pragma unroll
          for (int n = 0; n < GR; n++) M::mma(s[n0 + n], ql[kk], b[n][0], b[n][1]);
        }
    }
    // ---- scale, causal mask (blocks that reach past the warp's first row), running maximum
    float bm0 = -3.40282347e38f, bm1 = -3.40282347e38f;
    const bool masked = kb * FA_BC + FA_BC - 1 > a.base_pos + row_lo;
    const int lim0 = (int)(pos0 - kb * FA_BC) - 2 * t, lim1 = (int)(pos1 - kb * FA_BC) - 2 * t;
#pragma unroll
    for (int nt = 0; nt < NT; nt++) {
#pragma unroll
      for (int e = 0; e < 2; e++) {
        s[nt][e] = __fmul_rn(s[nt][e], ks0), s[nt][2 + e] = __fmul_rn(s[nt][2 + e], ks1);  // rounded on its own, not inside the difference below
        if (masked) {
          if (nt * 8 + e > lim0) s[nt][e] = -3.40282347e38f;
          if (nt * 8 + e > lim1) s[nt][2 + e] = -3.40282347e38f;
        }
        bm0 = fmaxf(bm0, s[nt][e]);
        bm1 = fmaxf(bm1, s[nt][2 + e]);
      }
    }
    bm0 = fmaxf(bm0, __shfl_xor_sync(0xffffffffu, bm0, 1));
    bm0 = fmaxf(bm0, __shfl_xor_sync(0xffffffffu, bm0, 2));
    bm1 = fmaxf(bm1, __shfl_xor_sync(0xffffffffu, bm1, 1));
    bm1 = fmaxf(bm1, __shfl_xor_sync(0xffffffffu, bm1, 2));
    const float mn0 = fmaxf(m0, bm0), mn1 = fmaxf(m1, bm1);
    const float f0 = expf(m0 - mn0), f1 = expf(m1 - mn1);
    m0 = mn0, m1 = mn1;
    l0 *= f0, l1 *= f1;
    if (!SPLIT && __any_sync(0xffffffffu, f0 != 1.0f || f1 != 1.0f)) {
#pragma unroll
      for (int dt = 0; dt < 16; dt++) {
        o[dt][0] *= f0, o[dt][1] *= f0;
        o[dt][2] *= f1, o[dt][3] *= f1;
      }
    }
    // ---- P = exp(S - m) (masked keys give exactly 0 once a real key has been seen), hi/lo fragments
    uint32_t ph[NT / 2][4], pl[NT / 2][4];
#pragma unroll
    for (int nt = 0; nt < NT; nt++) {
      float p[4];
#pragma unroll
      for (int e = 0; e < 2; e++) {
        p[e] = expf(s[nt][e] - m0) * PMUL;
        p[2 + e] = expf(s[nt][2 + e] - m1) * PMUL;
        if (masked) {
          if (nt * 8 + e > lim0) p[e] = 0.f;
          if (nt * 8 + e > lim1) p[2 + e] = 0.f;
        }
      }
      l0 += p[0] + p[1];
      l1 += p[2] + p[3];
      // accumulator tiles 2j, 2j+1 are the A fragment of k-step j of P V
      const int j = nt >> 1, half = nt & 1;
      M::split2(p[0], p[1], &ph[j][2 * half], &pl[j][2 * half]);          // row g
      M::split2(p[2], p[3], &ph[j][2 * half + 1], &pl[j][2 * half + 1]);  // row g + 8
    }
    // ---- O += P V: B fragments come transposed out of the [key][dim] tile, four groups of eight dims at a time
    const uint32_t va = (uint32_t)__cvta_generic_to_shared(&vs[lane & 15][8 * (lane >> 4)]);
#pragma unroll
    for (int d0 = 0; d0 < 16; d0 += 4) {
      float u[4][4];
#pragma unroll
      for (int j = 0; j < NT / 2; j++) {
        uint32_t b[4][2], c[4][2];
#pragma unroll
        for (int i = 0; i < 4; i += 2) {
          const uint32_t at = va + (uint32_t)((16 * j * FA_PITCH + (d0 + i) * 8) * 2);
          fa_ldsm4t(b[i][0], b[i][1], b[i + 1][0], b[i + 1][1], at);
          if constexpr (SPLIT) fa_ldsm4t(c[i][0], c[i][1], c[i + 1][0], c[i + 1][1], at + LO * 2);
        }
        if constexpr (SPLIT) {
          if (j == 0) {
#pragma unroll
            for (int i = 0; i < 4; i++) u[i][0] = u[i][1] = u[i][2] = u[i][3] = 0.f;
          }
#pragma unroll
          for (int i = 0; i < 4; i++) M::mma(u[i], ph[j], c[i][0], c[i][1]);
#pragma unroll
          for (int i = 0; i < 4; i++) M::mma(u[i], pl[j], b[i][0], b[i][1]);
#pragma unroll
          for (int i = 0; i < 4; i++) M::mma(u[i], ph[j], b[i][0], b[i][1]);
        } else {
#pragma unroll
          for (int i = 0; i < 4; i++) M::mma(o[d0 + i], ph[j], b[i][0], b[i][1]);
#pragma unroll
          for (int i = 0; i < 4; i++) M::mma(o[d0 + i], pl[j], b[i][0], b[i][1]);
        }
      }
      if constexpr (SPLIT) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
          fa_fold2(o[d0 + i][0], o[d0 + i][1], f0, u[i][0], u[i][1], vi);
          fa_fold2(o[d0 + i][2], o[d0 + i][3], f1, u[i][2], u[i][3], vi);
        }
      }
    }
    if (SPLIT && lost) {  // their pairs are zeros: rows that see one of them get no number, earlier rows are not touched
      const int64_t key = kb * FA_BC + __ffs(lost) - 1;
#pragma unroll
      for (int dt = 0; dt < 16; dt++) {
        if (key <= pos0) o[dt][0] = o[dt][1] = __int_as_float(0x7fffffff);
        if (key <= pos1) o[dt][2] = o[dt][3] = __int_as_float(0x7fffffff);
      }
    }
  }
  // ---- merge the two halves' running states (thread for thread: both cover the same rows and columns)
  if constexpr (HALVES == 2) {
  __syncthreads();  // the tiles are no longer read
  float* const mg = reinterpret_cast<float*>(fa_smem) + (size_t)(warp * 32 + lane) * 68;
  if (half == 1) {
    mg[0] = m0, mg[1] = m1, mg[2] = l0, mg[3] = l1;
#pragma unroll
    for (int dt = 0; dt < 16; dt++)
      *reinterpret_cast<float4*>(mg + 4 + 4 * dt) = make_float4(o[dt][0], o[dt][1], o[dt][2], o[dt][3]);
  }
  __syncthreads();
  if (half == 1) return;
  {
    const float mb0 = mg[0], mb1 = mg[1];
    const float mn0 = fmaxf(m0, mb0), mn1 = fmaxf(m1, mb1);
    const float fa0 = expf(m0 - mn0), fb0 = expf(mb0 - mn0), fa1 = expf(m1 - mn1), fb1 = expf(mb1 - mn1);
    l0 = l0 * fa0 + mg[2] * fb0;
    l1 = l1 * fa1 + mg[3] * fb1;
#pragma unroll
    for (int dt = 0; dt < 16; dt++) {
      const float4 ob = *reinterpret_cast<const float4*>(mg + 4 + 4 * dt);
      o[dt][0] = o[dt][0] * fa0 + ob.x * fb0, o[dt][1] = o[dt][1] * fa0 + ob.y * fb0;
      o[dt][2] = o[dt][2] * fa1 + ob.z * fb1, o[dt][3] = o[dt][3] * fa1 + ob.w * fb1;
    }
  }
  }
  // ---- out / sum
  l0 += __shfl_xor_sync(0xffffffffu, l0, 1);
  l0 += __shfl_xor_sync(0xffffffffu, l0, 2);
  l1 += __shfl_xor_sync(0xffffffffu, l1, 1);
  l1 += __shfl_xor_sync(0xffffffffu, l1, 2);
  const float i0 = (SPLIT ? PMUL : 1.0f) / l0, i1 = (SPLIT ? PMUL : 1.0f) / l1;  // pairs: o left the weights' scale with each step
#pragma unroll
  for (int dt = 0; dt < 16; dt++) {
    if (r0 < a.rows)
      *reinterpret_cast<float2*>(a.ctx + r0 * a.nh * FA_D + h * FA_D + dt * 8 + 2 * t) =
          make_float2(o[dt][0] * i0, o[dt][1] * i0);
    if (r1 < a.rows)
      *reinterpret_cast<float2*>(a.ctx + r1 * a.nh * FA_D + h * FA_D + dt * 8 + 2 * t) =
          make_float2(o[dt][2] * i1, o[dt][3] * i1);
  }
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
  FaArgs f;
  f.q = a.q, f.kcache = a.kcache, f.vcache = a.vcache, f.ctx = a.ctx;
  f.rows = a.rows, f.nh = a.nh, f.nkv = a.nkv, f.cap = a.cap, f.base_pos = base_pos, f.seq = seq;
  f.ldq = a.ldq ? a.ldq : a.nh * FA_D;
  f.kinv = f.vinv = nullptr, f.vlost = nullptr;
  const dim3 grid((unsigned)a.nh, (unsigned)((a.rows + FA_BR - 1) / FA_BR));
  // a grid that fits the GPU in one round: eight warps and pairs of key blocks; larger: four warps, two CTAs per
  // SM (2-byte caches; the f16 pairs of an f32 cache fill an SM's shared memory either way)
  const bool pairs = a.kv_type == E_F32 || (int64_t)grid.x * grid.y <= std::max(1, sm_count());
  void* pooled = nullptr;
  if (a.kv_type == E_F32) {
    const size_t bytes = attention_prefill_scratch_bytes(a);
    void* ws = a.pair_ws && a.pair_ws_bytes >= bytes ? a.pair_ws : nullptr;
    if (!ws) {
      if (keep_scratch_pool_cached()) return 1;
      DYN_CUDA(cudaMallocAsync(&pooled, bytes, s));
      ws = pooled;
    }
    __half* const out = reinterpret_cast<__half*>(ws);
    const size_t plane = (size_t)a.nkv * a.cap * 2 * FA_D;
    float* const inv = reinterpret_cast<float*>(out + 2 * plane);
    unsigned* const lost = reinterpret_cast<unsigned*>(inv + 2 * a.nkv * (a.cap / FA_SPLIT_TILE));
    const int64_t nkeys = base_pos + a.rows;
    fa_split_kernel<<<dim3((unsigned)((nkeys + FA_SPLIT_TILE - 1) / FA_SPLIT_TILE), (unsigned)a.nkv, 2), 256, 0, s>>>(
        reinterpret_cast<const float*>(a.kcache), reinterpret_cast<const float*>(a.vcache), a.nkv, a.cap, seq, nkeys, out, inv, lost);
    count_launch();
    f.kcache = out, f.vcache = out + plane;
    f.kinv = inv, f.vinv = inv + a.nkv * (a.cap / FA_SPLIT_TILE), f.vlost = lost;
  }
  auto run = [&](auto kernel, int halves) -> int {
    const int bytes = fa_smem_bytes(a.kv_type, halves);
    if (ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), bytes)) return 1;
    kernel<<<grid, fa_threads(halves), bytes, s>>>(f);
    return 0;
  };
  int rc;
  if (a.kv_type == E_F32)
    rc = run(attention_prefill_kernel<E_F32, 2>, 2);
  else if (a.kv_type == E_BF16)
    rc = pairs ? run(attention_prefill_kernel<E_BF16, 2>, 2) : run(attention_prefill_kernel<E_BF16, 1>, 1);
  else
    rc = pairs ? run(attention_prefill_kernel<E_F16, 2>, 2) : run(attention_prefill_kernel<E_F16, 1>, 1);
  const cudaError_t fe = pooled ? cudaFreeAsync(pooled, s) : cudaSuccess;
  if (rc) return 1;
  if (fe != cudaSuccess) return cuda_fail(fe, "cudaFreeAsync", __FILE__, __LINE__);
  count_launch();
  DYN_CUDA(cudaGetLastError());
  *handled = true;
  return 0;
}

}  // namespace dyn
