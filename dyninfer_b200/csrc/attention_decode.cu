// Decode attention (one query row per sequence, any number of sequences) on 2-byte KV caches, on the tensor
// cores: the query heads that share a kv head are worked on together.
//
// The form it replaces gave every (query head, row) CTAs of its own: the cached rows of a kv head were read
// once per query head, and a key cost a warp ~25 instructions (multiply, five shuffles, two exponentials for
// ONE head), so instruction issue and not the cache's bytes set the pace (8 rows of 32 heads at context 2048:
// 113 us for 67 MB). Here a CTA takes (row, kv head, slice of the keys); its warps walk 16 keys at a time:
//   S = Q K^T  A operand: the G <= 8 query heads as rows, row g = leading term of head g, row g + 8 = the second
//              term (Q enters as three terms of bf16, or as two of f16 after a power of two that keeps the second
//              term out of the subnormals, so an f32 query keeps its bits at any magnitude);
//              B operand: K rows as they lie in memory, 16 bytes per lane -- the order of the head
//              dimensions inside the product is free, so a lane's eight consecutive dimensions serve two steps.
//   O += P V   the accumulator layout of S is the A layout of P (terms again in rows g and g + 8);
//              V comes through shared memory (cp.async, a ring per warp) and ldmatrix.trans.
// Scores, maxima, sums and the output stay f32. An mma truncates where it adds to its accumulator (about 1.5e-8 of the
// sum each time, always toward zero), so a step's P V starts from zero, smallest terms first, and joins the running
// output by a rounded fma: as exact as the per-row kernel in f32, at the time per call it had (one row of 32 heads at
// 8191: f16 14.4, bf16 15.7 us). On f16 caches the weights, their sum included, enter times 2^14: what lies below 2^-14
// of the largest weight would lose its bits to the subnormals. Error against 64 bits with the mma adding up the output
// and nothing scaled / now / per-row kernel, f16, 256 rows at 7936: one-sided values 5.5e-6 / 1.0e-7 / 4.7e-7, a long
// tail 1.9e-5 / 8.1e-7 / 2.4e-6; one row at 300, small queries 1.7e-5 / 2.5e-7 / 1.6e-7.
// Each slice leaves (unnormalised output, max, sum) and the slices are combined in a fixed order: by the CTAs of a
// cluster through shared memory, or (many rows) by a merge kernel straight into the f16 operand of the following product.
// Per-head RMSNorm, rotation and the write of the new cache row happen here too: the preparation kernel they used to be
// cost a launch (3.4 us) per layer.
#include <algorithm>

#include "common.cuh"

namespace dyn {

namespace {

constexpr int AD_KEYS = 16;   // keys per warp and step
constexpr int AD_NST = 2;     // V stages per warp

template <int KV>
struct AdT;
template <>
struct AdT<E_BF16> {
  static constexpr int TERMS = 3;  // 8 bits each
  static constexpr bool SCALED = false;  // f32's range
  static constexpr float PMUL = 1.0f;
  __device__ static __forceinline__ uint16_t bits(float x) { return __bfloat16_as_ushort(__float2bfloat16_rn(x)); }
  __device__ static __forceinline__ uint32_t pack(float& x, float& y) {  // leading terms; x and y keep what is left
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    x -= __low2float(h), y -= __high2float(h);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
  __device__ static __forceinline__ void mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  }
};
template <>
struct AdT<E_F16> {
  static constexpr int TERMS = 2;  // 11 bits each
  static constexpr bool SCALED = true;
  static constexpr float PMUL = 16384.0f;
  __device__ static __forceinline__ uint16_t bits(float x) { return __half_as_ushort(__float2half_rn(x)); }
  __device__ static __forceinline__ uint32_t pack(float& x, float& y) {
    const __half2 h = __floats2half2_rn(x, y);
    x -= __low2float(h), y -= __high2float(h);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
  __device__ static __forceinline__ void mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  }
};

__device__ __forceinline__ void ad_cp16(uint32_t dst, const void* src, bool live) {
  const int n = live ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}

struct AdArgs {
  AttnArgs a;
  int prep;        // q, k, v are a product's raw output: per-head RMSNorm, rotation and the cache write happen here
  const float *k, *v;
  int64_t ldk, ldv;
  const void *q_norm_w, *k_norm_w;
  int norm_type, has_norm, has_rope;
  float eps;
  float* part;     // slices' results; NULL: the slices of a (row, kv head) are a cluster and meet in shared memory
  int nsplit, G;   // G: query heads per kv head
};

// Rotate-half RoPE of a pair, as the other kernels evaluate it.
__device__ __forceinline__ void ad_rope(float& lo, float& hi, float pos, float freq) {
  float sv, cv;
  sincosf(__fmul_rn(pos, freq), &sv, &cv);
  const float x = lo, y = hi;
  lo = __fsub_rn(__fmul_rn(x, cv), __fmul_rn(y, sv));
  hi = __fadd_rn(__fmul_rn(x, sv), __fmul_rn(y, cv));
}

// Grid (kv head, row, slice). D = head dim (64 or 128). The cached rows do not depend on the kernel in front, so
// every warp asks for its first 16 keys before it waits for the queries; the row written by this step is worked on
// out of shared memory, by the slice that would come next.
template <int KV, int D, int W>
__global__ void __launch_bounds__(W * 32)
attention_decode_kernel(const AdArgs p, const __grid_constant__ FreqTable ft) {
  using T = AdT<KV>;
  constexpr int TERMS = T::TERMS, CH = D / 32, NT = D / 8;  // 16-byte chunks of a row per lane; output tiles of 8 dims
  constexpr int PITCH = D * 2 + 16, STAGE = AD_KEYS * PITCH, E = D / 64;
  const AttnArgs& a = p.a;
  extern __shared__ __align__(16) uint8_t s_v[];  // [W][AD_NST][STAGE], then the warps' outputs [W][8][D]
  __shared__ float s_m[W][8], s_l[W][8], s_q[8][D + 4], s_o[8][D], s_ml[8][2];
  __shared__ __align__(16) uint16_t s_k[D], s_nv[D];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3, G = p.G, nsplit = p.nsplit;
  const int64_t kvh = blockIdx.x, r = blockIdx.y;
  const int sp = blockIdx.z;
  const int64_t pos = a.row_pos ? a.row_pos[r] : a.base_pos + r;
  const int64_t seq = a.row_seq ? a.row_seq[r] : 0;
  const int n = (int)pos + (p.prep ? 0 : 1);  // keys that lie in the cache
  const int per = ((n + nsplit - 1) / nsplit + AD_KEYS - 1) / AD_KEYS * AD_KEYS;
  const int k_lo = min(sp * per, n), k_hi = min(k_lo + per, n);
  const bool owner = p.prep && sp == min((per ? n / per : 0), nsplit - 1);  // takes the new key as well
  uint8_t* kb = reinterpret_cast<uint8_t*>(const_cast<void*>(a.kcache)) + (seq * a.nkv + kvh) * a.cap * (D * 2);
  uint8_t* vb = reinterpret_cast<uint8_t*>(const_cast<void*>(a.vcache)) + (seq * a.nkv + kvh) * a.cap * (D * 2);
  const int steps = (k_hi - k_lo + AD_KEYS - 1) / AD_KEYS;
  const uint32_t sv = (uint32_t)__cvta_generic_to_shared(s_v + warp * AD_NST * STAGE);
  // V of step s (keys past the slice arrive as zeros: their weights are 0, and 0 * anything must stay 0)
  auto load_v = [&](int s, int st) {
    if (s < steps) {
      const int key0 = k_lo + s * AD_KEYS;
#pragma unroll
      for (int i = 0; i < AD_KEYS * D * 2 / 16 / 32; i++) {
        const int e = i * 32 + lane, key = e / (D / 8), c = e % (D / 8);
        const bool live = key0 + key < k_hi;
        ad_cp16(sv + st * STAGE + key * PITCH + c * 16, vb + (int64_t)(live ? key0 + key : 0) * (D * 2) + c * 16, live);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  uint4 kr[2][CH];
  auto load_k = [&](int s) {
    const int key0 = k_lo + s * AD_KEYS + g;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int key = min(key0 + 8 * h, k_hi - 1);
#pragma unroll
      for (int j = 0; j < CH; j++) kr[h][j] = *reinterpret_cast<const uint4*>(kb + (int64_t)key * (D * 2) + 64 * j + 16 * t);
    }
  };
  if (!p.prep) pdl_wait_then_trigger();  // the kernel in front may have written cache rows
  if (warp < steps) load_k(warp);
  load_v(warp, 0);

  // ---- this step's heads: warps take the G query heads, the key and the value in turn -------------------------------
  struct __align__(4 * E) Vec { float v[E]; };
  const int i0 = E * lane;  // a lane holds the rotated pairs (i, i + D / 2), i = i0 ..
  if (!p.prep) {
    for (int h = warp; h < G; h += W) {
      const float* q = a.q + r * (a.ldq ? a.ldq : a.nh * D) + (kvh * G + h) * D;
      for (int i = lane; i < D; i += 32) s_q[h][i] = q[i];
    }
  } else {
    bool waited = false;
    for (int job = warp; job < G + 2; job += W) {  // 0 .. G - 1: query heads, then the key, the value
      const bool query = job < G, key = job == G;
      if (!query && !owner) break;
      float w[2 * E];
      if ((query || key) && p.has_norm) {
        const uint8_t* nw = reinterpret_cast<const uint8_t*>(query ? p.q_norm_w : p.k_norm_w);
#pragma unroll
        for (int e = 0; e < E; e++) w[e] = aux_load(nw, p.norm_type, i0 + e), w[E + e] = aux_load(nw, p.norm_type, D / 2 + i0 + e);
      }
      if (!waited) pdl_wait_then_trigger();
      waited = true;
      const float* src = query ? a.q + r * (a.ldq ? a.ldq : a.nh * D) + (kvh * G + job) * D
                               : key ? p.k + r * p.ldk + kvh * D : p.v + r * p.ldv + kvh * D;
      float x[2 * E];
      {
        const Vec lo = *reinterpret_cast<const Vec*>(src + i0), hi = *reinterpret_cast<const Vec*>(src + D / 2 + i0);
#pragma unroll
        for (int e = 0; e < E; e++) x[e] = lo.v[e], x[E + e] = hi.v[e];
      }
      if ((query || key) && p.has_norm) {
        // the order in which the stand-alone QKV preparation adds the squares: same bits
        float ss[E];
#pragma unroll
        for (int e = 0; e < E; e++) ss[e] = fmaf(x[E + e], x[E + e], x[e] * x[e]);
#pragma unroll
        for (int o = E == 2 ? 8 : 16; o > 0; o >>= 1) {
#pragma unroll
          for (int e = 0; e < E; e++) ss[e] += __shfl_xor_sync(0xffffffffu, ss[e], o);
        }
        if (E == 2) {
          ss[0] += ss[E - 1];
          ss[0] += __shfl_xor_sync(0xffffffffu, ss[0], 16);
        }
        const float inv = 1.0f / sqrtf(ss[0] / (float)D + p.eps);
#pragma unroll
        for (int e = 0; e < 2 * E; e++) x[e] = __fmul_rn(__fmul_rn(x[e], inv), w[e]);
      }
      if ((query || key) && p.has_rope) {
#pragma unroll
        for (int e = 0; e < E; e++) ad_rope(x[e], x[E + e], (float)pos, ft.f[i0 + e]);
      }
      if (query) {
#pragma unroll
        for (int e = 0; e < E; e++) s_q[job][i0 + e] = x[e], s_q[job][D / 2 + i0 + e] = x[E + e];
      } else {
        uint16_t* dst = key ? s_k : s_nv;
        uint16_t* out = reinterpret_cast<uint16_t*>((key ? kb : vb) + pos * (D * 2));
#pragma unroll
        for (int e = 0; e < E; e++) {
          dst[i0 + e] = out[i0 + e] = T::bits(x[e]);
          dst[D / 2 + i0 + e] = out[D / 2 + i0 + e] = T::bits(x[E + e]);
        }
      }
    }
    if (!waited) pdl_wait_then_trigger();  // the results may still be read by the kernels in front
  }
  __syncthreads();
  // Q: chunk j of lane t = dims 32 j + 8 t ..; products 2j and 2j + 1 take its first and last four
  uint32_t q[TERMS][CH][4];
  float scale = 1.0f / sqrtf((float)D);
  {
    const float* qv = s_q[g < G ? g : 0] + 8 * t;
    float qs = 1.0f;
    if constexpr (T::SCALED) {
      float mx = 0.f;
#pragma unroll
      for (int j = 0; j < CH; j++)
#pragma unroll
        for (int e = 0; e < 8; e++) mx = fmaxf(mx, fabsf(qv[32 * j + e]));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
      float inv;
      f16_scale_for(mx, &qs, &inv);
      scale *= inv;
    }
#pragma unroll
    for (int j = 0; j < CH; j++) {
      float4 x = *reinterpret_cast<const float4*>(qv + 32 * j), y = *reinterpret_cast<const float4*>(qv + 32 * j + 4);
      if constexpr (T::SCALED) {
        x.x *= qs, x.y *= qs, x.z *= qs, x.w *= qs;
        y.x *= qs, y.y *= qs, y.z *= qs, y.w *= qs;
      }
#pragma unroll
      for (int k = 0; k < TERMS; k++) {
        q[k][j][0] = T::pack(x.x, x.y), q[k][j][1] = T::pack(x.z, x.w);
        q[k][j][2] = T::pack(y.x, y.y), q[k][j][3] = T::pack(y.z, y.w);
      }
    }
  }
  float o[NT][2];  // head g, dims 8 i + 2 t, + 1
#pragma unroll
  for (int i = 0; i < NT; i++) o[i][0] = o[i][1] = 0.f;
  float m = -3.40282347e38f, l = 0.f;  // head g's running maximum, this lane's share of the sum

  // 16 keys key0 .. (those below k_end count): K in kr, V in stage st
  auto work = [&](int key0, int k_end, int st, auto after_scores) {
    float c[2][2][4];  // key group, independent chains
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
      for (int e = 0; e < 2; e++) c[h][e][0] = c[h][e][1] = c[h][e][2] = c[h][e][3] = 0.f;
    if constexpr (TERMS > 2) {
#pragma unroll
      for (int j = 0; j < CH; j++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
          T::mma(c[h][0], q[2][j][0], 0u, q[2][j][1], 0u, kr[h][j].x, kr[h][j].y);
          T::mma(c[h][1], q[2][j][2], 0u, q[2][j][3], 0u, kr[h][j].z, kr[h][j].w);
        }
    }
#pragma unroll
    for (int j = 0; j < CH; j++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        T::mma(c[h][0], q[0][j][0], q[1][j][0], q[0][j][1], q[1][j][1], kr[h][j].x, kr[h][j].y);
        T::mma(c[h][1], q[0][j][2], q[1][j][2], q[0][j][3], q[1][j][3], kr[h][j].z, kr[h][j].w);
      }
    after_scores();
    // head g's scores of keys 8 h + 2 t, + 1
    float pr[2][2];
    float bm = -3.40282347e38f;
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int key = key0 + 8 * h + 2 * t + e;
        const float v = (c[h][0][e] + c[h][0][2 + e]) + (c[h][1][e] + c[h][1][2 + e]);
        pr[h][e] = key < k_end ? v * scale : -3.40282347e38f;
        bm = fmaxf(bm, pr[h][e]);
      }
    bm = fmaxf(bm, __shfl_xor_sync(0xffffffffu, bm, 1));
    bm = fmaxf(bm, __shfl_xor_sync(0xffffffffu, bm, 2));
    const float mn = fmaxf(m, bm), f = expf(m - mn);
    m = mn, l *= f;
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int key = key0 + 8 * h + 2 * t + e;
        pr[h][e] = key < k_end ? expf(pr[h][e] - m) * T::PMUL : 0.f;
        l += pr[h][e];
      }
    uint32_t pa[TERMS][2];
#pragma unroll
    for (int k = 0; k < TERMS; k++) pa[k][0] = T::pack(pr[0][0], pr[0][1]), pa[k][1] = T::pack(pr[1][0], pr[1][1]);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();
    const uint32_t vrow = sv + st * STAGE + (lane & 15) * PITCH + (lane >> 4) * 16;
#pragma unroll
    for (int i = 0; i < NT; i += 2) {  // two tiles of eight dims per ldmatrix
      uint32_t b0, b1, b2, b3;
      asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                   : "=r"(b0), "=r"(b1), "=r"(b2), "=r"(b3)
                   : "r"(vrow + i * 16));
      float u[4] = {0.f, 0.f, 0.f, 0.f}, v[4] = {0.f, 0.f, 0.f, 0.f};
      if constexpr (TERMS > 2) {
        T::mma(u, pa[2][0], 0u, pa[2][1], 0u, b0, b1);
        T::mma(v, pa[2][0], 0u, pa[2][1], 0u, b2, b3);
      }
      T::mma(u, pa[0][0], pa[1][0], pa[0][1], pa[1][1], b0, b1);
      T::mma(v, pa[0][0], pa[1][0], pa[0][1], pa[1][1], b2, b3);
#pragma unroll
      for (int e = 0; e < 2; e++) {
        o[i][e] = fmaf(o[i][e], f, u[e] + u[2 + e]);
        o[i + 1][e] = fmaf(o[i + 1][e], f, v[e] + v[2 + e]);
      }
    }
    __syncwarp();  // the stage is read; the next round may overwrite it
  };
  int st = 0;
  for (int s = warp; s < steps; s += W) {
    load_v(s + W, st ^ 1);
    work(k_lo + s * AD_KEYS, k_hi, st, [&]() {
      if (s + W < steps) load_k(s + W);
    });
    st ^= 1;
  }
  if (owner && warp == W - 1) {  // the new key, alone in a step: its row in fragment row 0, zeros elsewhere
#pragma unroll
    for (int j = 0; j < CH; j++) {
      kr[0][j] = g == 0 ? *reinterpret_cast<const uint4*>(reinterpret_cast<const uint8_t*>(s_k) + 64 * j + 16 * t) : make_uint4(0, 0, 0, 0);
      kr[1][j] = make_uint4(0, 0, 0, 0);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    uint8_t* stage = s_v + (warp * AD_NST + st) * STAGE;
#pragma unroll
    for (int i = 0; i < AD_KEYS * D * 2 / 16 / 32; i++) {
      const int e = i * 32 + lane, key = e / (D / 8), c = e % (D / 8);
      *reinterpret_cast<uint4*>(stage + key * PITCH + c * 16) =
          key == 0 ? *reinterpret_cast<const uint4*>(reinterpret_cast<const uint8_t*>(s_nv) + c * 16) : make_uint4(0, 0, 0, 0);
    }
    __syncwarp();
    work((int)pos, (int)pos + 1, st, []() {});
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  l += __shfl_xor_sync(0xffffffffu, l, 1);
  l += __shfl_xor_sync(0xffffffffu, l, 2);
  if (t == 0) s_m[warp][g] = m, s_l[warp][g] = l;
  __syncthreads();  // also: every warp is done with its V ring, which now takes the warps' outputs
  float gm = s_m[0][g];
#pragma unroll
  for (int w = 1; w < W; w++) gm = fmaxf(gm, s_m[w][g]);
  const float wgt = expf(m - gm);
  float* so = reinterpret_cast<float*>(s_v);  // [warp][8 heads][D]
#pragma unroll
  for (int i = 0; i < NT; i++)
    *reinterpret_cast<float2*>(so + (warp * 8 + g) * D + i * 8 + 2 * t) =
        make_float2(o[i][0] * wgt, o[i][1] * wgt);
  __syncthreads();
  for (int i = threadIdx.x; i < G * D; i += W * 32) {
    const int h = i / D, d = i % D;
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < W; w++) v += so[(w * 8 + h) * D + d];
    float mm = s_m[0][h], ll = 0.f;
    if (d == 0) {
#pragma unroll
      for (int w = 1; w < W; w++) mm = fmaxf(mm, s_m[w][h]);
#pragma unroll
      for (int w = 0; w < W; w++) ll += s_l[w][h] * expf(s_m[w][h] - mm);
    }
    if (p.part) {
      float* out = p.part + ((r * a.nh + kvh * G + h) * nsplit + sp) * (D + 2);
      out[d] = v;
      if (d == 0) out[D] = mm, out[D + 1] = ll;
    } else {
      s_o[h][d] = v;
      if (d == 0) s_ml[h][0] = mm, s_ml[h][1] = ll;
    }
  }
  if (p.part) return;
  // ---- the cluster's slices, in order: a CTA takes every nsplit-th output ---------------------------------------------
  asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
  {
    const uint32_t ob = (uint32_t)__cvta_generic_to_shared(&s_o[0][0]), mb = (uint32_t)__cvta_generic_to_shared(&s_ml[0][0]);
    for (int i = threadIdx.x * nsplit + sp; i < G * D; i += W * 32 * nsplit) {
      const int h = i / D;
      float ov[8], mv[8], lv[8];
#pragma unroll
      for (int c = 0; c < 8; c++) {
        if (c >= nsplit) break;
        uint32_t ra, rm;
        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(ob + 4u * (uint32_t)i), "r"(c));
        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(rm) : "r"(mb + 8u * (uint32_t)h), "r"(c));
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(ov[c]) : "r"(ra) : "memory");
        asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(mv[c]), "=f"(lv[c]) : "r"(rm) : "memory");
      }
      float mx = -3.40282347e38f, lo = 0.f, oo = 0.f;
#pragma unroll
      for (int c = 0; c < 8; c++)
        if (c < nsplit) mx = fmaxf(mx, mv[c]);
#pragma unroll
      for (int c = 0; c < 8; c++)
        if (c < nsplit) {
          const float w = expf(mv[c] - mx);  // an empty slice has sum 0 and contributes nothing
          lo += lv[c] * w, oo += ov[c] * w;
        }
      a.ctx[r * a.nh * D + kvh * G * D + i] = oo / lo;
    }
  }
  asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}

// Slices -> the f16 operand of the following product (fragment order of `enc`, power-of-two scale, inverse in
// inv_s). One block per row, because the scale is the row's; a thread takes eight consecutive dims of a head.
__global__ void __launch_bounds__(1024)
attention_merge_frag_kernel(const float* part, int nsplit, int nh, int d, __half* frag, float* inv_s, int enc) {
  __shared__ float red[32];
  const int64_t r = blockIdx.x;
  const int k = threadIdx.x * 8, h = k / d, d0 = k - h * d;
  float o[8];
#pragma unroll
  for (int e = 0; e < 8; e++) o[e] = 0.f;
  pdl_wait_then_trigger();
  if (k < nh * d) {
    const float* p0 = part + (r * nh + h) * nsplit * (d + 2);
    float gm = -3.40282347e38f, gl = 0.f;
    constexpr int B = 4;  // slices in flight; an online maximum, so that one pass over them is enough
    for (int s0 = 0; s0 < nsplit; s0 += B) {
      float2 ml[B], v[B][4];
#pragma unroll
      for (int q = 0; q < B; q++) {
        const float* ps = p0 + min(s0 + q, nsplit - 1) * (d + 2);  // slices start on 8-byte boundaries
        ml[q] = *reinterpret_cast<const float2*>(ps + d);
#pragma unroll
        for (int e = 0; e < 4; e++) v[q][e] = *reinterpret_cast<const float2*>(ps + d0 + 2 * e);
      }
#pragma unroll
      for (int q = 0; q < B; q++) {
        if (s0 + q >= nsplit) break;
        const float mn = fmaxf(gm, ml[q].x), f = expf(gm - mn), w = expf(ml[q].x - mn);
        gm = mn;
        gl = gl * f + ml[q].y * w;  // an empty slice has sum 0 and contributes nothing
#pragma unroll
        for (int e = 0; e < 4; e++) o[2 * e] = o[2 * e] * f + v[q][e].x * w, o[2 * e + 1] = o[2 * e + 1] * f + v[q][e].y * w;
      }
    }
    const float il = 1.0f / gl;
#pragma unroll
    for (int e = 0; e < 8; e++) o[e] *= il;
  }
  float mx = 0.f;
#pragma unroll
  for (int e = 0; e < 8; e++) mx = fmaxf(mx, fabsf(o[e]));
  mx = warp_max(mx);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
  __syncthreads();
  mx = 0.f;
  for (int i = 0; i < (int)(blockDim.x >> 5); i++) mx = fmaxf(mx, red[i]);
  float sc, inv;
  f16_scale_for(mx, &sc, &inv);
  if (threadIdx.x == 0) inv_s[r] = inv;
  if (k < nh * d) sk_store_frag8(frag + r * nh * d, enc, k, o, sc);
}

}  // namespace

// Shapes the kernel takes: 2-byte caches, head dim 64 or 128, up to eight query heads per kv head.
bool attention_decode_takes(const AttnArgs& a) {
  return (a.kv_type == E_BF16 || a.kv_type == E_F16) && (a.d == 64 || a.d == 128) && a.nkv > 0 && a.nh % a.nkv == 0 &&
         a.nh / a.nkv <= 8 && a.nh * a.d <= 8192 && a.ldq % 4 == 0 && (reinterpret_cast<uintptr_t>(a.q) & 15) == 0;
}

// Slices of the form that leaves partial results: about three CTAs per SM, at least 64 keys each at full capacity.
// Depends on shapes only, so a captured graph stays valid as positions grow.
int attention_decode_splits(const AttnArgs& a) {
  const int64_t ctas = a.rows * a.nkv;
  int64_t n = (3 * (int64_t)std::max(1, sm_count())) / ctas;
  n = std::min<int64_t>(n, a.cap / 64);
  return (int)std::max<int64_t>(1, std::min<int64_t>(32, n));
}

template <int KV, int D, int W>
static int ad_run(const AdArgs& p, const FreqTable& ft, cudaStream_t s) {
  auto kernel = attention_decode_kernel<KV, D, W>;
  const int smem = std::max(W * AD_NST * AD_KEYS * (D * 2 + 16), W * 8 * D * 4);
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem)) return 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)p.a.nkv, (unsigned)p.a.rows, (unsigned)p.nsplit), cfg.blockDim = dim3(W * 32);
  cfg.dynamicSmemBytes = (size_t)smem, cfg.stream = s;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (pdl_enabled()) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (!p.part) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = attr[n].val.clusterDim.y = 1, attr[n].val.clusterDim.z = (unsigned)p.nsplit;
    n++;
  }
  cfg.attrs = attr, cfg.numAttrs = n;
  DYN_CUDA(cudaLaunchKernelEx(&cfg, kernel, p, ft));
  count_launch();
  return 0;
}

template <int W>
static int ad_dispatch(const AdArgs& p, const FreqTable& ft, cudaStream_t s) {
  if (p.a.kv_type == E_BF16) return p.a.d == 128 ? ad_run<E_BF16, 128, W>(p, ft, s) : ad_run<E_BF16, 64, W>(p, ft, s);
  return p.a.d == 128 ? ad_run<E_F16, 128, W>(p, ft, s) : ad_run<E_F16, 64, W>(p, ft, s);
}

// With `prep` the QKV preparation is part of it (its arguments beyond q describe k, v and the norms). Few rows: the
// slices of a (row, kv head) form a cluster of up to eight CTAs of eight warps and write f32 rows; many rows (`frag`):
// slices of four warps, merged into the f16 operand of the following product.
int launch_attention_decode(const AttnArgs& a, const QkvPrepArgs* prep, const FreqTable* ft, float* part, __half* frag, float* inv_s,
                            int enc, cudaStream_t s) {
  AdArgs p{};
  p.a = a, p.G = (int)(a.nh / a.nkv);
  static const FreqTable none{};
  if (prep) {
    p.prep = 1, p.k = prep->k, p.v = prep->v;
    p.ldk = prep->ldk ? prep->ldk : a.nkv * a.d, p.ldv = prep->ldv ? prep->ldv : a.nkv * a.d;
    p.q_norm_w = prep->q_norm_w, p.k_norm_w = prep->k_norm_w, p.norm_type = prep->norm_w_type;
    p.has_norm = prep->has_norm, p.has_rope = prep->has_rope, p.eps = prep->eps;
  }
  if (!frag) {
    // up to one CTA per SM, at least 64 keys each at full capacity
    int n = 8;
    while (n > 1 && ((int64_t)n * a.rows * a.nkv > std::max(1, sm_count()) || a.cap / n < 64)) n /= 2;
    p.nsplit = n;
    if (ad_dispatch<8>(p, ft ? *ft : none, s)) return 1;
    DYN_CUDA(cudaGetLastError());
    return 0;
  }
  p.part = part, p.nsplit = attention_decode_splits(a);
  if (ad_dispatch<4>(p, ft ? *ft : none, s)) return 1;
  const int threads = (int)((a.nh * a.d / 8 + 31) / 32 * 32);
  DYN_CUDA(launch_pdl(attention_merge_frag_kernel, dim3((unsigned)a.rows), dim3(threads), 0, s, (const float*)part, p.nsplit, (int)a.nh,
                      (int)a.d, frag, inv_s, enc));
  count_launch();
  DYN_CUDA(cudaGetLastError());
  return 0;
}

}  // namespace dyn
