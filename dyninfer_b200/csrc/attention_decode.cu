// Decode attention (one query row per sequence, any number of sequences) on 2-byte KV caches, on the tensor
// cores: the query heads that share a kv head are worked on together.
//
// The form it replaces gave every (query head, row) CTAs of its own: the cached rows of a kv head were read
// once per query head, and a key cost a warp ~25 instructions (multiply, five shuffles, two exponentials for
// ONE head), so instruction issue and not the cache's bytes set the pace (8 rows of 32 heads at context 2048:
// 113 us for 67 MB). Here a CTA takes (row, kv head, slice of the keys); its warps walk 16 keys at a time:
//   S = Q K^T  A operand: the G <= 8 query heads as rows, row g = leading term of head g, row g + 8 = the second
//              term (Q enters as two or three terms of the cache's type, so an f32 query keeps its bits);
//              B operand: K rows as they lie in memory, 16 bytes per lane -- the order of the head
//              dimensions inside the product is free, so a lane's eight consecutive dimensions serve two steps.
//   O += P V   the accumulator layout of S is the A layout of P (terms again in rows g and g + 8);
//              V comes through shared memory (cp.async, a ring per warp) and ldmatrix.trans.
// Scores, maxima, sums and the output stay f32; each slice leaves (unnormalised output, max, sum) and the
// merge kernel combines the slices in a fixed order, either into f32 rows or straight into the f16 operand of
// the following product.
#include <algorithm>

#include "common.cuh"

namespace dyn {

namespace {

constexpr int AD_WARPS = 4;
constexpr int AD_KEYS = 16;   // keys per warp and step
constexpr int AD_NST = 2;     // V stages per warp

template <int KV>
struct AdT;
template <>
struct AdT<E_BF16> {
  static constexpr int TERMS = 3;  // 8 bits each
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

// Grid (kv head, row, slice). D = head dim (64 or 128), G = query heads per kv head.
template <int KV, int D>
__global__ void __launch_bounds__(AD_WARPS * 32)
attention_decode_kernel(const AttnArgs a, float* __restrict__ part, int nsplit, int G) {
  using T = AdT<KV>;
  constexpr int TERMS = T::TERMS, CH = D / 32, NT = D / 8;  // 16-byte chunks of a row per lane; output tiles of 8 dims
  constexpr int PITCH = D * 2 + 16, STAGE = AD_KEYS * PITCH;
  __shared__ __align__(16) uint8_t s_v[AD_WARPS][AD_NST][STAGE];
  __shared__ float s_m[AD_WARPS][8], s_l[AD_WARPS][8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int64_t kvh = blockIdx.x, r = blockIdx.y;
  const int sp = blockIdx.z;
  pdl_trigger();
  pdl_wait();
  const int64_t pos = a.row_pos ? a.row_pos[r] : a.base_pos + r;
  const int64_t seq = a.row_seq ? a.row_seq[r] : 0;
  const int n = (int)pos + 1;
  const int per = ((n + nsplit - 1) / nsplit + AD_KEYS - 1) / AD_KEYS * AD_KEYS;
  const int k_lo = min(sp * per, n), k_hi = min(k_lo + per, n);
  const uint8_t* kb = reinterpret_cast<const uint8_t*>(a.kcache) + (seq * a.nkv + kvh) * a.cap * (D * 2);
  const uint8_t* vb = reinterpret_cast<const uint8_t*>(a.vcache) + (seq * a.nkv + kvh) * a.cap * (D * 2);
  // Q: chunk j of lane t = dims 32 j + 8 t ..; products 2j and 2j + 1 take its first and last four
  uint32_t q[TERMS][CH][4];
  {
    const float* qv = a.q + r * (a.ldq ? a.ldq : a.nh * D) + (kvh * G + (g < G ? g : 0)) * D + 8 * t;
    const float scale = 1.0f / sqrtf((float)D);
#pragma unroll
    for (int j = 0; j < CH; j++) {
      float4 x = *reinterpret_cast<const float4*>(qv + 32 * j), y = *reinterpret_cast<const float4*>(qv + 32 * j + 4);
      (void)scale;
#pragma unroll
      for (int k = 0; k < TERMS; k++) {
        q[k][j][0] = T::pack(x.x, x.y), q[k][j][1] = T::pack(x.z, x.w);
        q[k][j][2] = T::pack(y.x, y.y), q[k][j][3] = T::pack(y.z, y.w);
      }
    }
  }
  const float scale = 1.0f / sqrtf((float)D);
  float o[NT][4], ox[TERMS > 2 ? NT : 1][4];
#pragma unroll
  for (int i = 0; i < NT; i++) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
  (void)ox;
  float m = -3.40282347e38f, l = 0.f;  // head g's running maximum, this lane's share of the sum

  const int steps = (k_hi - k_lo + AD_KEYS - 1) / AD_KEYS;
  const uint32_t sv = (uint32_t)__cvta_generic_to_shared(&s_v[warp][0][0]);
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
  if (warp < steps) load_k(warp);
  load_v(warp, 0);
  int st = 0;
  for (int s = warp; s < steps; s += AD_WARPS) {
    load_v(s + AD_WARPS, st ^ 1);
    float c[2][2][4];  // key group, independent chains
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
      for (int e = 0; e < 2; e++) c[h][e][0] = c[h][e][1] = c[h][e][2] = c[h][e][3] = 0.f;
#pragma unroll
    for (int j = 0; j < CH; j++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        T::mma(c[h][0], q[0][j][0], q[1][j][0], q[0][j][1], q[1][j][1], kr[h][j].x, kr[h][j].y);
        T::mma(c[h][1], q[0][j][2], q[1][j][2], q[0][j][3], q[1][j][3], kr[h][j].z, kr[h][j].w);
        if constexpr (TERMS > 2) {
          T::mma(c[h][0], q[2][j][0], 0u, q[2][j][1], 0u, kr[h][j].x, kr[h][j].y);
          T::mma(c[h][1], q[2][j][2], 0u, q[2][j][3], 0u, kr[h][j].z, kr[h][j].w);
        }
      }
    if (s + AD_WARPS < steps) load_k(s + AD_WARPS);
    // head g's scores of keys 8 h + 2 t, + 1
    float p[2][2];
    float bm = -3.40282347e38f;
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int key = k_lo + s * AD_KEYS + 8 * h + 2 * t + e;
        const float v = (c[h][0][e] + c[h][1][e]) + (c[h][0][2 + e] + c[h][1][2 + e]);
        p[h][e] = key < k_hi ? v * scale : -3.40282347e38f;
        bm = fmaxf(bm, p[h][e]);
      }
    bm = fmaxf(bm, __shfl_xor_sync(0xffffffffu, bm, 1));
    bm = fmaxf(bm, __shfl_xor_sync(0xffffffffu, bm, 2));
    const float mn = fmaxf(m, bm), f = expf(m - mn);
    const bool rescale = __any_sync(0xffffffffu, f != 1.0f);
    m = mn, l *= f;
    if (rescale) {
#pragma unroll
      for (int i = 0; i < NT; i++) o[i][0] *= f, o[i][1] *= f, o[i][2] *= f, o[i][3] *= f;
    }
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int key = k_lo + s * AD_KEYS + 8 * h + 2 * t + e;
        p[h][e] = key < k_hi ? expf(p[h][e] - m) : 0.f;
        l += p[h][e];
      }
    uint32_t pa[TERMS][2];
#pragma unroll
    for (int k = 0; k < TERMS; k++) pa[k][0] = T::pack(p[0][0], p[0][1]), pa[k][1] = T::pack(p[1][0], p[1][1]);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();
    const uint32_t vrow = sv + st * STAGE + (lane & 15) * PITCH + (lane >> 4) * 16;
#pragma unroll
    for (int i = 0; i < NT; i += 2) {  // two tiles of eight dims per ldmatrix
      uint32_t b0, b1, b2, b3;
      asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                   : "=r"(b0), "=r"(b1), "=r"(b2), "=r"(b3)
                   : "r"(vrow + i * 16));
      T::mma(o[i], pa[0][0], pa[1][0], pa[0][1], pa[1][1], b0, b1);
      T::mma(o[i + 1], pa[0][0], pa[1][0], pa[0][1], pa[1][1], b2, b3);
      if constexpr (TERMS > 2) {
        T::mma(o[i], pa[2][0], 0u, pa[2][1], 0u, b0, b1);
        T::mma(o[i + 1], pa[2][0], 0u, pa[2][1], 0u, b2, b3);
      }
    }
    __syncwarp();  // the stage is read; the next round may overwrite it
    st ^= 1;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  l += __shfl_xor_sync(0xffffffffu, l, 1);
  l += __shfl_xor_sync(0xffffffffu, l, 2);
  if (t == 0) s_m[warp][g] = m, s_l[warp][g] = l;
  __syncthreads();  // also: every warp is done with its V ring, which now takes the warps' outputs
  float gm = s_m[0][g];
#pragma unroll
  for (int w = 1; w < AD_WARPS; w++) gm = fmaxf(gm, s_m[w][g]);
  const float wgt = expf(m - gm);
  float* so = reinterpret_cast<float*>(&s_v[0][0][0]);  // [warp][8 heads][D]
  static_assert(sizeof(s_v) >= AD_WARPS * 8 * D * 4, "outputs fit the rings");
#pragma unroll
  for (int i = 0; i < NT; i++)
    *reinterpret_cast<float2*>(so + (warp * 8 + g) * D + i * 8 + 2 * t) =
        make_float2((o[i][0] + o[i][2]) * wgt, (o[i][1] + o[i][3]) * wgt);
  __syncthreads();
  for (int i = threadIdx.x; i < G * D; i += AD_WARPS * 32) {
    const int h = i / D, d = i % D;
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < AD_WARPS; w++) v += so[(w * 8 + h) * D + d];
    float* out = part + ((r * a.nh + kvh * G + h) * nsplit + sp) * (D + 2);
    out[d] = v;
    if (d == 0) {
      float mm = s_m[0][h], ll = 0.f;
#pragma unroll
      for (int w = 1; w < AD_WARPS; w++) mm = fmaxf(mm, s_m[w][h]);
#pragma unroll
      for (int w = 0; w < AD_WARPS; w++) ll += s_l[w][h] * expf(s_m[w][h] - mm);
      out[D] = mm, out[D + 1] = ll;
    }
  }
}

// Slices -> the f16 operand of the following product (fragment order of `enc`, power-of-two scale, inverse in
// inv_s). One block per row, because the scale is the row's; a thread takes eight consecutive dims of a head.
__global__ void __launch_bounds__(1024)
attention_merge_frag_kernel(const float* __restrict__ part, int nsplit, int nh, int d, __half* __restrict__ frag,
                            float* __restrict__ inv_s, int enc) {
  __shared__ float red[32];
  pdl_trigger();
  const int64_t r = blockIdx.x;
  const int k = threadIdx.x * 8, h = k / d, d0 = k - h * d;
  float o[8];
#pragma unroll
  for (int e = 0; e < 8; e++) o[e] = 0.f;
  pdl_wait();
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

// Slices -> f32 rows. One block per (head, row): thread (slice group, pair of dims), eight groups of slices.
__global__ void __launch_bounds__(512)
attention_merge_f32_kernel(const float* __restrict__ part, int nsplit, int64_t nh, int d, float* __restrict__ ctx) {
  __shared__ float sw[32], so[8][128], sl;
  pdl_trigger();
  const int64_t h = blockIdx.x, r = blockIdx.y;
  const int tid = threadIdx.x, pairs = d >> 1, grp = tid / pairs, p = tid - grp * pairs;
  const float* p0 = part + (r * nh + h) * nsplit * (d + 2);
  pdl_wait();
  if (tid < 32) {  // the slices' weights
    const float2 ml = tid < nsplit ? *reinterpret_cast<const float2*>(p0 + tid * (d + 2) + d) : make_float2(-3.40282347e38f, 0.f);
    const float w = expf(ml.x - warp_max(ml.x));
    sw[tid] = w;
    const float l = warp_sum(ml.y * w);
    if (tid == 0) sl = 1.0f / l;
  }
  float2 v[4];
#pragma unroll
  for (int q = 0; q < 4; q++)
    v[q] = grp + 8 * q < nsplit ? *reinterpret_cast<const float2*>(p0 + (grp + 8 * q) * (d + 2) + 2 * p) : make_float2(0.f, 0.f);
  __syncthreads();
  float a = 0.f, b = 0.f;
#pragma unroll
  for (int q = 0; q < 4; q++) a += v[q].x * sw[grp + 8 * q], b += v[q].y * sw[grp + 8 * q];
  so[grp][2 * p] = a, so[grp][2 * p + 1] = b;
  __syncthreads();
  if (tid < d) {
    float o = 0.f;
#pragma unroll
    for (int q = 0; q < 8; q++) o += so[q][tid];
    ctx[r * nh * d + h * d + tid] = o * sl;
  }
}

}  // namespace

// Shapes the kernel takes: 2-byte caches, head dim 64 or 128, up to eight query heads per kv head.
bool attention_decode_takes(const AttnArgs& a) {
  return (a.kv_type == E_BF16 || a.kv_type == E_F16) && (a.d == 64 || a.d == 128) && a.nkv > 0 && a.nh % a.nkv == 0 &&
         a.nh / a.nkv <= 8 && a.nh * a.d <= 8192 && a.ldq % 4 == 0 && (reinterpret_cast<uintptr_t>(a.q) & 15) == 0;
}

// Slices per (row, kv head): about three CTAs per SM, at least 64 keys each at full capacity. Depends on shapes
// only, so a captured graph stays valid as positions grow.
int attention_decode_splits(const AttnArgs& a) {
  const int64_t ctas = a.rows * a.nkv;
  int64_t n = (3 * (int64_t)std::max(1, sm_count())) / ctas;
  n = std::min<int64_t>(n, a.cap / 64);
  return (int)std::max<int64_t>(1, std::min<int64_t>(32, n));
}

int launch_attention_decode(const AttnArgs& a, float* part, int nsplit, __half* frag, float* inv_s, int enc, cudaStream_t s) {
  const dim3 grid((unsigned)a.nkv, (unsigned)a.rows, (unsigned)nsplit);
  const int G = (int)(a.nh / a.nkv);
  cudaError_t e;
  if (a.kv_type == E_BF16)
    e = a.d == 128 ? launch_pdl(attention_decode_kernel<E_BF16, 128>, grid, dim3(AD_WARPS * 32), 0, s, a, part, nsplit, G)
                   : launch_pdl(attention_decode_kernel<E_BF16, 64>, grid, dim3(AD_WARPS * 32), 0, s, a, part, nsplit, G);
  else
    e = a.d == 128 ? launch_pdl(attention_decode_kernel<E_F16, 128>, grid, dim3(AD_WARPS * 32), 0, s, a, part, nsplit, G)
                   : launch_pdl(attention_decode_kernel<E_F16, 64>, grid, dim3(AD_WARPS * 32), 0, s, a, part, nsplit, G);
  DYN_CUDA(e);
  if (frag) {
    const int threads = (int)((a.nh * a.d / 8 + 31) / 32 * 32);
    DYN_CUDA(launch_pdl(attention_merge_frag_kernel, dim3((unsigned)a.rows), dim3(threads), 0, s, (const float*)part, nsplit, (int)a.nh,
                        (int)a.d, frag, inv_s, enc));
  } else {
    DYN_CUDA(launch_pdl(attention_merge_f32_kernel, dim3((unsigned)a.nh, (unsigned)a.rows), dim3((unsigned)a.d * 4), 0, s,
                        (const float*)part, nsplit, a.nh, (int)a.d, a.ctx));
  }
  count_launch(2);
  DYN_CUDA(cudaGetLastError());
  return 0;
}

}  // namespace dyn
