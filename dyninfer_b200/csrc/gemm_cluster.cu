// Dequant GEMM of 33 to 128 activation rows on the 5th-generation tensor cores, K split over a cluster:
// y[m, n] = sum_k x[m, k] * w[n, k], f32 accumulation, the residual or SwiGLU behind it, one launch.
//
// A product of a few dozen rows with a layer's matrix of a small model is over in a few microseconds; what it costs is the
// way from "the activations are there" to "the sums are stored". On mma.sync (gemm_skinny.cu) every CTA brings all rows
// of its K share for 16 to 128 weight rows, and that and one warp's chain of MMAs are the way. Here a CTA takes 128 weight
// rows and up to 768 of K:
//   * Weights do not depend on the kernel before: they are fetched, converted to f16(exact dequantised value) and stored as A
//     operands in tensor memory while that kernel still runs. Two CTAs fit an SM (544 threads of 56 registers). Behind the
//     wait only the activation boxes, sixteen MMAs per 256 of K and the sums are left.
//   * The sums meet through distributed shared memory: every CTA writes its accumulator into the CTA of the cluster that
//     finishes the rows; one cluster barrier; then the parts are added in the order of K, scaled back and stored.
//   * SwiGLU: a tile is 64 rows of gate and the same 64 of up, so both sums of an output are in one CTA.
// Waits for copies and products are bounded; one that runs out sets the device error word. The allocation of tensor memory and the
// cluster barriers have no bound: gemm_cluster_plan.h says why they end.
#include <algorithm>
#include <atomic>

#include "gemm_cluster_plan.h"
#include "raw_box.cuh"
#include "tensor_map.cuh"

namespace dyn {

namespace {

constexpr int GC_CONV = 16;  // conversion warps: lane quarter = warp % 4, quarter of the box = warp / 4
constexpr int GC_MMA_WARP = GC_CONV;
constexpr int GC_THREADS = (GC_CONV + 1) * 32;
static_assert(GC_TILE == TG_BM && GC_UNIT == GS_UNIT, "the plan's tile is the kernel's");

struct GcArgs {
  WRef w;
  const float* inv_s;     // [M]
  const float* residual;
  float* y;               // [M, N]
  int* error;
  int64_t N;              // columns of y (SwiGLU: rows of gate = rows of up)
  int M, bn, nunits, upc, CK, slice, nx, acc_cols, tmem_cols, swiglu;
};

__device__ __forceinline__ void gc_cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void gc_cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t gc_peer(uint32_t addr, int rank) {
  uint32_t p;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(p) : "r"(addr), "r"(rank));
  return p;
}
__device__ __forceinline__ void gc_st_peer(uint32_t addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t addr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(addr)
               : "memory");
}

// Every instruction here runs once or a few times per launch, out of a cold instruction cache (about six cycles each, as in the
// persistent decode kernel), so loops stay rolled.
template <int ENC>
__global__ void __launch_bounds__(GC_THREADS, 2)
gemm_cluster_kernel(const GcArgs a, const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap) {
  constexpr uint32_t RAW_BYTES = TG_BM * gs_words(ENC) * 4;
  extern __shared__ __align__(1024) uint8_t gc_smem[];
  __shared__ uint64_t raw_full[GC_MAX_UPC], a_full, x_full[GC_MAX_UPC], x_free[GC_MAX_UPC], acc_full;
  __shared__ uint32_t tmem_base_s;
  __shared__ int s_abort;
  __shared__ uint32_t s_dst[GC_MAX_BN];  // where row m is finished: its first sum of this CTA's part
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int bn = a.bn, CK = a.CK, M = a.M, slice = a.slice;
  const int rank = (int)(blockIdx.x % (unsigned)CK);
  const int64_t tile = blockIdx.x / (unsigned)CK;
  const int k0 = rank * a.upc, nu = min(a.nunits - k0, a.upc);  // units of 256
  const int64_t n0 = tile * (a.swiglu ? 64 : TG_BM);            // first column of y
  uint8_t* const smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(gc_smem) + 1023) & ~uintptr_t(1023));
  const uint32_t xb = (uint32_t)bn * 128;                       // bytes of a 64-wide chunk of x
  uint8_t* const xs = smem;                                     // operand: [stage][chunk][row][128 bytes, swizzled]
  // one region in turn: raw weights [unit]; the cluster's sums [rank][row of the slice][128]
  uint8_t* const raw = smem + (size_t)a.nx * 4 * xb;
  float* const red = reinterpret_cast<float*>(raw);

  if (tid == GC_MMA_WARP * 32) {
    s_abort = 0;
    for (int i = 0; i < GC_MAX_UPC; i++) mbar_init(raw_full + i, 1), mbar_init(x_full + i, 1), mbar_init(x_free + i, 1);
    mbar_init(&a_full, GC_CONV), mbar_init(&acc_full, 1);
    mbar_fence_init();
    // weights are not produced by the kernels before: they are asked for at once
    for (int u = 0; u < nu; u++) {
      mbar_expect_tx(raw_full + u, RAW_BYTES);
      uint8_t* dst = raw + (size_t)u * RAW_BYTES;
      tma_box_g2s(dst, &wmap, (k0 + u) * gs_words(ENC), (int)n0, raw_full + u);
      if (a.swiglu) tma_box_g2s(dst + RAW_BYTES / 2, &wmap, (k0 + u) * gs_words(ENC), (int)(a.N + n0), raw_full + u);
    }
  }
  // Tensor memory is taken before this block lets the next kernel start, so that kernel cannot take it first and then wait for this one.
  if (warp == GC_MMA_WARP) {
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "r"((uint32_t)a.tmem_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid < M) {
    const int owner = tid / slice;
    s_dst[tid] = gc_peer(smem_u32(red + (rank * slice + tid - owner * slice) * TG_BM), owner);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base_s;
  const int quarter = warp & 3, g = warp >> 2, row = quarter * 32 + lane;
  const uint32_t tlane = tmem + ((uint32_t)(quarter * 32) << 16);

  if (warp < GC_CONV) {
    // ---- A: this thread's weight row, quarter g of every unit ---------------------------------------------------------
    GsRow<ENC> r;
    int gshift = 5;
    const uint8_t *scp = nullptr, *bip = nullptr;
    if constexpr (ENC == E_MLX_U4) {
      while ((1 << gshift) < a.w.group) gshift++;
      const int64_t wrow = min(a.swiglu ? (row < 64 ? n0 + row : a.N + n0 + row - 64) : n0 + row, a.w.rows - 1);
      const int64_t rowb = (a.w.cols >> gshift) * (a.w.aux == E_F32 ? 4 : 2);
      scp = a.w.scales + wrow * rowb, bip = a.w.biases + wrow * rowb;
    }
#pragma unroll 1
    for (int u = 0; u < nu; u++) {
      if constexpr (ENC == E_MLX_U4) {
        const int64_t e = ((int64_t)(k0 + u) * GS_UNIT + g * 64) >> gshift;
        r.sc[0] = __float_as_uint(aux_load(scp, a.w.aux, e)), r.bi[0] = __float_as_uint(aux_load(bip, a.w.aux, e));
        r.sc[1] = r.sc[0], r.bi[1] = r.bi[0];
        if (gshift == 5) r.sc[1] = __float_as_uint(aux_load(scp, a.w.aux, e + 1)), r.bi[1] = __float_as_uint(aux_load(bip, a.w.aux, e + 1));
      }
      // a failed wait is not left with a break: every warp keeps the same sequence of barriers (and the next waits return
      // at once, because they look at s_abort)
      if (!mbar_wait_bounded(raw_full + u, 0, TG_SPINS, &s_abort) && !s_abort) s_abort = 1;
      r.load(raw + (size_t)u * RAW_BYTES, row, g);
      r.align();
      uint32_t out[16];
      const uint32_t taddr = tlane + (uint32_t)a.acc_cols + (uint32_t)(4 * u + g) * 32u;
      r.half(0, out);
      tmem_st16(taddr, out);
      r.half(1, out);
      tmem_st16(taddr + 16, out);
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(&a_full);
    pdl_wait();  // inverse scales, residual; y may still be read by the kernels before
  } else {
    // ---- MMA issue ----------------------------------------------------------------------------------------------------------
    auto ask = [&](int u, int stage) {  // the activations of a unit
      mbar_expect_tx(x_full + stage, 4 * xb);
#pragma unroll 1
      for (int c = 0; c < 4; c++) tma_box_g2s(xs + (size_t)(stage * 4 + c) * xb, &xmap, ((k0 + u) * 4 + c) * (TG_BK / 2), 0, x_full + stage);
    };
    if (lane == 0) {
      pdl_wait_then_trigger();
      for (int u = 0; u < min(nu, a.nx); u++) ask(u, u);
    }
    __syncwarp();
    const uint32_t idesc = umma_idesc(bn);
    const uint64_t dchunk = xb >> 4, desc0 = umma_desc(smem_u32(xs));
    bool ok = mbar_wait_bounded(&a_full, 0, TG_SPINS, &s_abort);
    int stage = 0;
    unsigned phase = 0;
#pragma unroll 1
    for (int u = 0; u < nu && ok; u++) {
      ok = mbar_wait_bounded(x_full + stage, phase, TG_SPINS, &s_abort);
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
        uint32_t acol = tmem + (uint32_t)(a.acc_cols + 128 * u);
        uint64_t desc = desc0 + dchunk * (4 * stage);
#pragma unroll 1
        for (int c = 0; c < 4; c++, acol += 32u, desc += dchunk) {
#pragma unroll
          for (int k4 = 0; k4 < TG_BK / 16; k4++) umma_f16_ts(tmem, acol + 8u * k4, desc + 2 * k4, idesc, (u | c | k4) ? 1u : 0u);
        }
        umma_commit(x_free + stage);
      }
      __syncwarp();
      if (u + a.nx < nu) {  // the stage's next unit, when the MMAs have read it
        ok = mbar_wait_bounded(x_free + stage, phase, TG_SPINS, &s_abort);
        if (ok && elect_one()) ask(u + a.nx, stage);
        __syncwarp();
      }
      if (++stage == a.nx) stage = 0, phase ^= 1u;
    }
    if (!ok && !s_abort) s_abort = 7;
    if (elect_one()) umma_commit(&acc_full);
    __syncwarp();
  }
  // this warp has used up its raw weights: when every warp has, the cluster's sums may take their place (awaited before the first write)
  gc_cluster_arrive();

  // ---- the cluster's sums ------------------------------------------------------------------------------------------------
  if (warp < GC_CONV) {
    if (!mbar_wait_bounded(&acc_full, 0, TG_SPINS, &s_abort) && !s_abort) s_abort = 3;
    tc_fence_after();
  }
  __syncwarp();
  gc_cluster_wait();
  if (warp < GC_CONV) {
    // eight activation rows at a time; the four warps of a lane quarter take turns
#pragma unroll 1
    for (int j0 = g * 8; j0 < M; j0 += 32) {
      uint32_t v[8];
      tmem_ld8(tlane + (uint32_t)j0, v);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int j = 0; j < 8; j++)
        if (j0 + j < M) gc_st_peer(s_dst[j0 + j] + 4u * row, __uint_as_float(v[j]));
    }
    tc_fence_before();
  }
  __syncwarp();
  gc_cluster_arrive();
  // while the others' parts come in: the first residuals of this thread's outputs (column tid % 128, every fourth row of the slice)
  constexpr int Q = 4;
  const int n = tid & 127, mrow = rank * slice, mq = tid >> 7;
  const int mend = warp < GC_CONV && n0 + n < a.N && (!a.swiglu || n < 64) ? min(slice, M - mrow) : 0;
  float* const yp = a.y + (int64_t)mrow * a.N + n0 + n;
  const float* const rp = a.residual ? a.residual + (int64_t)mrow * a.N + n0 + n : nullptr;
  float res[Q], inv[Q];
#pragma unroll
  for (int q = 0; q < Q; q++) inv[q] = mq + 4 * q < mend ? __ldcg(a.inv_s + mrow + mq + 4 * q) : 0.f;
#pragma unroll
  for (int q = 0; q < Q; q++) res[q] = rp && mq + 4 * q < mend ? __ldcg(rp + (int64_t)(mq + 4 * q) * a.N) : 0.f;
  gc_cluster_wait();  // also: nobody writes into this CTA's shared memory from here on, and it may exit
#pragma unroll 1
  for (int mb = mq; mb < mend; mb += 4 * Q) {
    float s[Q], up[Q];
#pragma unroll
    for (int q = 0; q < Q; q++) s[q] = up[q] = 0.f;
    const float* p = red + mb * TG_BM + n;
#pragma unroll 2
    for (int c = 0; c < CK; c++, p += slice * TG_BM)
#pragma unroll
      for (int q = 0; q < Q; q++)
        if (mb + 4 * q < mend) {
          s[q] += p[4 * q * TG_BM];
          if (a.swiglu) up[q] += p[4 * q * TG_BM + 64];
        }
#pragma unroll
    for (int q = 0; q < Q; q++) {
      const int m = mb + 4 * q;
      if (m >= mend) break;
      if (mb != mq) inv[q] = __ldcg(a.inv_s + mrow + m), res[q] = rp ? __ldcg(rp + (int64_t)m * a.N) : 0.f;
      float o = __fmul_rn(s[q], inv[q]);
      if (a.swiglu) o = (o / (1.0f + expf(-o))) * __fmul_rn(up[q], inv[q]);
      yp[(int64_t)m * a.N] = __fadd_rn(o, res[q]);
    }
  }
  __syncwarp();
  if (s_abort) {  // copies and products in flight land before shared and tensor memory are given back
    const long long t0 = clock64();
    while (clock64() - t0 < (1LL << 22)) {
    }
  }
  __syncthreads();
  tc_fence_after();
  if (warp == GC_MMA_WARP)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)a.tmem_cols) : "memory");
  if (tid == 0 && s_abort) report_wait_expired(a.error, DEV_ERR_GEMM_PIPE);
}

// CTAs in clusters of `ck` that the device holds at a time, one per SM: GPCs differ in size, and a cluster does not span two.
int gc_places(int ck) {
  static std::atomic<int> kept[16][9];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  std::atomic<int>* const slot = dev < 16 ? &kept[dev][ck] : nullptr;
  int n = slot ? slot->load(std::memory_order_relaxed) : 0;
  if (n) return n;
  const void* kernel = reinterpret_cast<const void*>(gemm_cluster_kernel<E_Q4_0>);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(ck * 64)), cfg.blockDim = dim3(GC_THREADS), cfg.dynamicSmemBytes = GC_SMEM_OWN;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = (unsigned)ck, attr.val.clusterDim.y = 1, attr.val.clusterDim.z = 1;
  cfg.attrs = &attr, cfg.numAttrs = 1;
  int clusters = 0;
  if (ensure_dynamic_smem(kernel, GC_SMEM) || cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) != cudaSuccess) {
    cudaGetLastError();
    clusters = sm_count() * 3 / 4 / ck;
  }
  n = std::max(1, clusters * ck);
  if (slot) slot->store(n, std::memory_order_relaxed);
  return n;
}
bool gc_plan(const WRef& w, int64_t M, bool swiglu, GcPlan* p) {
  return gc_plan(w.rows, w.cols, gs_words(w.enc), M, swiglu, std::max(1, sm_count()), gc_places, p);
}

template <int ENC>
int gc_launch(const GcArgs& a, const CUtensorMap& wmap, const CUtensorMap& xmap, const GcPlan& p, cudaStream_t s) {
  auto kernel = gemm_cluster_kernel<ENC>;
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), GC_SMEM)) return 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(p.tiles * p.CK)), cfg.blockDim = dim3(GC_THREADS), cfg.dynamicSmemBytes = p.smem, cfg.stream = s;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (pdl_enabled()) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (a.CK > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = (unsigned)a.CK, attr[n].val.clusterDim.y = 1, attr[n].val.clusterDim.z = 1;
    n++;
  }
  cfg.attrs = attr, cfg.numAttrs = n;
  DYN_CUDA(cudaLaunchKernelEx(&cfg, kernel, a, wmap, xmap));
  count_launch();
  return 0;
}

}  // namespace

bool gemm_cluster_prefers(const WRef& w, int64_t M, bool swiglu) {
  return gemm_stream_takes(w) && w.rows <= (1 << 30) && gc_prefers(w.rows, w.cols, gs_words(w.enc), M, swiglu, std::max(1, sm_count()), gc_places);
}

// Activation rows the kernel's boxes read: x has this many rows allocated (those from M on may hold anything).
int64_t gemm_cluster_rows(int64_t M) { return (M + 15) / 16 * 16; }

// y[M, N] = x w^T + residual, or with `swiglu` (the matrix is [gate; up], N = rows / 2) silu(x gate^T) * (x up^T).
// x: f16 rows in natural order, scaled by a power of two per row, x_inv their inverse scales.
int launch_gemm_cluster(const WRef& w, const __half* x, const float* x_inv, int64_t M, float* y, const float* residual, bool swiglu,
                        cudaStream_t s) {
  GcPlan p;
  DYN_CHECK(gc_plan(w, M, swiglu, &p), "dequant GEMM over a cluster: no plan for a product it had accepted");
  GcArgs a{};
  a.w = w, a.inv_s = x_inv;
  a.residual = residual, a.y = y, a.error = device_error_word();
  if (!a.error) return 1;
  a.N = swiglu ? w.rows / 2 : w.rows, a.M = (int)M, a.bn = p.bn, a.nunits = p.nunits, a.upc = p.upc, a.CK = p.CK, a.slice = p.slice, a.nx = p.nx;
  a.swiglu = swiglu ? 1 : 0;
  a.acc_cols = p.acc_cols, a.tmem_cols = p.tmem_cols;
  CUtensorMap wmap, xmap;
  if (make_row_box_map(w.data, w.enc == E_MLX_U4 ? (size_t)w.cols / 2 : (size_t)w.row_bytes(), w.rows, gs_words(w.enc), swiglu ? 64 : TG_BM,
                       &wmap, w.enc == E_MLX_U4) ||
      make_row_box_map(reinterpret_cast<const uint8_t*>(x), (size_t)w.cols * 2, p.bn, TG_BK / 2, p.bn, &xmap, true))
    return 1;
  switch (w.enc) {
    case E_Q4_0: return gc_launch<E_Q4_0>(a, wmap, xmap, p, s);
    case E_Q4_1: return gc_launch<E_Q4_1>(a, wmap, xmap, p, s);
    case E_Q8_0: return gc_launch<E_Q8_0>(a, wmap, xmap, p, s);
    case E_Q4_K: return gc_launch<E_Q4_K>(a, wmap, xmap, p, s);
    case E_Q5_K: return gc_launch<E_Q5_K>(a, wmap, xmap, p, s);
    case E_MLX_U4: return gc_launch<E_MLX_U4>(a, wmap, xmap, p, s);
    default: break;
  }
  DYN_CHECK(false, "dequant GEMM over a cluster: encoding %d", w.enc);
  return 1;
}

}  // namespace dyn
