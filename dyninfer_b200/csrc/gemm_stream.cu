// Dequant GEMM on the 5th-generation tensor cores for quantised matrices whose rows the tensor-copy engine can read:
// y[m, n] = sum_k x[m, k] * w[n, k], f32 accumulation, one launch for any number of activation rows.
//
// The form it replaces for these matrices (gemm_tcgen05.cu keeps the other encodings and odd row sizes) took about 1000 cycles
// per chunk of 128 weight rows x 64, whatever the number of activation rows, against 512 that the MMAs of 256 rows need:
// a warp fetched 36-byte pieces of 32 rows itself and turned them to "thread = row" through a scratch in shared
// memory, 400 instructions per 2048 weights. It also handed out whole tiles, so that 1.3 waves of them took two.
//   * Raw blocks arrive as boxes of 128 rows x 256 weights (one tensor copy each, a ring of three or more). Thread = row
//     reads its row's piece with 16-byte loads: box rows are an odd multiple of 16 bytes apart (MLX-U4: swizzled), so
//     eight lanes hit all banks.
//   * Sixteen warps convert (a warp: the 32 rows of its tensor-memory lanes x one 64-wide quarter of the box) and store the A
//     operand into tensor memory; activations come as f16 boxes of 64 x bn; one thread issues the MMAs. Values are
//     those of gemm_tcgen05.cu: f16(exact dequantised value).
//   * The grid is at most one CTA per SM; the (tile, K) space is cut into equal runs of whole tiles or of 256-wide units. A tile
//     that several CTAs work on is finished by the one that arrives last: the others leave their sums in scratch and
//     count themselves in, nobody waits for anybody. The sums are added in the order of K, so results do not depend on
//     who was last.
// All waits are bounded; one that runs out sets the device error word.
#include <algorithm>

#include "raw_box.cuh"
#include "tensor_map.cuh"

namespace dyn {

namespace {

constexpr int GS_CONV = 16;   // conversion warps: lane quarter = warp % 4, quarter of the box = warp / 4
constexpr int GS_RAW_WARP = GS_CONV, GS_X_WARP = GS_CONV + 1, GS_MMA_WARP = GS_CONV + 2;
constexpr int GS_THREADS = (GS_CONV + 3) * 32;
constexpr int GS_MAX_RAW = 6, GS_MAX_X = 8;
constexpr int GS_SMEM = 220 * 1024;

struct GsArgs {
  WRef w;
  const float* inv_s;     // [Mpad]
  const float* residual;
  float* y;               // [M, N]
  float* part;            // [CTA][2][bn][128]: sums of a run's first tile (begun by another CTA) and of its last (left unfinished)
  unsigned* count;        // [CTA]: arrivals at the tile whose first unit the CTA holds; zero between launches
  int* error;
  int64_t M, N, total;    // total: units over all tiles
  int mtiles, nunits, bn, nraw, nx;
  int gran;               // units that stay together: 1, or a tile's
  int xc;                 // chunks per activation stage (2 or 4)
};

struct GsSeg {
  int64_t tile;
  int k0, k1;             // units [k0, k1) of the tile
};
__device__ __forceinline__ GsSeg gs_segment(int64_t u, int64_t end, int nunits) {
  GsSeg s;
  s.tile = u / nunits;
  s.k0 = (int)(u - s.tile * nunits);
  s.k1 = (int)min((int64_t)nunits, s.k0 + (end - u));
  return s;
}
// the CTA whose run [c * total / grid, (c + 1) * total / grid) holds unit u
__device__ __forceinline__ int gs_owner(int64_t u, int64_t total, int grid) { return (int)(((u + 1) * grid + total - 1) / total - 1); }

template <int ENC>
__global__ void __launch_bounds__(GS_THREADS, 1)
gemm_stream_kernel(const GsArgs a, const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap) {
  constexpr uint32_t RAW_BYTES = TG_BM * gs_words(ENC) * 4;
  extern __shared__ __align__(1024) uint8_t gs_smem[];
  __shared__ uint64_t raw_full[GS_MAX_RAW], raw_empty[GS_MAX_RAW], x_full[GS_MAX_X], x_empty[GS_MAX_X];
  __shared__ uint64_t a_full[2], a_empty[2], acc_full, acc_free;
  __shared__ uint32_t tmem_base_s;
  __shared__ int s_abort;
  __shared__ unsigned s_count;
  __shared__ float s_inv[256];
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int bn = a.bn, nunits = a.nunits, nraw = a.nraw, nx = a.nx;
  const int64_t N = a.N;
  const int64_t parts = a.total / a.gran;
  const int64_t u0 = (int64_t)blockIdx.x * parts / gridDim.x * a.gran, u1 = ((int64_t)blockIdx.x + 1) * parts / gridDim.x * a.gran;
  uint8_t* const smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(gs_smem) + 1023) & ~uintptr_t(1023));
  uint8_t* const xbase = smem + (size_t)nraw * RAW_BYTES;
  const uint32_t xb = (uint32_t)bn * 128, x_bytes = xb * a.xc;  // of a chunk, of a stage

  if (tid == 0) {
    s_abort = 0;
    for (int i = 0; i < GS_MAX_RAW; i++) mbar_init(raw_full + i, 1), mbar_init(raw_empty + i, GS_CONV);
    for (int i = 0; i < GS_MAX_X; i++) mbar_init(x_full + i, 1), mbar_init(x_empty + i, 1);
    for (int i = 0; i < 2; i++) mbar_init(a_full + i, GS_CONV), mbar_init(a_empty + i, 1);
    mbar_init(&acc_full, 1), mbar_init(&acc_free, GS_CONV);
    mbar_fence_init();
  }
  if (warp == GS_MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base_s;

  if (warp < GS_CONV) {
    const int quarter = warp & 3, g = warp >> 2;
    const int row = quarter * 32 + lane;  // of the tile
    const uint32_t tlane = tmem + ((uint32_t)(quarter * 32) << 16);
    int rs = 0, gshift = 5;
    unsigned rphase = 0, unit = 0, nseg = 0;
    bool waited = false;
    if constexpr (ENC == E_MLX_U4) {
      while ((1 << gshift) < a.w.group) gshift++;
    }
    for (int64_t u = u0; u < u1; nseg++) {
      const GsSeg sg = gs_segment(u, u1, nunits);
      const int64_t n0 = sg.tile / a.mtiles * TG_BM, m0 = sg.tile % a.mtiles * bn;
      const int64_t n = n0 + row;
      const uint8_t *scp = nullptr, *bip = nullptr;
      GsRow<ENC> r;
      auto aux = [&](int k) {  // MLX: the unit's scales and biases of this thread's row
        const int64_t e = ((int64_t)k * GS_UNIT + g * 64) >> gshift;
        r.sc[0] = __float_as_uint(aux_load(scp, a.w.aux, e)), r.bi[0] = __float_as_uint(aux_load(bip, a.w.aux, e));
        r.sc[1] = r.sc[0], r.bi[1] = r.bi[0];
        if (gshift == 5) r.sc[1] = __float_as_uint(aux_load(scp, a.w.aux, e + 1)), r.bi[1] = __float_as_uint(aux_load(bip, a.w.aux, e + 1));
      };
      uint32_t nsc[2], nbi[2];  // of the next unit, on the way while this one is converted
      if constexpr (ENC == E_MLX_U4) {
        const int64_t rowb = (a.w.cols >> gshift) * (a.w.aux == E_F32 ? 4 : 2);
        scp = a.w.scales + min(n, N - 1) * rowb, bip = a.w.biases + min(n, N - 1) * rowb;
        aux(sg.k0);
        nsc[0] = r.sc[0], nsc[1] = r.sc[1], nbi[0] = r.bi[0], nbi[1] = r.bi[1];
      }
      for (int k = sg.k0; k < sg.k1; k++, unit++) {
        // a failed wait is not left with a break: every warp keeps the same sequence of barriers (and the next waits return
        // at once, because they look at s_abort)
        if (!mbar_wait_bounded(raw_full + rs, rphase, TG_SPINS, &s_abort) && !s_abort) s_abort = 1;
        r.load(smem + (size_t)rs * RAW_BYTES, row, g);
        if constexpr (ENC == E_MLX_U4) {
          const uint32_t s0 = nsc[0], s1 = nsc[1], b0 = nbi[0], b1 = nbi[1];
          if (k + 1 < sg.k1) aux(k + 1);
          nsc[0] = r.sc[0], nsc[1] = r.sc[1], nbi[0] = r.bi[0], nbi[1] = r.bi[1];
          r.sc[0] = s0, r.sc[1] = s1, r.bi[0] = b0, r.bi[1] = b1;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(raw_empty + rs);
        if (++rs == nraw) rs = 0, rphase ^= 1u;
        r.align();
        uint32_t out[16];
        r.half(0, out);
        const int slot = (int)(unit & 1u);
        if (unit >= 2 && !mbar_wait_bounded(a_empty + slot, ((unit >> 1) - 1u) & 1u, TG_SPINS, &s_abort) && !s_abort) s_abort = 2;
        tc_fence_after();
        const uint32_t taddr = tlane + TG_TMEM_A_COL + (uint32_t)(4 * slot + g) * 32u;
        tmem_st16(taddr, out);
        r.half(1, out);
        tmem_st16(taddr + 16, out);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(a_full + slot);
      }
      // ---- the tile's sums: y, or this CTA's part of a tile that several share ---------------------------------------
      if (!waited) pdl_wait();
      waited = true;
      auto sync = [] { asm volatile("bar.sync 1, %0;" ::"n"(GS_CONV * 32) : "memory"); };
      if (tid < bn) s_inv[tid] = m0 + tid < a.M ? __ldcg(a.inv_s + m0 + tid) : 0.f;
      const bool whole = sg.k1 - sg.k0 == nunits;
      int first = 0, last = 0;
      if (!whole) {
        first = gs_owner(sg.tile * nunits, a.total, gridDim.x), last = gs_owner((sg.tile + 1) * nunits - 1, a.total, gridDim.x);
        if (tid == 0) s_count = *reinterpret_cast<volatile unsigned*>(a.count + first);
      }
      sync();
      if (!mbar_wait_bounded(&acc_full, nseg & 1u, TG_SPINS, &s_abort) && !s_abort) s_abort = 3;
      tc_fence_after();
      const int mleft = (int)min((int64_t)bn, a.M - m0);
      auto slot_of = [&](int c) { return a.part + ((size_t)(2 * c + (c == first ? 1 : 0)) * bn) * TG_BM + row; };
      bool finish = whole;
      if (!whole) {
        finish = s_count == (unsigned)(last - first);  // everybody else has been here: no need to write the sums down
        if (!finish) {
          float* p = slot_of((int)blockIdx.x);
          for (int j0 = g * 16; j0 < mleft; j0 += 64) {
            uint32_t v[16];
            tmem_ld16(tlane + (uint32_t)j0, v);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int j = 0; j < 16; j++)
              if (j0 + j < mleft) p[(j0 + j) * TG_BM] = __uint_as_float(v[j]);
          }
          __threadfence();
          sync();
          if (tid == 0) s_count = atomicAdd(a.count + first, 1u);
          sync();
          finish = s_count == (unsigned)(last - first);
        }
        if (finish) {
          __threadfence();
          if (tid == 0) a.count[first] = 0;
        }
      }
      if (finish) {
        float* const out = a.y + m0 * N + n;
        const float* const res = a.residual ? a.residual + m0 * N + n : nullptr;
        for (int j0 = g * 16; j0 < mleft; j0 += 64) {
          uint32_t v[16];
          tmem_ld16(tlane + (uint32_t)j0, v);
          float q[16];
          if (res && n < N) {
#pragma unroll
            for (int j = 0; j < 16; j++) q[j] = j0 + j < mleft ? res[(int64_t)(j0 + j) * N] : 0.f;
          } else {
#pragma unroll
            for (int j = 0; j < 16; j++) q[j] = 0.f;
          }
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          float t[16];
          if (whole) {
#pragma unroll
            for (int j = 0; j < 16; j++) t[j] = __uint_as_float(v[j]);
          } else {
#pragma unroll
            for (int j = 0; j < 16; j++) t[j] = 0.f;
            for (int c = first; c <= last; c++) {
              if (c == (int)blockIdx.x) {
#pragma unroll
                for (int j = 0; j < 16; j++) t[j] += __uint_as_float(v[j]);
              } else {
                const float* p = slot_of(c) + j0 * TG_BM;
                float e[16];
#pragma unroll
                for (int j = 0; j < 16; j++) e[j] = j0 + j < mleft ? __ldcg(p + j * TG_BM) : 0.f;
#pragma unroll
                for (int j = 0; j < 16; j++) t[j] += e[j];
              }
            }
          }
          if (n < N) {
#pragma unroll
            for (int j = 0; j < 16; j++)
              if (j0 + j < mleft) out[(int64_t)(j0 + j) * N] = __fadd_rn(__fmul_rn(t[j], s_inv[j0 + j]), q[j]);
          }
        }
      }
      tc_fence_before();
      sync();  // also: s_inv and s_count are no longer read
      if (lane == 0) mbar_arrive(&acc_free);
      u += sg.k1 - sg.k0;
    }
    if (!waited) pdl_wait();
  } else if (warp == GS_RAW_WARP) {
    // ---------------- raw weights: not produced by the kernels before, so they are asked for at once ------------------
    if (lane == 0) {
      int rs = 0;
      unsigned phase = 1, i = 0;
      bool ok = true;
      for (int64_t u = u0; u < u1 && ok;) {
        const GsSeg sg = gs_segment(u, u1, nunits);
        const int n0 = (int)(sg.tile / a.mtiles * TG_BM);
        for (int k = sg.k0; k < sg.k1; k++, i++) {
          if (i >= (unsigned)nraw && !mbar_wait_bounded(raw_empty + rs, phase, TG_SPINS, &s_abort)) {
            if (!s_abort) s_abort = 4;
            ok = false;
            break;
          }
          mbar_expect_tx(raw_full + rs, RAW_BYTES);
          tma_box_g2s(smem + (size_t)rs * RAW_BYTES, &wmap, k * gs_words(ENC), n0, raw_full + rs);
          if (++rs == nraw) rs = 0, phase ^= 1u;
        }
        u += sg.k1 - sg.k0;
      }
    }
  } else if (warp == GS_X_WARP) {
    // ---------------- activations -------------------------------------------------------------------------------------
    if (lane == 0) {
      pdl_wait_then_trigger();
      int xs = 0;
      unsigned phase = 1, i = 0;
      bool ok = true;
      for (int64_t u = u0; u < u1 && ok;) {
        const GsSeg sg = gs_segment(u, u1, nunits);
        const int m0 = (int)(sg.tile % a.mtiles * bn);
        for (int c = sg.k0 * 4; c < sg.k1 * 4; c += a.xc, i++) {
          if (i >= (unsigned)nx && !mbar_wait_bounded(x_empty + xs, phase, TG_SPINS, &s_abort)) {
            if (!s_abort) s_abort = 5;
            ok = false;
            break;
          }
          mbar_expect_tx(x_full + xs, x_bytes);
          for (int j = 0; j < a.xc; j++)
            tma_box_g2s(xbase + (size_t)xs * x_bytes + j * xb, &xmap, (c + j) * (TG_BK / 2), m0, x_full + xs);
          if (++xs == nx) xs = 0, phase ^= 1u;
        }
        u += sg.k1 - sg.k0;
      }
    }
  } else {
    // ---------------- MMA issue: the pipeline's serial section ------------------------------------------------------------
    // The whole warp walks along so that slots, phases and descriptors stay in uniform registers; one lane issues. A
    // hand-over per 256 (128) of K: one per 64 took 290 cycles of waits and commits beside 290 of issuing, for MMAs that
    // need 96 (48 rows) to 512 (256 rows).
    const uint32_t idesc = umma_idesc(bn);
    const uint64_t desc0 = umma_desc(smem_u32(xbase)), dchunk = xb >> 4;
    const int per = 4 / a.xc;
    uint64_t desc = desc0;
    int xs = 0;
    unsigned xphase = 0, unit = 0, nseg = 0;
    bool ok = true;
    for (int64_t u = u0; u < u1 && ok; nseg++) {
      const GsSeg sg = gs_segment(u, u1, nunits);
      uint32_t accumulate = 0u;
      if (nseg && !mbar_wait_bounded(&acc_free, (nseg - 1u) & 1u, TG_SPINS, &s_abort)) {
        if (!s_abort) s_abort = 6;
        break;
      }
      for (int k = sg.k0; k < sg.k1 && ok; k++, unit++) {
        const int slot = (int)(unit & 1u);
        ok = mbar_wait_bounded(a_full + slot, (unit >> 1) & 1u, TG_SPINS, &s_abort);
        uint32_t acol = tmem + TG_TMEM_A_COL + (uint32_t)slot * 128u;
        for (int h = 0; h < per && ok; h++) {
          ok = mbar_wait_bounded(x_full + xs, xphase, TG_SPINS, &s_abort);
          if (!ok) break;
          tc_fence_after();
          if (elect_one()) {
            for (int c = 0; c < a.xc; c++) {
#pragma unroll
              for (int k4 = 0; k4 < TG_BK / 16; k4++)
                umma_f16_ts(tmem, acol + 32u * c + 8u * k4, desc + dchunk * c + 2 * k4, idesc, k4 ? 1u : accumulate);
              accumulate = 1u;
            }
            umma_commit(x_empty + xs);
            if (h == per - 1) umma_commit(a_empty + slot);
          }
          accumulate = 1u;
          __syncwarp();
          acol += 32u * a.xc, desc += dchunk * a.xc;
          if (++xs == nx) xs = 0, desc = desc0, xphase ^= 1u;
        }
        if (!ok && !s_abort) s_abort = 7;
      }
      if (elect_one()) umma_commit(&acc_full);
      __syncwarp();
      u += sg.k1 - sg.k0;
    }
  }
  __syncwarp();
  if (s_abort) {  // copies and products in flight land before shared and tensor memory are given back
    const long long t0 = clock64();
    while (clock64() - t0 < (1LL << 22)) {
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == GS_MMA_WARP)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  if (tid == 0 && s_abort) report_wait_expired(a.error, DEV_ERR_GEMM_PIPE);
}

template <int ENC>
int gs_launch(const GsArgs& a, const CUtensorMap& wmap, const CUtensorMap& xmap, int grid, size_t smem, cudaStream_t s) {
  auto kernel = gemm_stream_kernel<ENC>;
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), GS_SMEM + 1024)) return 1;
  DYN_CUDA(launch_pdl(kernel, dim3((unsigned)grid), dim3(GS_THREADS), smem, s, a, wmap, xmap));
  return 0;
}

// Bytes of a row; 0 when the encoding has no fixed row here.
size_t gs_row_bytes(const WRef& w) { return w.enc == E_MLX_U4 ? (size_t)w.cols / 2 : (size_t)w.row_bytes(); }

}  // namespace

// Matrices the kernel reads: whole 256-wide units, rows a tensor copy can take.
bool gemm_stream_takes(const WRef& w) {
  switch (w.enc) {
    case E_Q4_0:
    case E_Q4_1:
    case E_Q8_0:
    case E_Q4_K:
    case E_Q5_K: break;
    case E_MLX_U4:
      if (w.group < 32 || (w.group & (w.group - 1)) || w.cols % w.group) return false;
      break;
    default: return false;
  }
  return w.rows >= 1 && w.cols >= GS_UNIT && w.cols % GS_UNIT == 0 && gs_row_bytes(w) % 16 == 0 &&
         (reinterpret_cast<uintptr_t>(w.data) & 15) == 0;
}

// Tile width and split with the least estimated time. Cycles fitted to products of 2000 x 2048 to 40000 x 2560 at 40 to 1500
// rows (within 20 %): a unit costs the conversion's 1400 and 9 per activation row (bringing the rows out of L2 takes longer than
// their MMAs); a tile that one CTA finishes alone 1500 + 12 per row; a tile shared between CTAs 4500 + 22 per row,
// and 10 per row for every further part that is added up. Whole tiles win where they fill their last wave (282 tiles of
// 6016 x 5120 x 1500: 92 against 99 us), equal shares elsewhere (192 tiles of 12288 x 4096 x 512: 60 against 68 us),
// narrow tiles where there are few (2000 x 2048 x 512: 17 against 28 us).
GsPlan gemm_stream_plan(const WRef& w, int64_t M, bool whole_tiles) {
  const int64_t sms = std::max(1, sm_count()), ntiles = (w.rows + TG_BM - 1) / TG_BM, nunits = w.cols / GS_UNIT;
  GsPlan best{};
  double least = 1e30;
  const int64_t t0 = (M + 255) / 256;
  for (int64_t mt = t0; mt <= 2 * t0 + 2 && (mt == t0 || (M + mt - 1) / mt > 48); mt++) {
    const int64_t bn = ((M + mt - 1) / mt + 15) / 16 * 16, tiles = ntiles * mt, total = tiles * nunits;
    if ((mt - 1) * bn >= M) continue;
    const double unit = 1400 + 9.0 * bn;
    auto take = [&](int64_t grid, int64_t gran, double cycles) {
      if (cycles >= least) return;
      least = cycles;
      best.mtiles = (int)mt, best.bn = (int)bn, best.nunits = (int)nunits, best.total = total, best.grid = (int)grid, best.gran = (int)gran;
    };
    const int64_t waves = (tiles + sms - 1) / sms;
    take((tiles + waves - 1) / waves, nunits, waves * (nunits * unit + 1500 + 12.0 * bn));
    for (int64_t q = (total + sms - 1) / sms, i = 0; i < 4 && !whole_tiles; i++, q *= 2) {
      const int64_t grid = (total + q - 1) / q;
      take(grid, 1, q * unit + (1.3 + (double)q / nunits) * (4500 + 22.0 * bn) + std::max(0.0, (double)nunits / q - 1) * 10 * bn);
      if (q >= nunits) break;
    }
  }
  best.part_bytes = best.gran > 1 ? 0 : (size_t)2 * best.grid * best.bn * TG_BM * 4;
  return best;
}

// xh: f16 rows [mtiles * bn, K] in natural order with inverse scales; part: plan's part_bytes; count: grid words, zero (left zero)
int launch_gemm_stream(const WRef& w, const GsPlan& p, const __half* xh, const float* inv_s, int64_t M, float* y, const float* residual,
                       float* part, unsigned* count, cudaStream_t s) {
  GsArgs a{};
  a.w = w, a.inv_s = inv_s, a.residual = residual, a.y = y, a.part = part, a.count = count;
  a.error = device_error_word();
  if (!a.error) return 1;
  a.M = M, a.N = w.rows, a.total = p.total, a.mtiles = p.mtiles, a.nunits = p.nunits, a.bn = p.bn, a.gran = p.gran;
  const int raw = TG_BM * gs_words(w.enc) * 4, xb = p.bn * 128;
  // three boxes of weights keep enough of them in flight for the memory's rate; activation chunks come out of L2 and are used up
  // faster: at least three as well, then as many as fit
  a.xc = 2 * 4 * xb + 3 * raw <= GS_SMEM ? 4 : 2;
  a.nraw = 3;
  while (a.nraw > 2 && 2 * a.xc * xb + a.nraw * raw > GS_SMEM) a.nraw--;
  a.nx = std::min(GS_MAX_X, (GS_SMEM - a.nraw * raw) / (xb * a.xc));
  while (a.nraw < GS_MAX_RAW && (a.nraw + 1) * raw + a.nx * a.xc * xb <= GS_SMEM) a.nraw++;
  CUtensorMap wmap, xmap;
  if (make_row_box_map(w.data, gs_row_bytes(w), w.rows, gs_words(w.enc), TG_BM, &wmap, w.enc == E_MLX_U4)) return 1;
  if (make_row_box_map(reinterpret_cast<const uint8_t*>(xh), (size_t)w.cols * 2, (int64_t)p.mtiles * p.bn, TG_BK / 2, p.bn, &xmap, true)) return 1;
  const size_t smem = (size_t)a.nraw * raw + (size_t)a.nx * a.xc * xb + 1024;
  int rc = 1;
  switch (w.enc) {
    case E_Q4_0: rc = gs_launch<E_Q4_0>(a, wmap, xmap, p.grid, smem, s); break;
    case E_Q4_1: rc = gs_launch<E_Q4_1>(a, wmap, xmap, p.grid, smem, s); break;
    case E_Q8_0: rc = gs_launch<E_Q8_0>(a, wmap, xmap, p.grid, smem, s); break;
    case E_Q4_K: rc = gs_launch<E_Q4_K>(a, wmap, xmap, p.grid, smem, s); break;
    case E_Q5_K: rc = gs_launch<E_Q5_K>(a, wmap, xmap, p.grid, smem, s); break;
    case E_MLX_U4: rc = gs_launch<E_MLX_U4>(a, wmap, xmap, p.grid, smem, s); break;
    default: break;
  }
  if (rc) return rc;
  count_launch();
  DYN_CUDA(cudaGetLastError());
  return 0;
}

}  // namespace dyn
