// Plans of the dequant GEMM over a cluster (gemm_cluster.cu): how a product is cut, and what a block of it takes of an SM.
// Host code without CUDA, so that it can be checked on a machine that has none.
//
// A block takes its tensor memory with an instruction that waits until the columns are free, and the blocks of a cluster then
// wait for one another. Two clusters (of two streams; a stream's next kernel starts when all blocks of this one have their columns) that meet
// on two SMs, each ahead on one of them, would wait for ever if their columns did not fit one SM together. The hardware does not
// count columns when it places blocks, so shared memory keeps them apart. There are two kinds of plan:
//   256 columns, 77 KB or more: two fit an SM, and all its 512 columns; three do not fit;
//   512 columns, 150 KB or more: none of either kind fits beside it.
// So no block of this kernel ever waits for the columns of another one. Beside a block of another kernel that takes tensor memory it may
// wait, but those wait for no other block while they hold it, and end.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>

namespace dyn {

constexpr int GC_TILE = 128;       // weight rows of a block
constexpr int GC_UNIT = 256;       // K elements of a unit
constexpr int GC_MAX_UPC = 3;      // units of A operands in tensor memory (128 columns each) behind the accumulator
constexpr int GC_MAX_BN = 128;
constexpr int GC_SMEM = 222 * 1024;
constexpr int GC_SMEM_256 = 77 * 1024, GC_SMEM_512 = 150 * 1024;  // least dynamic shared memory by columns
constexpr int GC_SMEM_OWN = 116 * 1024;                           // two blocks of this do not fit an SM
constexpr int GC_SM_SMEM = 228 * 1024, GC_SM_COLS = 512;          // an SM's; a block's shared memory counts 1 KB more
static_assert(3 * (GC_SMEM_256 + 1024) > GC_SM_SMEM && GC_SMEM_512 + GC_SMEM_256 + 2048 > GC_SM_SMEM, "see above");

struct GcPlan {
  int bn, CK, upc, nunits, slice, nx, acc_cols, tmem_cols;
  int64_t tiles;
  size_t smem;
};

// A product of M activation rows with a matrix of rows x cols, `words` 32-bit words per row and unit. places(ck): blocks in clusters of
// `ck` that the device holds at a time.
// K is split as far as one CTA per SM allows (two of a product on an SM take almost twice as long), with an eighth of the SMs left
// over because clusters do not fill every GPC (6144 x 1280 in 144 CTAs of three: 16.2 us, 64 rows, against 12.8 on mma.sync). With more
// than 64 rows, whose CTAs have an SM each, what does not fit at once costs a whole second round (2048 x 2048, 100 rows, in 16
// clusters of eight 15.3 us).
template <class Places>
bool gc_plan(int64_t rows, int64_t cols, int words, int64_t M, bool swiglu, int64_t sms, Places places, GcPlan* p) {
  p->bn = (int)((M + 15) / 16 * 16);
  p->nunits = (int)(cols / GC_UNIT);
  p->tiles = swiglu ? (rows / 2 + GC_TILE / 2 - 1) / (GC_TILE / 2) : (rows + GC_TILE - 1) / GC_TILE;
  p->CK = 0;
  for (int ck = 1; ck <= 8; ck++) {
    const int upc = (p->nunits + ck - 1) / ck;
    if (8 * p->tiles * ck > 7 * sms || upc > GC_MAX_UPC || (ck - 1) * upc >= p->nunits) continue;
    if (M > 64 && p->tiles * ck > places(ck)) continue;
    p->CK = ck, p->upc = upc;
  }
  if (!p->CK) return false;
  p->slice = (int)((M + p->CK - 1) / p->CK);  // rows of y that a CTA finishes
  for (p->nx = p->upc; p->nx >= 1; p->nx--) {  // units of activations at a time
    p->smem = 1024 + (size_t)p->nx * p->bn * 512 +
              std::max((size_t)p->upc * GC_TILE * words * 4, (size_t)p->CK * p->slice * GC_TILE * 4);
    if (p->smem <= (size_t)GC_SMEM) break;
  }
  if (!p->nx) return false;
  p->acc_cols = p->bn <= 64 ? 64 : 128;
  p->tmem_cols = p->acc_cols + 128 * p->upc <= 256 ? 256 : 512;
  p->smem = std::max<size_t>(p->smem, p->tmem_cols == 512 ? GC_SMEM_512 : p->bn > 64 ? GC_SMEM_OWN : GC_SMEM_256);
  return true;
}

// Where the kernel is ahead of gemm_skinny.cu among the products that one takes: more rows than 32 (with up to 32 the activations that
// every CTA of that kernel reads weigh less: 1024 x 2048 Q4_0, activation pass included, 24 rows 6.6 there and 6.9 us here, 37
// rows 8.2 and 7.0, 64 rows 9.7 and 7.4; 65 rows, against the kernels behind that one, 13.1 and 7.8, 128 rows 13.5 and 9.8; a
// second tile of 128 rows is slower than they are), and a K that four CTAs share, or two with a third of the SMs to spare (6144 x 1024, 64
// rows 12.4 and 8.7; 12288 x 512 in whole tiles 11.6 and 12.9, 8192 x 768 Q8_0 in 128 CTAs 11.5 and 11.8).
template <class Places>
bool gc_prefers(int64_t rows, int64_t cols, int words, int64_t M, bool swiglu, int64_t sms, Places places) {
  GcPlan p;
  if (M <= 32 || M > GC_MAX_BN || (swiglu && rows % 2) || !gc_plan(rows, cols, words, M, swiglu, sms, places, &p)) return false;
  if (M > 64) return !swiglu && p.CK >= 2 && cols >= 1536 && p.tiles <= 20;
  return p.CK >= 4 || (p.CK >= 2 && p.upc <= 2 && 3 * p.tiles * p.CK <= 2 * sms);
}

}  // namespace dyn
