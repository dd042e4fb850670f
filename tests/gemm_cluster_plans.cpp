// Plans of the cluster GEMM over many shapes: what a block takes of an SM, one line per different plan kind:
// columns, least and largest dynamic shared memory, plans seen, and whether a plan's columns hold its accumulator and units.
// With rows, matrix rows, columns and words of products behind the SM count: for each, the blocks along K that it is given, or 0.
#include <cstdio>
#include <cstdlib>
#include <map>

#include "gemm_cluster_plan.h"

int main(int argc, char** argv) {
  const long sms = argc > 1 ? atol(argv[1]) : 148;
  auto places = [&](int ck) { return (int)(sms / ck * ck); };
  if (argc > 2) {
    for (int i = 2; i + 3 < argc; i += 4) {
      const long M = atol(argv[i]), rows = atol(argv[i + 1]), cols = atol(argv[i + 2]), words = atol(argv[i + 3]);
      dyn::GcPlan p;
      printf("%d\n", dyn::gc_prefers(rows, cols, (int)words, M, false, sms, places) && dyn::gc_plan(rows, cols, (int)words, M, false, sms, places, &p) ? p.CK : 0);
    }
    return 0;
  }
  struct Kind {
    size_t lo, hi;
    long n;
    bool fits;
  };
  std::map<int, Kind> kinds;
  for (int words : {32, 36, 40, 44, 68})
    for (long cols = 256; cols <= 24 * 256; cols += 256)
      for (long rows = 1; rows <= 20000; rows += rows < 300 ? 61 : 509)
        for (long M = 33; M <= dyn::GC_MAX_BN; M++)
          for (int swiglu = 0; swiglu < 2; swiglu++) {
            dyn::GcPlan p;
            if ((swiglu && rows % 2) || !dyn::gc_plan(rows, cols, words, M, swiglu, sms, places, &p)) continue;
            Kind& k = kinds.try_emplace(p.tmem_cols, Kind{p.smem, p.smem, 0, true}).first->second;
            k.lo = std::min(k.lo, p.smem), k.hi = std::max(k.hi, p.smem), k.n++;
            k.fits &= p.acc_cols >= p.bn && p.acc_cols + 128 * p.upc <= p.tmem_cols && p.CK * p.upc >= p.nunits;
          }
  for (const auto& [cols, k] : kinds) printf("%d %zu %zu %ld %d\n", cols, k.lo, k.hi, k.n, (int)k.fits);
  return 0;
}
