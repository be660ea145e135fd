// Host-side check of the blocked FP64 LU kernel's plan and launch shape
// (alglin_b200/csrc/bcr_lub_plan.cuh): for every shape it takes, the panel block and
// the kernel's static arrays fit in shared memory, every row has a thread, and a
// level never starts more CTAs than there are slabs, however many clusters the
// device may hold at once.
#include <cstdio>

#include "bcr_common.cuh"

namespace bcr {
#include "bcr_lub_plan.cuh"
}

int main() {
  using namespace bcr;
  int checked = 0, failures = 0;
  for (int n = 1; n <= 128; ++n)
    for (int nr = 0; 2 * n + nr <= LUB_ROWS_MAX + 1; ++nr) {
      const int rows = 2 * n + nr;
      LubPlan p = lub_plan(rows, n);
      bool ok = (p.threads != 0) == (rows <= LUB_ROWS_MAX);
      if (p.threads) {
        ok &= rows <= p.threads && (p.threads == 256 || p.threads == 512);
        ok &= p.bw % 8 == 0 && p.bw <= p.depth && p.depth <= LUB_W && p.depth % 16 == 0 && p.depth >= 32;
        ok &= p.smem == lub_smem(rows, p.depth) && p.smem + 16 * 1024 <= 227 * 1024;
        ok &= p.threads == 512 || 2 * (p.smem + 7 * 1024) <= 228 * 1024;
        // residency from none to more clusters than today's registers allow
        for (int most : {0, 16, 74, 148, 222, 296, 4096})
          for (long np : {1L, 2L, 3L, 16L, 37L, 74L, 75L, 148L, 149L, 222L, 296L, 297L, 100000L})
            for (int slots : {148, 296}) {
              for (int i = 0; i < 3; ++i) p.clusters[i] = most >> i;
              const LubGrid g = lub_grid(p, np, 2 * n + 8, slots);
              ok &= g.ctas >= 1 && (long)g.ctas <= slots && g.ctas % g.slices == 0;
              ok &= g.slices == 1 || (long)g.ctas == np * g.slices;
              ok &= g.slices >= 1 && g.slices <= LUB_SLICES_MAX && (g.slices & (g.slices - 1)) == 0;
            }
      }
      if (!ok) {
        std::printf("plan check failed: n=%d nr=%d\n", n, nr);
        ++failures;
      }
      ++checked;
    }
  std::printf("%d shapes checked, %d failures\n", checked, failures);
  return failures ? 1 : 0;
}
