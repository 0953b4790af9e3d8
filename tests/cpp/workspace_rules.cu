// Host-only check of gemm_overlap_allowed() (csrc/kernels/gemm.h): a product that writes its workspace
// may not start in the tail of one that still reads the same memory.
#include "gemm.h"
#include <stdio.h>

using namespace lt;

static int fails = 0;
#define EXPECT(c) do { if (!(c)) { printf("line %d: %s\n", __LINE__, #c); ++fails; } } while (0)

int main() {
  for (GemmWorkspaceUse first : {GEMM_WS_NONE, GEMM_WS_SPLIT_K, GEMM_WS_PACKED})
    for (int overlap : {0, 1, 2}) {
      bool prev = false;
      // the first product, behind one that reads no workspace
      EXPECT(gemm_overlap_allowed(prev, first, overlap) == (first == GEMM_WS_PACKED ? 0 : overlap));
      const bool reads = first != GEMM_WS_NONE;
      bool p = prev;
      EXPECT(gemm_overlap_allowed(p, GEMM_WS_SPLIT_K, overlap) == (reads ? 0 : overlap));   // writes partial sums
      EXPECT(p);
      p = prev;
      EXPECT(gemm_overlap_allowed(p, GEMM_WS_NONE, overlap) == overlap);                    // writes no workspace
      EXPECT(!p);
      p = prev;
      EXPECT(gemm_overlap_allowed(p, GEMM_WS_PACKED, overlap) == 0);
      EXPECT(p);
    }
  if (fails == 0) printf("RULES_OK\n");
  return fails != 0;
}
