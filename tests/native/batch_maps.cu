// Host harness of the batched engine's block maps (tests/test_batch_maps.py).  No kernel is
// launched and no CUDA call made.
#include "../../include/pycfd_b200.h"
#include "../../pycfd_b200/csrc/batch.cuh"

using namespace pcfd;

extern "C" {

// Column tiles a structure of spn problems has, or -1 where the map cannot name them.
int bm_tail_cols(int spn) {
  const int cts = (spn + kTailBN - 1) / kTailBN;
  return cts > kTailMaxCols ? -1 : cts;
}
int bm_tail_tile(int row_tile, int col_tile) { return b_tail_tile(row_tile, col_tile); }
int bm_tail_row(int tile) { return b_tail_row(tile); }
int bm_tail_col(int tile) { return b_tail_col(tile); }

// Problems per block of the pattern products: of a coarse level, or of level 0.
int bm_pat_group(int single, int level0, int nsm, int n, const int* probs, const int* blocks) {
  const int half = single ? 1 : 2;
  const std::vector<int> p(probs, probs + n), b(blocks, blocks + n);
  return level0 ? b_pick_group(kUpGroup / half, kUpGroup, kUpMaxGroups, nsm, p, b)
                : b_pick_group(kPatGroup / half, kPatGroup, kPatMaxGroups, nsm, p, b);
}
int bm_max_groups(int level0) { return level0 ? kUpMaxGroups : kPatMaxGroups; }

}  // extern "C"
