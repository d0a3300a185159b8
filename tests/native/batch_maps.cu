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

}  // extern "C"
