// What the token-contracted GEMMs read: the two operands and how they lie in memory.
#pragma once
#include "common.cuh"

namespace gb {

struct XtyOperands {
  const void* ptr[2];      // X, Y: [samples, T, cols] bf16, or [samples, 2, T, ld] (parts == 2: values, then residuals)
  int cols[2];
  long long ld[2];         // row pitch
  int parts;
  long long part_rows;     // rows of a part in memory (parts == 2); 0: those that are read
  // Whether one TMA box may cover several 64-column blocks: the columns are a multiple of 64, or the rows are zero
  // up to the next one (`padded`, which the split layout always is).
  bool padded;
  bool blocked(int i) const { return cols[i] % 64 == 0 || (padded && ld[i] >= padded_cols(i)); }
  long long padded_cols(int i) const { return (cols[i] + 63ll) / 64 * 64; }
};

// Per-sample column sums that a GEMM pass takes along: of operand 1 (X) or 2 (Y), whose values they are (parts == 1);
// of == 0: none
struct XtyColsum {
  int of;
  float* out;
};

// Zeroes the sums of a launch's samples where several of its units add to each
inline int xty_colsum_clear(const XtyColsum& cs, int parts, int sample0, int samples, int cols, cudaStream_t st) {
  if (cs.of == 0 || parts == 1) return GHOST_OK;
  return clear_ahead(cs.out + static_cast<long long>(sample0) * cols, sizeof(float) * static_cast<size_t>(samples) * cols, st);
}

// Map of operand i for boxes of `rows_box` tokens and `blocks` 64-column blocks (both parts of a split operand)
inline int xty_operand_map(CUtensorMap* t, const XtyOperands& o, int i, long long samples, long long rows, int rows_box, int blocks) {
  if (o.parts == 2) return make_tmap_bf16_parts(t, o.ptr[i], samples, o.part_rows ? o.part_rows : rows, rows, o.ld[i], rows_box, blocks);
  if (!o.blocked(i)) return make_tmap_bf16_3d(t, o.ptr[i], samples, rows, o.cols[i], o.ld[i], rows_box);
  return make_tmap_bf16_blocks(t, o.ptr[i], samples, rows, o.padded_cols(i), o.ld[i], rows_box, blocks);
}

}  // namespace gb
