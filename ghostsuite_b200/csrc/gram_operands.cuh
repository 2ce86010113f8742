// What the Gram kernels read, and what their two translation units call of each other.
#pragma once
#include "common.cuh"

namespace gb {

// Operands of the two Grams: rows of train and validation tokens
struct GramOperands {
  const void *a_t, *a_v, *g_t, *g_v;
  long long ld_at, ld_av, ld_gt, ld_gv;
  int ka, kg;
  int parts;
  long long part_rows;     // parts == 2: rows of a part in memory
};

// Maps of the four operands: train rows in boxes of box_t, validation rows of box_v (ghost_gram.cu)
int gram_maps(CUtensorMap (&t)[4], const GramOperands& o, long long rows_t, long long rows_v, int box_t, int box_v);

// The kernel on CTA pairs (ghost_gram_pair.cu)
int launch_gram_pair(const GramOperands& o, int n_train, int n_val, long long T, int round_mode, float scale, float* M,
                     const DeviceState* ds, cudaStream_t stream);

}  // namespace gb
