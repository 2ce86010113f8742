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

// Merged operands as the entry points for parts take them: A [parts, (n_train + n_val) T, ld_a], G alike.
inline GramOperands gram_operands(const void* A, const void* G, int parts, int n_train, int n_val, long long T, int d, int p, long long ld_a,
                                  long long ld_g) {
  const long long rows_t = static_cast<long long>(n_train) * T;
  const char *a = static_cast<const char*>(A), *g = static_cast<const char*>(G);
  return {a, a + rows_t * ld_a * 2, g, g + rows_t * ld_g * 2, ld_a, ld_a, ld_g, ld_g, d, p, parts, rows_t + static_cast<long long>(n_val) * T};
}

// M_out, which a kernel ahead in the stream has `cleared`, or which is cleared here
int gram_dot(const GramOperands& o, int n_train, int n_val, long long T, int round_mode, float scale, float* M_out, bool cleared, void* stream);

}  // namespace gb
