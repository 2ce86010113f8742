// Per-sample column sums of one GEMM operand (the bias terms' input) taken by four extra warps of
// the per-sample GEMM kernels while the tensor core works on the same rows.
//
// The warps read the operand rows straight from global memory -- L2 hits, because the TMA producer
// is fetching the same rows for the tensor core -- instead of re-reading the shared-memory stages:
// an earlier version did that and slowed the GEMM by two thirds, its reads competing with the
// tensor core's own operand fetch.  No barrier is shared with the pipeline warps; the 128 threads
// synchronise among themselves on a named barrier.
#pragma once
#include <cuda_bf16.h>
#include <stdint.h>

namespace gb {

// Rows [t0, t1) of a sample that unit `part` of the `parts` sharing a (sample, column block) adds up: its share, so
// that a unit's column-sum warps never have more to read than its tensor-core work covers and read the rows that
// the TMA producer is fetching at that moment.  (One unit for all rows, in turn, saves the zeroed results
// and the atomics but not the time: 139.7 -> 147 us on 40 x 1024 tokens of 768 x 3072.)
struct XtyRows { long long t0, t1; };
__device__ __forceinline__ XtyRows xty_colsum_rows(int part, int parts, long long T) {
  const long long per = ((T + parts - 1) / parts + 7) / 8 * 8, t0 = part * per;
  return {t0, t0 + per < T ? t0 + per : T};
}

// Partial sums of the eight row lanes -> out[cbase ..]; not `alone`: other units add to it too (zeroed by the host)
__device__ __forceinline__ void xty_colsum_finish(const float (&a)[8], int cbase, int total_cols, float* red,
                                                  float* __restrict__ out, bool alone, int ct, int bar_id) {
  const int cv = ct & 15, rl = ct >> 4;
#pragma unroll
  for (int j = 0; j < 8; ++j) red[rl * 128 + cv * 8 + j] = a[j];
  named_bar_sync(bar_id, 128);
  float sum = 0.f;
#pragma unroll
  for (int r = 0; r < 8; ++r) sum += red[r * 128 + ct];
  if (cbase + ct < total_cols) {
    if (alone) out[cbase + ct] = sum;
    else if (sum != 0.f) atomicAdd(out + cbase + ct, sum);
  }
  named_bar_sync(bar_id, 128);
}

// Sums rows of columns [cbase, cbase + 128) of `src` (row pitch ld, 16-byte aligned, rows readable up to
// the next multiple of eight columns) into out[cbase ..].  ct = 0..127 is the thread's index among
// the column-sum warps; red is 8 * 128 floats of shared memory; up to sixteen 16-byte loads are in flight
// per thread.
__device__ __forceinline__ void xty_colsum_128(const __nv_bfloat16* src, XtyRows rows, bool alone, long long ld,
                                               int cbase, int total_cols, float* red, float* __restrict__ out, int ct, int bar_id) {
  const int cv = ct & 15, rl = ct >> 4;     // 16 column vectors x 8 row lanes
  const int c0 = cbase + cv * 8;
  float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (c0 < total_cols) {
    const __nv_bfloat16* base = src + c0;
    auto lo = [](uint32_t w) { return __uint_as_float(w << 16); };
    auto hi = [](uint32_t w) { return __uint_as_float(w & 0xffff0000u); };
    // rows are added in pairs before they join a lane's sum
    auto add4 = [&](const uint4& w0, const uint4& w1, const uint4& w2, const uint4& w3) {
      const uint32_t x0[4] = {w0.x, w0.y, w0.z, w0.w}, x1[4] = {w1.x, w1.y, w1.z, w1.w};
      const uint32_t x2[4] = {w2.x, w2.y, w2.z, w2.w}, x3[4] = {w3.x, w3.y, w3.z, w3.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        a[2 * e] += (lo(x0[e]) + lo(x1[e])) + (lo(x2[e]) + lo(x3[e]));
        a[2 * e + 1] += (hi(x0[e]) + hi(x1[e])) + (hi(x2[e]) + hi(x3[e]));
      }
    };
    const long long T = rows.t1;
    long long t = rows.t0 + rl;
    for (; t + 120 < T; t += 128) {
      uint4 w[16];
#pragma unroll
      for (int q = 0; q < 16; ++q) w[q] = *reinterpret_cast<const uint4*>(base + (t + 8 * q) * ld);
#pragma unroll
      for (int q = 0; q < 16; q += 4) add4(w[q], w[q + 1], w[q + 2], w[q + 3]);
    }
    for (; t + 24 < T; t += 32) {
      const uint4 w0 = *reinterpret_cast<const uint4*>(base + t * ld);
      const uint4 w1 = *reinterpret_cast<const uint4*>(base + (t + 8) * ld);
      const uint4 w2 = *reinterpret_cast<const uint4*>(base + (t + 16) * ld);
      const uint4 w3 = *reinterpret_cast<const uint4*>(base + (t + 24) * ld);
      add4(w0, w1, w2, w3);
    }
    for (; t < T; t += 8) {
      const uint4 w = *reinterpret_cast<const uint4*>(base + t * ld);
      const uint32_t x[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) { a[2 * e] += lo(x[e]); a[2 * e + 1] += hi(x[e]); }
    }
  }
  xty_colsum_finish(a, cbase, total_cols, red, out, alone, ct, bar_id);
}

}  // namespace gb
