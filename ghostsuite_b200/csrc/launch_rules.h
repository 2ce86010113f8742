// Rules by which the host picks a path or a launch shape from sizes alone: plain C++, for the library and for the torch binding.
#pragma once
#include <algorithm>

namespace gb {

// Whether bf16 rows of a GradProj call that TMA cannot read are copied, padded, instead of being brought through the kernel's loader
// warps.  A copy is a launch and two passes over them; what the loaders add is about half a microsecond per 64 columns of a CTA's
// chain.  Loaders and copies, us: 26 x 471 tokens of 9408 + 795 109 and 62 (only the 795 columns are copied); 10 x 30 of
// 6912 + 2579 19.2 and 12.1; 28 x 5 of 3957 + 9063 44.8 and 21.2; 14 x 1894 of 1007 + 1088 51.7 and 54; 32 x 3000 of 1001 + 2003 217 and 369.
inline bool gradproj_copies(long long B, long long T, long long n_r, long long n_c, bool ready_r, bool ready_c, int sm_count) {
  if ((ready_r && ready_c) || B <= 0 || T <= 0) return false;      // nothing to copy; an empty call is the kernel's to refuse
  const long long units = B * ((T + 127) / 128), sms = std::max(1, sm_count);
  const double stages = (n_r + 63) / 64 + (n_c + 63) / 64;
  const double chain = 2 * units > sms ? stages * ((units + sms - 1) / sms) : stages / std::min(8ll, sms / units);
  const double bytes = 2. * B * T * ((ready_r ? 0 : n_r) + (ready_c ? 0 : n_c));
  return 0.45 * chain > 4.0 + 2. * bytes / 4.5e6;
}

// Split-K factor of a train-gradient pass with the shortest critical path, in units of one row block of one tile: ceil(units /
// workers) rounds of (row blocks per split + a fixed cost per unit for the accumulator hand-over and the epilogue: `add_cost` with red.add
// into the workspace, a quarter of it with plain stores).  Splitting also pays for zeroing the fp32 workspace and for the
// scaling pass: two launches (5 us) and ten bytes per weight element at 5 TB/s; one split stores the result itself.
// `block_us` is the time of a row block while a tile's loads are bound by their latency: 0.65 us on the CTA pairs, 0.35 on single CTAs,
// whose blocks hold half the rows, 0.5 there of operands in two parts.  (With one time for both kernels splits came too soon on the
// single CTAs: 3000 rows of 1600 x 1200 27.0 us in two, 23.3 in one, 2048 of 1152 x 1152 19.9 and 17.2.)
// bf16 results, us, splits by the costs of an epilogue that stored a row a lane and half the time a block, and by these: 4096 rows of 128 x 128
// 32.8 and 13.3, 768 x 768 29.9 and 22.2, 1600 x 1200 36.9 and 34.8, 8192 rows of it 61 and 48, of 3072 x 768 55 and 48.
// The tensor core's accumulator truncates, so the error grows with the rows one split covers.  A bf16
// result does not show it; a float32 result does (4096 rows of 768 x 768, bf16 operands: 4.2e-6 off the
// 64-bit result in one split, 4.5e-7 in ten), so there the merge is not counted against splitting, and a higher add_cost
// stands for it, which keeps large results in one split.
inline int pick_k_splits(long long tiles, int workers, int kb, double block_us, int add_cost, double weight_elems, bool f32_result) {
  int splits = 1;
  double best = static_cast<double>((tiles + workers - 1) / workers) * (kb + (f32_result ? add_cost : add_cost / 4));
  const double merge = f32_result ? 0. : (5.0 + weight_elems * 10.0 / 5e6) / block_us;
  for (int s = 2; s <= 64 && s <= kb; ++s) {
    const double cost = static_cast<double>((tiles * s + workers - 1) / workers) * ((kb + s - 1) / s + add_cost) + merge;
    if (cost < best) { best = cost; splits = s; }
  }
  return splits;
}

}  // namespace gb
