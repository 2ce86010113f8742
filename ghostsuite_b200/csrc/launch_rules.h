// Rules by which the host picks a path or a launch shape from sizes alone: plain C++, for the library and for the torch binding.
#pragma once
#include <algorithm>

namespace gb {

// Whether bf16 rows of a GradProj call that TMA cannot read are copied, padded, instead of being brought through the kernel's loader
// warps.  A copy is a launch and two passes over them; what the loaders add is about half a microsecond per 64 columns of a CTA's
// chain.  Loaders and copies, us: 26 x 471 tokens of 9408 + 795 109 and 62 (only the 795 columns are copied); 10 x 30 of
// 6912 + 2579 19.2 and 12.1; 28 x 5 of 3957 + 9063 44.8 and 21.2; 32 x 3000 of 1001 + 2003 217 and 369; 14 x 1894 of 1007 + 1088, where the two
// meet, 51.1 and 51.3.  A copy counts as 4 us, more than it takes on the GPU, for the launch on the host: hook of 44 x 211 of 384 + 79 13.3
// and 15.5, its kernels 13.6 and 11.3.
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

// CTAs that share a tile of a Gram: as many as make its chain of K steps shortest while all clusters are resident, against what the
// cluster costs, 4 us, in steps, rounded up for those that share the L2 (us alone and split, bf16 and float32: 8 + 2 x 128 of 512 + 512 13.3 and 15.4,
// 23.5 and 23.3; 1024 + 1024 17.4 and 17.5, 33.8 and 25.6; 768 + 3072 23.5 and 19.8, 54 and 33; 40 + 4 x 64, 40 tiles,
// of 768 + 3072 26.5 and 21.9, 65 and 46, of 4096 + 4096 44 and 31, 122 and 77).
// `resident(r)`: clusters of r CTAs that the device holds at a time.
template <typename Resident>
int gram_cluster(long long tiles, int k_steps, int sms, Resident&& resident) {
  constexpr double kSplitCost = 10.;
  int best = 1;
  double cost = k_steps;
  for (int r = 2; r <= 8 && r <= k_steps; ++r) {
    const double c = (k_steps + r - 1) / r + kSplitCost;
    if (c < cost && tiles * r <= sms && tiles <= resident(r)) { best = r; cost = c; }
  }
  return best;
}

// Blocks that share a pair of groups of samples in the kernel of few-row layers.  A step of 1024 columns takes a block 1.1 us, and the
// pairs are few where the rows are long (4 + 12 samples of one token, float32 108 -> 27072: 36.9 us in two blocks, 14.5 in sixteen; 8 + 2 of 20000 -> 10 35.9 and 14.3;
// 2 + 2 x 8 of 4096 -> 512 17.0 and 14.5).  A tile costs a cluster's barrier, 1.5 us, on top (8 + 2 x 16 of 2048 -> 1024, eight
// tiles a pair: 38.9, 41 shared).  Where the gradient's blocks take longer than the chain nothing is gained, and
// they come up slower in clusters (2 + 1 of 768 -> 50000 71 and 77; 16 + 4 of 4095 -> 4097 47 and 53).
inline int small_cluster(long long gram, long long tiles, long long wgrad, long long rows, long long d, long long p, int sms) {
  const double others = static_cast<double>((wgrad + 2 * sms - 1) / (2 * sms)) * (2.0 + 0.045 * rows);
  int best = 1;
  double cost = 1.1 * ((d + 1023) / 1024 + (p + 1023) / 1024) * tiles;
  for (int r = 2; r <= 8 && gram * r <= 2ll * sms && cost > others; r *= 2) {
    const double c = (1.1 * ((d + 1024 * r - 1) / (1024 * r) + (p + 1024 * r - 1) / (1024 * r)) + 1.5) * tiles;
    if (c < cost) { best = r; cost = c; }
  }
  return best;
}

}  // namespace gb
