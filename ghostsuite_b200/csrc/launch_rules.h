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

}  // namespace gb
