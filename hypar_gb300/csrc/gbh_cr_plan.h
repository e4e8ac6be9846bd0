// gbh_cr_plan.h -- launch shape of the compact scheme's flux pass (gbh_crweno.cu).
#pragma once

namespace gbh {

// Cells a thread of the flux pass walks along lines of N cells: `asked` where a shape was asked
// for (0: none).  By itself the pass takes short segments of at most 32, for 16 warps per SM,
// which hide the latency of its reads (64^3: two segments of 32 per line left 256 warps in
// all, 117 / 162 / 247 us per direction).
inline int cr_segment(int asked, int N, long long nlines, int sms) {
  if (asked > 0) return asked;
  const long long fill = N * nlines / (sms * 16LL * 32);
  return fill < 2 ? 2 : (fill > 32 ? 32 : (int)fill);
}

}  // namespace gbh
