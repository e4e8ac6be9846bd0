// gbh_pair_plan.h -- block shapes of the float-pair kernels (gbh_pair_flux.cuh).
#pragma once

namespace gbh {

// The block shape of one direction: XL lines of L cells each, T threads (T >= XL (L + 6)).
struct PairPlan {
  int L, XL, T;
};

// The shape that covers nlines lines of N cells with the fewest threads, at most `cap` per
// block.  Slots are lost to the six halo cells of each piece of a line, to the last piece
// of a line and to the last block of lines; along the strided directions fewer than four
// neighbouring lines read less than a 128-byte line of memory at a time, which is weighed
// as an eighth more.
// fixed: every block of the launch has `cap` threads (ensembles), so blocks are counted.
inline PairPlan pair_plan(int N, long long nlines, int dir, int cap, bool fixed = false) {
  PairPlan best = {1, 1, 32};
  double cost = 1e300;
  for (int XL = 1; XL <= 16 && XL <= nlines; XL++) {
    const int Lmax = cap / XL - 6;
    if (Lmax < 1) break;
    const int n0 = (N + Lmax - 1) / Lmax;
    for (int n = n0; n < n0 + 3; n++) {
      const int L = (N + n - 1) / n, nt = (N + L - 1) / L;
      const int T = (XL * (L + 6) + 31) / 32 * 32;
      double c = (double)((nlines + XL - 1) / XL) * nt * (fixed ? cap : T);
      if (dir > 0 && XL < 4) c *= 1.125;
      if (c < cost) {
        cost = c;
        best = {L, XL, T};
      }
    }
  }
  return best;
}

// Threads per block: large blocks lose fewer slots, small ones spread a small grid over the
// 152 SMs.  Euler2D steps with blocks of 64 / 128 / 256: 128^2 121 / 123 / 165 us, 192^2 158 /
// 157 / 181, 320^2 343 / 331 / 346, 384^2 432 / 419 / 406, 640^2 1096 / 1058 / 989.
inline int pair_cap(long long cells) { return cells >= 150000 ? 256 : (cells >= 30000 ? 128 : 64); }

// Most threads of a block: 224 in the 3-D component-wise kernels (Taylor-Green 256^3 71.1 ms per
// step against 72.2 with 256, bubble 64^3 1.93 against 1.96), 256 in the others (vortex 1024^2
// 2.25 ms against 2.45 with 224).
inline int pair_threads(bool ns3d, bool chr) { return ns3d && !chr ? 224 : 256; }

}  // namespace gbh
