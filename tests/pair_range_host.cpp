// The range guard of the float-pair WENO5 weights (gbh_pair.cuh, host build): windows whose
// smoothness terms overflow, underflow or are not finite.  A window that is accepted has to
// have finite results; a line per formulation holds how many windows were accepted and how
// many of those had a result that is not finite.  The last line holds the conversions of
// values that are not finite.
#include <cmath>
#include <cstdio>
#include <initializer_list>

#include "gbh_pair.cuh"

using namespace gbh;

int main() {
  for (int wt = 0; wt < 5; wt++) {
    long accepted = 0, wrong = 0;
    for (int e = -60; e <= 130; e++)
      for (int m = 0; m < 16; m++) {
        const double J = std::ldexp(1.0 + m / 16.0, e);
        for (int pos = 1; pos < 6; pos++)        // the first cell behind the jump
          for (int spike = 0; spike < 2; spike++)  // a step, or one cell only
            for (double base : {1.0, 0.0, 1e19, 1e-20}) {
              double v[6];
              for (int i = 0; i < 6; i++) v[i] = base + ((spike ? i == pos : i >= pos) ? J : 0.0);
              ff dl[5], s6, d6;
              float mag;
              for (int i = 0; i < 5; i++) dl[i] = to_pair(v[i + 1] - v[i]);
              const ff e4 = to_pair(4e-6);
              const bool ok = wt == 0 ? weno_window_corr<false>(dl, e4, wt, s6, d6, mag)
                                      : weno_window_corr<true>(dl, e4, wt, s6, d6, mag);
              if (!ok || !(mag <= 3.0e38f)) continue;
              accepted++;
              const double a = to_double(s6), b = to_double(d6);
              if (!std::isfinite(s6.h) || !std::isfinite(d6.h) || !std::isfinite(a) || !std::isfinite(b)) wrong++;
            }
      }
    std::printf("%d %ld %ld\n", wt, accepted, wrong);
  }
  const ff nan = {NAN, 0.0f}, inf = {INFINITY, 0.0f}, ninf = {-INFINITY, 0.0f};
  const double big = to_double(ff{3.0e38f, 0.0f});
  std::printf("conv %d\n", (int)(std::isnan(to_double(nan)) && std::isinf(to_double(inf)) && to_double(inf) > 0.0 &&
                                 std::isinf(to_double(ninf)) && to_double(ninf) < 0.0 && big == (double)3.0e38f));
  return 0;
}
