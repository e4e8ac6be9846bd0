// The float-pair WENO5 correction (gbh_pair.cuh, host build) against long double, over
// random windows of every kind the kernels meet.  Prints one line per weight formulation:
// the largest error of the mean and of the difference over the magnitude of their terms
// (times 2^47), and the share of windows whose weight sums were in range.
#include <cfloat>
#include <cmath>
#include <cstdio>
#include <random>

#include "gbh_pair.cuh"

using namespace gbh;
typedef long double Q;

static void sides(const Q* v, Q eps, int wt, Q& oL, Q& oR) {
  auto side = [&](Q m0, Q m1, Q m2, Q m3, Q m4) {
    const Q b[3] = {Q(13) / 12 * (m0 - 2 * m1 + m2) * (m0 - 2 * m1 + m2) + (m0 - 4 * m1 + 3 * m2) * (m0 - 4 * m1 + 3 * m2) / 4 + eps,
                    Q(13) / 12 * (m1 - 2 * m2 + m3) * (m1 - 2 * m2 + m3) + (m1 - m3) * (m1 - m3) / 4 + eps,
                    Q(13) / 12 * (m2 - 2 * m3 + m4) * (m2 - 2 * m3 + m4) + (3 * m2 - 4 * m3 + m4) * (3 * m2 - 4 * m3 + m4) / 4 + eps};
    Q tau = 0;
    if (wt == 2) tau = b[0] - b[2];
    if (wt == 3) tau = (m0 - 4 * m1 + 6 * m2 - 4 * m3 + m4) * (m0 - 4 * m1 + 6 * m2 - 4 * m3 + m4);
    const Q c[3] = {Q(1) / 10, Q(6) / 10, Q(3) / 10};
    Q a[3], s = 0;
    for (int k = 0; k < 3; k++) {
      a[k] = wt == 4 ? c[k] : (wt == 2 || wt == 3) ? c[k] * (1 + tau * tau / (b[k] * b[k])) : c[k] / (b[k] * b[k]);
      s += a[k];
    }
    for (int k = 0; k < 3; k++) a[k] /= s;
    if (wt == 1) {
      s = 0;
      for (int k = 0; k < 3; k++) {
        a[k] = a[k] * (c[k] + c[k] * c[k] - 3 * c[k] * a[k] + a[k] * a[k]) / (c[k] * c[k] + a[k] * (1 - 2 * c[k]));
        s += a[k];
      }
      for (int k = 0; k < 3; k++) a[k] /= s;
    }
    return (a[0] * (2 * m0 - 7 * m1 + 11 * m2) + a[1] * (-m1 + 5 * m2 + 2 * m3) + a[2] * (2 * m2 + 5 * m3 - m4)) / 6;
  };
  oL = side(v[0], v[1], v[2], v[3], v[4]);
  oR = side(v[5], v[4], v[3], v[2], v[1]);
}

int main() {
  std::mt19937_64 g(7);
  std::uniform_real_distribution<double> U(-1, 1);
  for (int wt = 0; wt < 5; wt++) {
    double worst_s = 0, worst_d = 0;
    long n = 0, in = 0;
    for (int it = 0; it < 20000; it++) {
      double v[6];
      const int kind = it % 5;
      const double ph = 3 * U(g), A = 0.3 * (1 + 0.5 * U(g)), base = 1 + 0.2 * U(g), J = U(g);
      const double h = kind == 0 ? 0.01 : 0.3, sc = kind == 4 ? 2.5e5 : 1.0;
      const int pos = (int)(3 + 2.9 * U(g));
      for (int i = 0; i < 6; i++) {
        v[i] = base + A * std::sin(ph + h * i);
        if (kind == 2) v[i] = base + (i >= pos ? J : 0.0);
        if (kind == 3) v[i] = base + J * U(g);
        v[i] *= sc;
      }
      Q q[6], oL, oR;
      for (int i = 0; i < 6; i++) q[i] = v[i];
      sides(q, 1e-6, wt, oL, oR);
      ff dl[5], s6, d6;
      float mag;
      for (int i = 0; i < 5; i++) dl[i] = to_pair(v[i + 1] - v[i]);
      const ff e4 = to_pair(4e-6);
      const bool ok = wt == 0 ? weno_window_corr<false>(dl, e4, wt, s6, d6, mag) : weno_window_corr<true>(dl, e4, wt, s6, d6, mag);
      n++;
      if (!ok) continue;
      in++;
      const Q cen = (-q[1] + 7 * q[2] + 7 * q[3] - q[4]) / 12;
      Q t = 0;  // the rounding of the FP64 differences the pairs start from
      for (int i = 0; i < 6; i++) t = std::max(t, std::fabs(q[i]));
      const Q scale = Q(mag) + Q(64) * t * DBL_EPSILON * Q(140737488355328.0) / 64;
      worst_s = std::max(worst_s, (double)(std::fabs(Q(to_double(s6)) - 6 * (oL + oR - 2 * cen)) / scale * Q(140737488355328.0)));
      worst_d = std::max(worst_d, (double)(std::fabs(Q(to_double(d6)) - 6 * (oR - oL)) / scale * Q(140737488355328.0)));
    }
    std::printf("%d %.3f %.3f %.4f\n", wt, worst_s, worst_d, (double)in / n);
  }
  // conversions: exact to 48 bits, zero and the ends of the range
  double worst = 0;
  for (int it = 0; it < 100000; it++) {
    const double x = std::ldexp(1 + 0.5 * (1 + U(g)), (int)(90 * U(g))) * (U(g) < 0 ? -1 : 1);
    worst = std::max(worst, std::fabs(to_double(to_pair(x)) - x) / std::fabs(x) * 281474976710656.0);
  }
  const bool ends = to_pair(0.0).h == 0.0f && to_double(to_pair(-0.0)) == 0.0 && to_pair(1e-40).h == 0.0f &&
                    std::isinf(to_pair(1e39).h) && std::isinf(to_pair(INFINITY).h) && !std::isfinite(to_pair(NAN).h);
  std::printf("conv %.3f %d\n", worst, (int)ends);
  return 0;
}
