// gbh_pair.cuh -- pairs of 32-bit floats for the small terms of the WENO5 interface flux.
//
// GB300 retires 2 FP64 operations per clock and SM against 128 FP32 ones, so a term that
// is small against the flux it is added to is cheaper as an unevaluated sum h + l of two
// FP32 numbers (about 48 significant bits).  The algorithms are Dekker's and Knuth's
// error-free transformations (T. J. Dekker, Numer. Math. 18 (1971); D. E. Knuth, The Art
// of Computer Programming, vol. 2, 4.2.2) with the FMA for the product's error.
//
// Every operation goes through the explicitly rounded intrinsics, so that no contraction
// or reassociation touches them and the same inputs give the same pair in every kernel.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define GBH_HD __host__ __device__ __forceinline__
#else
#include <cmath>
#include <cstring>
#define GBH_HD inline
#endif

namespace gbh {

#ifdef __CUDA_ARCH__
GBH_HD float fadd(float a, float b) {
  float r;
  asm("add.rn.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
GBH_HD float fsub(float a, float b) {
  float r;
  asm("sub.rn.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
GBH_HD float fmul(float a, float b) {
  float r;
  asm("mul.rn.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
GBH_HD float ffma(float a, float b, float c) {
  float r;
  asm("fma.rn.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
GBH_HD uint32_t f2u(float a) { return __float_as_uint(a); }
GBH_HD float u2f(uint32_t a) { return __uint_as_float(a); }
GBH_HD float rcp32(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
GBH_HD float rsqrt32(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
GBH_HD uint32_t dhi(double x) { return (uint32_t)__double2hiint(x); }
GBH_HD uint32_t dlo(double x) { return (uint32_t)__double2loint(x); }
GBH_HD double mkd(uint32_t hi, uint32_t lo) { return __hiloint2double((int)hi, (int)lo); }
GBH_HD uint32_t shl64hi(uint32_t hi, uint32_t lo, int s) { return __funnelshift_l(lo, hi, s); }
GBH_HD float u32tof(uint32_t a) { return __uint2float_rn(a); }
#else
inline float fadd(float a, float b) { return a + b; }
inline float fsub(float a, float b) { return a - b; }
inline float fmul(float a, float b) { return a * b; }
inline float ffma(float a, float b, float c) { return ::fmaf(a, b, c); }
inline uint32_t f2u(float a) { uint32_t u; ::memcpy(&u, &a, 4); return u; }
inline float u2f(uint32_t a) { float f; ::memcpy(&f, &a, 4); return f; }
inline float rcp32(float x) { return 1.0f / x; }
inline float rsqrt32(float x) { return (float)(1.0 / ::sqrt((double)x)); }
inline uint32_t dhi(double x) { uint64_t u; ::memcpy(&u, &x, 8); return (uint32_t)(u >> 32); }
inline uint32_t dlo(double x) { uint64_t u; ::memcpy(&u, &x, 8); return (uint32_t)u; }
inline double mkd(uint32_t hi, uint32_t lo) { uint64_t u = ((uint64_t)hi << 32) | lo; double d; ::memcpy(&d, &u, 8); return d; }
inline uint32_t shl64hi(uint32_t hi, uint32_t lo, int s) { return (hi << s) | (lo >> (32 - s)); }
inline float u32tof(uint32_t a) { return (float)a; }
#endif

// The value h + l.  Normalised: |l| <= ulp(h) / 2.
struct alignas(8) ff {
  float h, l;
};

// s + e = a + b exactly; fast2 for |a| >= |b| (or a == 0).
GBH_HD ff two_sum(float a, float b) {
  ff r;
  r.h = fadd(a, b);
  const float bb = fsub(r.h, a);
  r.l = fadd(fsub(a, fsub(r.h, bb)), fsub(b, bb));
  return r;
}
GBH_HD ff fast2(float a, float b) {
  ff r;
  r.h = fadd(a, b);
  r.l = fsub(b, fsub(r.h, a));
  return r;
}
GBH_HD ff neg(ff a) {
  ff r = {-a.h, -a.l};
  return r;
}
GBH_HD ff operator+(ff a, ff b) {
  const ff s = two_sum(a.h, b.h);
  return fast2(s.h, fadd(s.l, fadd(a.l, b.l)));
}
GBH_HD ff operator-(ff a, ff b) { return a + neg(b); }
GBH_HD ff operator*(ff a, ff b) {
  const float p = fmul(a.h, b.h);
  float e = ffma(a.h, b.h, -p);
  e = ffma(a.h, b.l, e);
  e = ffma(a.l, b.h, e);
  return fast2(p, e);
}
// a b for a single-precision factor, and a times a power of two.
GBH_HD ff mulf(ff a, float b) {
  const float p = fmul(a.h, b);
  const float e = ffma(a.l, b, ffma(a.h, b, -p));
  return fast2(p, e);
}
GBH_HD ff mul2(ff a, float p2) {
  ff r = {fmul(a.h, p2), fmul(a.l, p2)};
  return r;
}
GBH_HD ff sqr(ff a) {
  const float p = fmul(a.h, a.h);
  float e = ffma(a.h, a.h, -p);
  e = ffma(fadd(a.h, a.h), a.l, e);
  return fast2(p, e);
}
// 1 / x: the hardware estimate r (relative error e of some 2^-23) and r (e + e^2), the
// next two terms of 1/x = r / (1 - e).
GBH_HD ff rcp(ff x) {
  const float r = rcp32(x.h);
  const float e = ffma(-x.l, r, ffma(-x.h, r, 1.0f));
  return fast2(r, fmul(r, ffma(e, e, e)));
}
// 1 / sqrt(x) from the estimate y: y (1 + e/2 + 3 e^2 / 8), e = 1 - x y^2, with x y^2
// formed as the product of the pairs x and y^2.
GBH_HD ff rsqrt(ff x) {
  const float y = rsqrt32(x.h);
  const float q = fmul(y, y), ql = ffma(y, y, -q);
  const float p = fmul(x.h, q);
  float e = ffma(-x.h, q, p);
  e = ffma(-x.h, ql, e);
  e = ffma(-x.l, q, e);
  e = fadd(fsub(1.0f, p), e);
  return fast2(y, fmul(fmul(y, e), ffma(0.375f, e, 0.5f)));
}

// A double as a pair, and back.  The FP64 pipe also executes the conversions between
// FP32 and FP64, so both take the bits apart with integer instructions instead: the
// leading 24 significand bits become h exactly, the other 29 l (rounded to 24).  A
// magnitude below 2^-103 becomes 0, one of 2^128 or above (infinities and NaN too)
// infinity, which the range check of the caller rejects.
GBH_HD ff to_pair(double x) {
  const uint32_t H = dhi(x), L = dlo(x);
  // 2^(e - 23) of the double's exponent e as a float's bits; (e_biased - 919) << 23
  int32_t sc = (int32_t)(H & 0x7ff00000u) - (919 << 20);
  sc = sc < 0 ? 0 : sc;
  sc = sc > (255 << 20) ? (255 << 20) : sc;
  const float s = u2f(((uint32_t)sc << 3) | (H & 0x80000000u));
  const float m = u2f((shl64hi(H, L, 3) & 0x7fffffu) | 0x4b000000u);
  ff r;
  r.h = fmul(m, s);
  r.l = fmul(fmul(u32tof(L & 0x1fffffffu), 1.862645149230957e-9f), s);
  return r;
}
// The magnitude of a double as a float, rounded down (0 below 2^-126, infinity for what is
// too large or not finite).
GBH_HD float d2f_mag(double x) {
  const uint32_t H = dhi(x) & 0x7fffffffu;
  const int32_t e = (int32_t)(H & 0x7ff00000u) - (896 << 20);
  const uint32_t m = shl64hi(H, dlo(x), 3) & 0x7fffffu;
  return e <= 0 ? 0.0f : (e >= (255 << 20) ? u2f(0x7f800000u) : u2f(((uint32_t)e << 3) | m));
}
// (Denormals become 0; infinities and NaN stay what they are.)
GBH_HD double f2d(float a) {
  const uint32_t b = f2u(a), e = b & 0x7f800000u;
  const uint32_t hi = (((b >> 3) & 0x0fffffffu) + (e == 0x7f800000u ? 0x70000000u : 0x38000000u)) | (b & 0x80000000u);
  return e ? mkd(hi, b << 29) : 0.0;
}
GBH_HD double to_double(ff a) { return f2d(a.h) + f2d(a.l); }


// Constants as pairs (h the nearest float, l the rest).
GBH_HD ff ffc(double c) {
  ff r;
  r.h = (float)c;
  r.l = (float)(c - (double)r.h);
  return r;
}
// (A normalised pair: a NaN of the second word is in the first one too.)
GBH_HD bool is_finite(ff a) { return fabsf(a.h) <= 3.0e38f; }
GBH_HD ff ffabs(ff a) { return a.h < 0.0f ? neg(a) : a; }
GBH_HD ff ffmax(ff a, ff b) { return (a.h > b.h || (a.h == b.h && a.l > b.l)) ? a : b; }
GBH_HD ff ffsqrt(ff x) { return x * rsqrt(x); }

// The sum of two pairs not normalised (for a following reciprocal, product or sum).
GBH_HD ff addu(ff a, ff b) {
  ff s = two_sum(a.h, b.h);
  s.l = fadd(s.l, fadd(a.l, b.l));
  return s;
}

// Products and squares not normalised (|l| up to some 2^-22 of h), for sums of positive
// terms, reciprocals and sums of products; l l is kept where an operand may be unnormalised.
GBH_HD ff mulu(ff a, ff b) {
  ff r;
  r.h = fmul(a.h, b.h);
  r.l = ffma(a.l, b.h, ffma(a.h, b.l, ffma(a.h, b.h, -r.h)));
  return r;
}
// (both operands unnormalised)
GBH_HD ff muluu(ff a, ff b) {
  ff r;
  r.h = fmul(a.h, b.h);
  r.l = ffma(a.l, b.l, ffma(a.l, b.h, ffma(a.h, b.l, ffma(a.h, b.h, -r.h))));
  return r;
}
GBH_HD ff mulfu(ff a, float b) {
  ff r;
  r.h = fmul(a.h, b);
  r.l = ffma(a.l, b, ffma(a.h, b, -r.h));
  return r;
}
GBH_HD ff sqru(ff a) {
  ff r;
  r.h = fmul(a.h, a.h);
  r.l = ffma(fadd(a.h, a.h), a.l, ffma(a.h, a.h, -r.h));
  return r;
}
// 1 / x not normalised, and 1 / x^2.
GBH_HD ff rcpu(ff x) {
  ff r;
  r.h = rcp32(x.h);
  const float e = ffma(-x.l, r.h, ffma(-x.h, r.h, 1.0f));
  r.l = fmul(r.h, ffma(e, e, e));
  return r;
}
GBH_HD ff inv_sq(ff x) {
  const ff y = rcpu(x);
  ff r;
  r.h = fmul(y.h, y.h);
  r.l = ffma(y.l, y.l, ffma(fadd(y.h, y.h), y.l, ffma(y.h, y.h, -r.h)));
  return r;
}

// A sum of products of pairs: the leading products are added without error, the rest
// collects in the second word.
struct FAcc {
  float h, l;
};
GBH_HD FAcc acc_mul(ff a, ff b) {
  FAcc r;
  r.h = fmul(a.h, b.h);
  r.l = ffma(a.l, b.h, ffma(a.h, b.l, ffma(a.h, b.h, -r.h)));
  return r;
}
GBH_HD void acc_fma(FAcc& c, ff a, ff b) {
  const float p = fmul(a.h, b.h);
  const float e = ffma(a.l, b.h, ffma(a.h, b.l, ffma(a.h, b.h, -p)));
  const ff s = two_sum(c.h, p);
  c.h = s.h;
  c.l = fadd(c.l, fadd(s.l, e));
}
GBH_HD void acc_add(FAcc& c, ff a) {
  const ff s = two_sum(c.h, a.h);
  c.h = s.h;
  c.l = fadd(c.l, fadd(s.l, a.l));
}
GBH_HD ff acc_get(FAcc c) { return fast2(c.h, c.l); }

// ---------------------------------------------------------------------------
// WENO5 as a correction of the fourth-order central interface value.
//
// With the third differences t1, t2, t3 of the window (around the left, the central and
// the right face of the interface) and the weights (w1, w2, w3) of a side, w1+w2+w3 = 1:
//   left-biased value  = cA - (w1/3) t1 - (w3/6) t2,   cA = (-v1 + 5 v2 + 2 v3) / 6,
//   right-biased value = cB + (w1/3) t3 + (w3/6) t2,   cB = (2 v2 + 5 v3 - v4) / 6,
// where w1 weighs the sub-stencil farthest upwind and w3 the downwind one; and
//   (cA + cB)/2 = (-v1 + 7 v2 + 7 v3 - v4)/12,   cB - cA = -t2/6.
// So the mean of the sides is the central value plus, and their difference is, a
// combination of the three third differences.
// ---------------------------------------------------------------------------

// One cell's sub-stencil (differences dm to its left, dp to its right) for the places it
// takes in the pairs around it (weno5_cell_q): second difference d and 1/B^2, the central
// one times 6; bl, br: B itself (Borges' tau).
struct PRow {
  ff d, l, c, r, bl, br;
};
// SIX: with the factor 6 (the optimal weights' ratio) in c.
template <bool ALTW, bool SIX = true>
GBH_HD PRow weno_row(ff dm, ff dp, ff eps4, bool none) {
  PRow o;
  o.d = dp - dm;
  if (ALTW && none) {
    o.l = o.r = o.bl = o.br = ff{1.0f, 0.0f};
    o.c = ff{SIX ? 6.0f : 1.0f, 0.0f};
    return o;
  }
  // 3 dp - dm, dp + dm and 3 dm - dp: the first differences of weno5_cell_q
  const ff base = addu(mulu(ffc(13.0 / 3.0), sqr(o.d)), eps4);
  const ff Bl = addu(base, sqru(o.d + mul2(dp, 2.0f))), Bc = addu(base, sqru(dp + dm)),
           Br = addu(base, sqru(mul2(dm, 2.0f) - o.d));
  o.l = inv_sq(Bl);
  o.c = SIX ? mulfu(inv_sq(Bc), 6.0f) : inv_sq(Bc);
  o.r = inv_sq(Br);
  if (ALTW) {
    o.bl = Bl;
    o.br = Br;
  }
  return o;
}

enum { PW_JS = 0, PW_MAPPED = 1, PW_BORGES = 2, PW_YC = 3, PW_NONE = 4 };  // WENO_W_*

// One unnormalised weight of the mapped formulation (weno5_side_alt):
// w (c + c^2 - 3 c w + w^2) / (c^2 + w (1 - 2c)) of the Jiang-Shu weight w, a quotient of
// positive terms, so that a small weight keeps its relative precision.
GBH_HD ff mapped_weight(ff w, double c) {
  const ff num = muluu(w - ffc(3.0 * c), w) + ffc(c + c * c);
  const ff den = addu(mulu(w, ffc(1.0 - 2.0 * c)), ffc(c * c));
  return muluu(muluu(w, num), rcpu(den));
}

// Whether a sum of sub-stencils' terms is in the range in which pairs keep their precision:
// below 2^-100 its second word has none left, above 2^100 the smoothness terms are so small
// that eps, or their second words, may lie below what pairs hold.  The second word of the sum
// is tested too: a smoothness term that overflows leaves 1/B^2 = (0, NaN), which the first
// word does not show where another sub-stencil is smooth.
GBH_HD bool sum_in_range(ff S) {
  return (S.h >= 7.888609e-31f) & (S.h <= 1.2676506e30f) & (fabsf(S.l) <= S.h);  // 2^-100, 2^100; false for NaN
}

// The weights (w1, w3) of one side from the terms i1, i2, i3 (1/q of the three
// sub-stencils times 1, 6, 3), tau (4 tau of the side; Borges and Yamaleev-Carpenter).
// Returns false where the sum leaves its range.
template <bool ALTW>
GBH_HD bool side_weights(ff i1, ff i2, ff i3, ff tau, int wtype, ff& w1, ff& w3) {
  bool ok = true;
  if (ALTW && (wtype == PW_BORGES || wtype == PW_YC)) {
    // c_k (1 + T / q_k) with T = (4 tau)^2; T is off by up to 2^-149, so 1/q_k has to be in
    // range by itself
    ok = sum_in_range(addu(addu(i1, i2), i3));
    const ff T = sqr(tau);
    i1 = T * i1 + ff{1.0f, 0.0f};
    i2 = T * i2 + ff{6.0f, 0.0f};
    i3 = T * i3 + ff{3.0f, 0.0f};
  }
  const ff S = addu(addu(i1, i2), i3);
  const ff R = rcpu(S);
  w1 = muluu(i1, R);
  w3 = muluu(i3, R);
  if (ALTW && wtype == PW_MAPPED) {
    const ff m1 = mapped_weight(w1, 0.1), m2 = mapped_weight(muluu(i2, R), 0.6), m3 = mapped_weight(w3, 0.3);
    const ff n = rcpu(addu(addu(m1, m2), m3));
    w1 = muluu(m1, n);
    w3 = muluu(m3, n);
  }
  return ok & sum_in_range(S);
}

// The weights of a pair: the farthest upwind sub-stencils' doubled, the downwind ones'.
struct PWeights {
  ff l1, l3, r1, r3;  // 2 w1 and w3 of the left-biased side, of the right-biased side
};

// From the third differences t1, t2, t3 of the values the weights are formed from
// (Yamaleev-Carpenter's tau) and the sub-stencils' terms.
template <bool ALTW>
GBH_HD bool weno_pair_weights(ff t1, ff t2, ff t3, ff l1, ff c2, ff r3, ff r4, ff c3, ff l2, ff bl1, ff br3, ff br4,
                              ff bl2, int wtype, PWeights& W) {
  ff tauL = {0.0f, 0.0f}, tauR = {0.0f, 0.0f};
  if (ALTW && wtype == PW_BORGES) {
    tauL = bl1 - br3;
    tauR = br4 - bl2;
  } else if (ALTW && wtype == PW_YC) {
    tauL = mul2(sqr(t2 - t1), 4.0f);
    tauR = mul2(sqr(t3 - t2), 4.0f);
  }
  bool ok = side_weights<ALTW>(l1, c2, mulfu(r3, 3.0f), tauL, wtype, W.l1, W.l3);
  ok = side_weights<ALTW>(r4, c3, mulfu(l2, 3.0f), tauR, wtype, W.r1, W.r3) & ok;
  W.l1 = mul2(W.l1, 2.0f);
  W.r1 = mul2(W.r1, 2.0f);
  return ok;
}
// Twice the mean of the two sides less the central value, and the right value less the
// left one, times 6, of values with the third differences t1, t2, t3.
GBH_HD ff weno_sum6(const PWeights& W, ff t1, ff t2, ff t3) {
  FAcc s = acc_mul(W.r1, t3);
  acc_fma(s, W.l1, neg(t1));
  acc_fma(s, W.r3 - W.l3, t2);
  return acc_get(s);
}
GBH_HD ff weno_dif6(const PWeights& W, ff t1, ff t2, ff t3) {
  FAcc d = acc_mul(W.r1, t3);
  acc_fma(d, W.l1, t1);
  acc_fma(d, (W.r3 + W.l3) - ff{1.0f, 0.0f}, t2);
  return acc_get(d);
}
// The sum of the terms' magnitudes, which bounds the rounding of both (some 2^-47 of it),
// cancellation or not.
GBH_HD float weno_mag6(const PWeights& W, ff t1, ff t2, ff t3) {
  return ffma(fabsf(W.r1.h), fabsf(t3.h), ffma(fabsf(W.l1.h), fabsf(t1.h), fmul(fadd(W.r3.h, W.l3.h), fabsf(t2.h))));
}

// All three from the second differences d1..d4 of window cells 1..4 where weights and
// values come from the same array.
template <bool ALTW>
GBH_HD bool weno_pair_corr(ff d1, ff d2, ff d3, ff d4, ff l1, ff c2, ff r3, ff r4, ff c3, ff l2, ff bl1, ff br3,
                           ff br4, ff bl2, int wtype, ff& sum6, ff& dif6, float& mag6) {
  const ff t1 = d2 - d1, t2 = d3 - d2, t3 = d4 - d3;
  PWeights W;
  const bool ok = weno_pair_weights<ALTW>(t1, t2, t3, l1, c2, r3, r4, c3, l2, bl1, br3, br4, bl2, wtype, W);
  sum6 = weno_sum6(W, t1, t2, t3);
  dif6 = weno_dif6(W, t1, t2, t3);
  mag6 = weno_mag6(W, t1, t2, t3);
  return ok;
}

// The weights from the five differences of a window whose sub-stencils no other interface
// shares (characteristic fields), with its third differences.
template <bool ALTW>
GBH_HD bool weno_window_weights(const ff* dl, ff eps4, int wtype, PWeights& W, ff& t1, ff& t2, ff& t3) {
  ff d[4], l1, c2, l2, c3, r3, r4, bl1, bl2, br3, br4;
#pragma unroll
  for (int k = 0; k < 4; k++) d[k] = dl[k + 1] - dl[k];
  l1 = r4 = l2 = r3 = ff{1.0f, 0.0f};
  c2 = c3 = ff{6.0f, 0.0f};
  bl1 = bl2 = br3 = br4 = ff{0.0f, 0.0f};
  if (!(ALTW && wtype == PW_NONE)) {
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const ff base = addu(mulu(ffc(13.0 / 3.0), sqr(d[k])), eps4);
      if (k < 2) {
        const ff B = addu(base, sqru(d[k] + mul2(dl[k + 1], 2.0f)));
        (k == 0 ? l1 : l2) = inv_sq(B);
        (k == 0 ? bl1 : bl2) = B;
      }
      if (k == 1 || k == 2) (k == 1 ? c2 : c3) = mulfu(inv_sq(addu(base, sqru(dl[k + 1] + dl[k]))), 6.0f);
      if (k > 1) {
        const ff B = addu(base, sqru(mul2(dl[k], 2.0f) - d[k]));
        (k == 2 ? r3 : r4) = inv_sq(B);
        (k == 2 ? br3 : br4) = B;
      }
    }
  }
  t1 = d[1] - d[0];
  t2 = d[2] - d[1];
  t3 = d[3] - d[2];
  return weno_pair_weights<ALTW>(t1, t2, t3, l1, c2, r3, r4, c3, l2, bl1, br3, br4, bl2, wtype, W);
}
template <bool ALTW>
GBH_HD bool weno_window_corr(const ff* dl, ff eps4, int wtype, ff& sum6, ff& dif6, float& mag6) {
  PWeights W;
  ff t1, t2, t3;
  const bool ok = weno_window_weights<ALTW>(dl, eps4, wtype, W, t1, t2, t3);
  sum6 = weno_sum6(W, t1, t2, t3);
  dif6 = weno_dif6(W, t1, t2, t3);
  mag6 = weno_mag6(W, t1, t2, t3);
  return ok;
}
// Third differences of a window from its five differences.
GBH_HD void third_differences(const ff* dl, ff& t1, ff& t2, ff& t3) {
  const ff d1 = dl[1] - dl[0], d2 = dl[2] - dl[1], d3 = dl[3] - dl[2], d4 = dl[4] - dl[3];
  t1 = d2 - d1;
  t2 = d3 - d2;
  t3 = d4 - d3;
}

}  // namespace gbh
