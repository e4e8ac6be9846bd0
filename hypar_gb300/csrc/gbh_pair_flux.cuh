// gbh_pair_flux.cuh -- the fused hyperbolic kernel with the small terms in float pairs.
//
// HyPar's interface flux (ReconstructHyperbolic, HyperbolicFunction.c:167-222: WENO5 of
// fL, fR, uL, uR and the upwind scheme) is written as
//   F_{j+1/2} = (-f_{j-1} + 7 f_j + 7 f_{j+1} - f_{j+2}) / 12 + G_{j+1/2},
// the fourth-order central value and a correction G: the nonlinear weights' deviation from
// it and the upwind dissipation.  Both parts of G are combinations of third differences
// (gbh_pair.cuh), small against the flux wherever the solution is resolved.  The central
// part (and the cells' fluxes and primitives) is computed in FP64, G in pairs of FP32
// numbers, whose arithmetic has 64 times the FP64 pipe's throughput on GB300.
//
// What bounds the error: a pair carries 48 bits, the chain from the differences to G loses
// two or three of them, so G is off by some 2^-46 of the magnitude of its terms.  The
// interface takes the FP64 evaluation (iface_flux) instead where
//   - its terms exceed a bound times its flux scale (rho lam, rho lam^2, rho lam H with
//     lam = |u_n| + a; pair_bound, dissipation terms at the dissipation's own speed),
//   - what the characteristic projections add up exceeds one (PROJ_BOUND): a field may cancel
//     out of large differences, their rounding does not,
//   - a scale of the states or the fluxes leaves the range 2^-44 .. 2^100 (scales_in_range), a
//     weight's sum leaves its own, or anything is not finite:
// shocks, contacts, under-resolved fields, odd units.  The decision uses the interface's own
// window only, so every kernel that evaluates an interface takes the same one and neighbouring
// blocks agree on the flux between them.
#pragma once

#include "gbh_pair.cuh"

namespace gbh {

// Eigen-system of a Roe average in pairs (Eig in gbh_device.cuh).
struct PEig {
  ff vel[3], un, a, ek, H, hac, rs, gi, lamn;  // gi = (gamma-1)/a^2
};

// Bounds of an interface's terms (12 x their share of its flux scale) and of its projections'.
// Set so that a right-hand side is no further from one in extended precision than that of
// the FP64 kernels: over waves of 6 to 100 cells and noise of 0.1 to 8 %, root mean square in
// units of 2^-53 of the flux scale over the spacing, 1-D 0.22-0.63 (FP64 kernels 0.27-0.63),
// 2-D 0.20-0.51 (0.21-0.51; at worst 3 % more, 0.263 for 0.256), 3-D component-wise 0.23-0.40 (0.44-0.57; there 2^-7 is enough),
// 3-D characteristic 0.31-0.60 (0.45-0.73).  With 2^-7 and without the projections' bound a
// wave of 6 cells was 0.67 off for 0.37, one of 24 cells (characteristic) 0.45 for 0.24.
// Time: Euler2D ensemble 16.9 -> 19.0 ms, the other workloads within 5 %.
__host__ __device__ constexpr float pair_bound(int model, bool chr) {
  return 12.0f * (model == MODEL_NS3D ? (chr ? 0.001953125f : 0.0078125f) : 0.0009765625f);  // 2^-9, 2^-7, 2^-10
}
constexpr float PROJ_BOUND = 1.0f;  // 1-D and 2-D (3-D needs none)

// Whether an interface's scales (density, speed, enthalpy) are such that pairs hold its terms:
// to_pair drops what lies below 2^-103, which has to be below 2^-53 of the states and the
// fluxes by a margin (2^-44 leaves 2^-6 of it; kap: gravity's factor of the dissipation, on
// the differences of the modified solution), products of the largest must not overflow, and
// the eigenvectors' 1/(2a), 1/a^2 need second words above 2^-149.  False for NaN.
__device__ __forceinline__ bool scales_in_range(float rho, float lam, float H, float kap = 1.0f) {
  constexpr float LO = 5.684342e-14f, HI = 1.2676506e30f;  // 2^-44, 2^100
  const float lo = LO * fmaxf(kap, 1.0f), s0 = rho * lam, uE = rho * H, sm = s0 * lam, sE = s0 * H;
  return (rho >= lo) & (s0 >= lo) & (uE >= lo) & (sm >= LO) & (sE >= LO) & (rho <= HI) & (s0 <= HI) & (uE <= HI) &
         (sm <= HI) & (sE <= HI) & (lam >= 9.094947e-13f) & (lam <= 1.0995116e12f);  // 2^-40, 2^40
}

// The same for gravity's source, rt per unit difference of the hydrostatic pressure field.
__device__ __forceinline__ bool source_in_range(float rt, float lam, float sm, float sE) {
  return (rt * 5.684342e-14f <= sm) & (rt * lam * 5.684342e-14f <= sE);
}

// Per-cell ingredients in pairs: sqrt(rho), velocity, enthalpy, wave speed.
template <int M>
struct PCell {
  ff t, vel[3], H, c;
};

struct PParams {
  ff gm1, gamma, eps4;
};

template <int M, int DIR>
__device__ __forceinline__ void peig_finish(PEig& E, ff rho, const PParams& q) {
  constexpr int ND = ModelTraits<M>::ND;
  FAcc v2 = acc_mul(E.vel[0], E.vel[0]);
#pragma unroll
  for (int k = 1; k < ND; k++) acc_fma(v2, E.vel[k], E.vel[k]);
  E.ek = mul2(acc_get(v2), 0.5f);
  const ff a2 = q.gm1 * (E.H - E.ek);
  const ff ia = rsqrt(a2);
  E.a = a2 * ia;
  const ff ia2 = sqr(ia);
  E.un = E.vel[DIR];
  E.hac = mul2(ia2, 0.5f);
  E.rs = ff{1.0f, 0.0f};
  if (M == MODEL_EULER1D) {  // hac = 1/(rho a), rs = rho/(2a)
    E.hac = rcp(rho) * ia;
    E.rs = mul2(rho * ia, 0.5f);
  }
  E.gi = q.gm1 * ia2;
}

// Roe average of two cells (or states) given by their ingredients.
template <int M, int DIR>
__device__ __forceinline__ PEig peig(const PCell<M>& L, const PCell<M>& R, const PParams& q) {
  constexpr int ND = ModelTraits<M>::ND;
  PEig E;
  const ff th = R.t * rcp(L.t + R.t);  // weight of the right state
#pragma unroll
  for (int k = 0; k < ND; k++) E.vel[k] = L.vel[k] + th * (R.vel[k] - L.vel[k]);
  E.H = L.H + th * (R.H - L.H);
  peig_finish<M, DIR>(E, L.t * R.t, q);
  return E;
}

// Ingredients of a conserved state (c: its sound speed).
template <int M>
__device__ __forceinline__ PCell<M> pcell(const ff* u, const PParams& q, bool want_c) {
  constexpr int ND = ModelTraits<M>::ND, NV = ModelTraits<M>::NV;
  PCell<M> s;
  const ff rinv = rcp(u[0]);
  s.t = u[0] * rsqrt(u[0]);
#pragma unroll
  for (int k = 0; k < ND; k++) s.vel[k] = u[1 + k] * rinv;
  FAcc m = acc_mul(u[1], s.vel[0]);
#pragma unroll
  for (int k = 1; k < ND; k++) acc_fma(m, u[1 + k], s.vel[k]);
  const ff P = q.gm1 * (u[NV - 1] - mul2(acc_get(m), 0.5f));
  s.H = (u[NV - 1] + P) * rinv;
  s.c = ff{0.0f, 0.0f};
  if (want_c) {
    const ff c2 = q.gamma * (P * rinv);
    s.c = c2 * rsqrt(c2);
  }
  return s;
}

// Roe average of two conserved states in one pass, with neither 1/rho nor the velocities
// of the states (roe_eig_cons in gbh_device.cuh).
template <int M, int DIR>
__device__ __forceinline__ PEig peig_cons(const ff* a, const ff* b, const PParams& q) {
  constexpr int ND = ModelTraits<M>::ND, NV = ModelTraits<M>::NV;
  const ff ra = rsqrt(a[0]), rb = rsqrt(b[0]);
  const ff ta = a[0] * ra, tb = b[0] * rb;
  const ff inv = rcp(addu(ta, tb));
  FAcc qa, qb;
  PEig E;
#pragma unroll
  for (int k = 0; k < ND; k++) {
    const ff wa = a[1 + k] * ra, wb = b[1 + k] * rb;
    if (k == 0) {
      qa = acc_mul(wa, wa);
      qb = acc_mul(wb, wb);
    } else {
      acc_fma(qa, wa, wa);
      acc_fma(qb, wb, wb);
    }
    E.vel[k] = (wa + wb) * inv;
  }
  // e + P = e + (gamma-1) (e - |m|^2/(2 rho))
  const ff Ha = a[NV - 1] + mulu(q.gm1, a[NV - 1] - mul2(acc_get(qa), 0.5f));
  const ff Hb = b[NV - 1] + mulu(q.gm1, b[NV - 1] - mul2(acc_get(qb), 0.5f));
  E.H = (mulu(Ha, ra) + mulu(Hb, rb)) * inv;
  peig_finish<M, DIR>(E, E.H, q);  // (the density serves Euler1D only, which averages cells)
  return E;
}

// R diag(c0, c1, c2, ..., c2) L x in the eigen-system E, fields as in projL (0: u_n - a,
// 1: u_n + a, the rest u_n): since R L = I this is c2 x + (c0 - c2) w0 r0 + (c1 - c2) w1 r1.
template <int M, int DIR>
__device__ __forceinline__ void pdissip(const PEig& E, const PParams& q, const ff* x, ff c0, ff c1, ff c2, ff* y) {
  constexpr int ND = ModelTraits<M>::ND, NV = ModelTraits<M>::NV;
  FAcc sa = acc_mul(E.ek, x[0]);
#pragma unroll
  for (int k = 0; k < ND; k++) acc_fma(sa, neg(E.vel[k]), x[1 + k]);
  acc_add(sa, x[NV - 1]);
  const ff h2 = mul2(E.gi, 0.5f);  // (gamma-1)/(2 a^2)
  const ff s = h2 * acc_get(sa);
  // t/(2 a^2) = (u_n x_0 - x_n)/(2a), and 1/(2a) = a (gamma-1)/(2a^2) / (gamma-1)
  const ff th = E.lamn * (E.un * x[0] - x[1 + DIR]);
  const ff p0 = (c0 - c2) * (s + th), p1 = (c1 - c2) * (s - th);
  const ff sum = p0 + p1, dif = E.a * (p1 - p0);
  FAcc r = acc_mul(c2, x[0]);
  acc_add(r, sum);
  y[0] = acc_get(r);
#pragma unroll
  for (int k = 0; k < ND; k++) {
    r = acc_mul(c2, x[1 + k]);
    acc_fma(r, E.vel[k], sum);
    if (k == DIR) acc_add(r, dif);
    y[1 + k] = acc_get(r);
  }
  r = acc_mul(c2, x[NV - 1]);
  acc_fma(r, E.H, sum);
  acc_fma(r, E.un, dif);
  y[NV - 1] = acc_get(r);
}

// 1/(2a), which pdissip's acoustic strengths need.
__device__ __forceinline__ void peig_upwind(PEig& E, const PParams&) { E.lamn = mul2(rcp(E.a), 0.5f); }

template <int M, int DIR>
__device__ __forceinline__ void pprojL(const PEig& E, const PParams& q, const ff* x, ff* w) {
  constexpr int ND = ModelTraits<M>::ND, NV = ModelTraits<M>::NV;
  FAcc sa = acc_mul(E.ek, x[0]);
#pragma unroll
  for (int k = 0; k < ND; k++) acc_fma(sa, neg(E.vel[k]), x[1 + k]);
  acc_add(sa, x[NV - 1]);
  const ff s = acc_get(sa);
  const ff gs = (q.gm1 * E.hac) * s, th = (E.a * E.hac) * (E.un * x[0] - x[1 + DIR]);
  w[0] = gs + th;
  w[1] = gs - th;
  w[2] = x[0] - E.gi * s;
  int j = 3;
#pragma unroll
  for (int k = 0; k < ND; k++)
    if (k != DIR) w[j++] = E.vel[k] * x[0] - x[1 + k];
}

template <int M, int DIR>
__device__ __forceinline__ void pprojR(const PEig& E, const ff* w, ff* y) {
  constexpr int ND = ModelTraits<M>::ND, NV = ModelTraits<M>::NV;
  ff Wm = w[0], Wp = w[1];
  if (M == MODEL_EULER1D) {
    Wm = Wm * E.rs;
    Wp = Wp * E.rs;
  }
  const ff sa = Wm + Wp, da = E.a * (Wp - Wm);
  const ff y0 = sa + w[2];
  FAcc yE = acc_mul(E.H, sa);
  acc_fma(yE, E.un, da);
  acc_fma(yE, E.ek, w[2]);
  int j = 3;
#pragma unroll
  for (int k = 0; k < ND; k++) {
    FAcc r = acc_mul(E.vel[k], y0);
    if (k == DIR) {
      acc_add(r, da);
    } else {
      acc_add(r, neg(w[j]));
      acc_fma(yE, neg(E.vel[k]), w[j]);
      j++;
    }
    y[1 + k] = acc_get(r);
  }
  y[0] = y0;
  y[NV - 1] = acc_get(yE);
}

__device__ __forceinline__ ff pharten(ff lam) {
  ff d = ffabs(lam);
  if (d.h < 0.000001f) d = mulf(sqr(d) + ffc(0.000001 * 0.000001), 500000.0f);
  return d;
}

// The reconstructed states' mean central value + us6/12 of component v, from the cell's
// value, its right difference and the second differences of the two cells.
__device__ __forceinline__ ff pmean(ff u2, ff dr, ff d2, ff d3, ff us6) {
  const ff tw = ffc(1.0 / 12.0);
  return u2 + (mul2(dr, 0.5f) + mulu(tw, us6 - (d2 + d3)));
}

// Coefficients of one field for LLF / RF: dissipation alpha, or the side taken (sg).
template <int UPW>
__device__ __forceinline__ void pfield(ff l, ff c, ff r, ff& al, float& sg) {
  al = ffmax(ffmax(ffabs(l), ffabs(c)), ffabs(r));
  sg = 0.0f;
  if (UPW == UPW_RF) {
    if (l.h > 0.0f && c.h > 0.0f && r.h > 0.0f) sg = 1.0f;
    else if (l.h < 0.0f && c.h < 0.0f && r.h < 0.0f) sg = -1.0f;
    if (sg != 0.0f) al = ff{0.0f, 0.0f};
  }
}

// G of one interface times 12 from the conserved sums and differences of the
// reconstructions (fs6 = 6 (fL + fR - 2 central), fd6 = 6 (fR - fL), ud6 = 6 (uR - uL)),
// mean states um where the scheme averages the reconstructed states, and the cells'
// ingredients.  lam, rho, H: the interface's scales; alm: the largest dissipation speed, which
// may exceed lam by far (the entropy fix, Euler1D's Rusanov speed, gravity).  kappa: gravity's
// factor of the dissipation.
template <int M, int UPW, int DIR>
__device__ __forceinline__ void pupwind(const ff* fs6, const ff* fd6, const ff* ud6, const ff* um, const PEig& Ecc,
                                        const PCell<M>& cl, const PCell<M>& cr, const PParams& q, ff* g12, float& lam,
                                        float& rho, float& Hs, float& alm, const ff* kappa = nullptr) {
  constexpr int NV = ModelTraits<M>::NV, ND = ModelTraits<M>::ND;
  constexpr bool STATES = (UPW == UPW_ROE && M == MODEL_EULER2D) ||
                          ((UPW == UPW_LLF || UPW == UPW_RF) && M != MODEL_EULER1D);
  PEig E;
  PCell<M> sL, sR;
  if (STATES) {
    const ff tw = ffc(1.0 / 12.0);
    ff a[NV], b[NV];
#pragma unroll
    for (int v = 0; v < NV; v++) {
      const ff h = mulu(tw, ud6[v]);
      a[v] = um[v] - h;
      b[v] = um[v] + h;
    }
    if (UPW == UPW_ROE) {
      E = peig_cons<M, DIR>(a, b, q);
    } else {
      sL = pcell<M>(a, q, true);
      sR = pcell<M>(b, q, true);
      E = peig<M, DIR>(sL, sR, q);
    }
    rho = um[0].h;
  } else {
    E = Ecc;
    sL = cl;
    sR = cr;
    rho = cl.t.h * cr.t.h;
  }
  lam = fadd(fabsf(E.un.h), E.a.h);
  Hs = E.H.h;
  if (UPW == UPW_RUS) {
    const ff avg = (M == MODEL_EULER1D ? sqr(E.a) : E.a) + ffabs(E.un);
    ff al = ffmax(ffmax(cl.c, cr.c), avg);
    if (kappa) al = al * *kappa;
    alm = al.h;
#pragma unroll
    for (int v = 0; v < NV; v++) g12[v] = fs6[v] - al * ud6[v];
    return;
  }
  peig_upwind(E, q);
  ff y[NV];
  if (UPW == UPW_ROE) {
    ff c0 = E.un - E.a, c1 = E.un + E.a, c2 = E.un;
    if (M == MODEL_EULER1D) {
      c0 = ffabs(c0);
      c1 = ffabs(c1);
      c2 = ffabs(c2);
    } else {
      c0 = pharten(c0);
      c1 = pharten(c1);
      c2 = pharten(c2);
    }
    if (kappa) {  // Euler1D with gravity
      c0 = c0 * *kappa;
      c1 = c1 * *kappa;
      c2 = c2 * *kappa;
    }
    alm = fmaxf(c0.h, c1.h);
    pdissip<M, DIR>(E, q, ud6, c0, c1, c2, y);
#pragma unroll
    for (int v = 0; v < NV; v++) g12[v] = fs6[v] - y[v];
    return;
  }
  ff al[3];
  float sg[3];
  pfield<UPW>(sL.vel[DIR] - sL.c, E.un - E.a, sR.vel[DIR] - sR.c, al[0], sg[0]);
  pfield<UPW>(sL.vel[DIR] + sL.c, E.un + E.a, sR.vel[DIR] + sR.c, al[1], sg[1]);
  pfield<UPW>(sL.vel[DIR], E.un, sR.vel[DIR], al[2], sg[2]);
  if (kappa) {
#pragma unroll
    for (int k = 0; k < 3; k++) al[k] = al[k] * *kappa;
  }
  alm = fmaxf(al[0].h, fmaxf(al[1].h, al[2].h));
  if (UPW == UPW_RF) alm = fmaxf(alm, lam);  // fields taken from one side count f's terms twice
  pdissip<M, DIR>(E, q, ud6, al[0], al[1], al[2], y);
#pragma unroll
  for (int v = 0; v < NV; v++) g12[v] = fs6[v] - y[v];
  if (UPW == UPW_RF && (sg[0] != 0.0f || sg[1] != 0.0f || sg[2] != 0.0f)) {
    // fields taken from one side: (fL - fR)/2 more, or less, than the mean
    pdissip<M, DIR>(E, q, fd6, ff{sg[0], 0.0f}, ff{sg[1], 0.0f}, ff{sg[2], 0.0f}, y);
#pragma unroll
    for (int v = 0; v < NV; v++) g12[v] = g12[v] - y[v];
  }
  (void)ND;
}

// The FP64 evaluation of one interface by its own thread (gravity, 3-D characteristic): its
// flux less the left cell's, written to G[v S]; with gravity (sgf, sgg: the hydrostatic
// fields) also the source function's interface values as corrections of its central value,
// to Gs.  Window: cells i-2 .. i+3 of the line with
// base point pb (states from memory), own cell = slot w (fluxes in shared memory).
template <int M, bool CHAR, int UPW, int DIR, bool ALTW, bool GRAV>
__device__ __forceinline__ void iface_fp64(const double* __restrict__ U, long long pb, int i, const DevGeom& geo,
                                           const double* sf, const double* sgf, const double* sgg, int S, int w,
                                           const PhysParams& pp, bool src_dir, double* G, double* Gs) {
  constexpr int NV = ModelTraits<M>::NV;
  double wu[6][NV], wf[6][NV], wuc[6], wgf[6], wgg[6], fI[NV], SI[NV];
  CellAux<M> ax[6];
#pragma unroll
  for (int p = 0; p < 6; p++) {
    const double* src = U + (pb + (long long)fold_index(i - 2 + p, geo.dim[DIR], geo.bclo[DIR], geo.bchi[DIR]) *
                                      geo.stride[DIR]) * NV;
#pragma unroll
    for (int v = 0; v < NV; v++) {
      wu[p][v] = src[v];
      wf[p][v] = sf[v * S + w - 2 + p];
    }
    const Prim<M> q = to_prim<M>(wu[p], pp);
    if (GRAV) {
      wgf[p] = sgf[w - 2 + p];
      wgg[p] = sgg[w - 2 + p];
      wuc[p] = modified_energy<M>(q, wu[p][NV - 1], wgf[p], wgg[p], pp);
    } else {
      wuc[p] = ufunc_energy<M>(q, pp, wu[p][NV - 1]);
    }
    if (p == 2 || p == 3) {
      ax[p].rs = roe_side<M>(q);
      if (UPW == UPW_RUS) ax[p].c = rusanov_speed<M, DIR>(q, pp);
      else if (M == MODEL_EULER1D && UPW != UPW_ROE) ax[p].c = sound_speed<M>(q, pp);
    }
  }
  StageEpi ep;
  ep.tape = nullptr;
  iface_flux<M, CHAR, UPW, DIR, ALTW, GRAV, false>(wu, wf, wuc, wgf, wgg, ax, pp, ep, 4.0 * pp.eps, src_dir, 0, fI, SI);
#pragma unroll
  for (int v = 0; v < NV; v++) G[v * S] = GRAV ? fI[v] - wf[2][v] : fI[v];
  if (GRAV && src_dir) {
    const double d1 = wgg[2] - wgg[1], d2 = wgg[3] - wgg[2], d3 = wgg[4] - wgg[3];
    const double c = fma(6.0, d2, d1 - d3) * (1.0 / 12.0);
    Gs[0] = (SI[1 + DIR] - wgg[2]) - c;
    Gs[S] = (SI[NV - 1] - wgg[2]) - c;
  }
}

// The FP64 evaluation of a block's flagged interfaces by all its threads (COOP): few
// interfaces lie side by side at a shock, and one thread's chain of some 700 dependent FP64
// operations takes 20 microseconds, which launches of one or two waves of blocks wait for
// (shock-entropy line of 20001: 591 -> 437 us for 15 launches; Riemann problem 601x403:
// 2030 -> 1680 us for 12).  With gravity and in the 3-D characteristic form each thread
// evaluates its own interface (iface_fp64).  A task is one side of one reconstruction
// (component-wise) or one field's pair of sides (characteristic); its values go to scr, 4 NV per interface: the pair of
// quantity 2 v + (0: f, 1: u) at 2 (2 v + h).  Then one thread per interface upwinds.
// Everything is relative to the interface's left cell, as in iface_flux.
template <int M, bool CHAR>
struct Fp64Tasks {
  static constexpr int NV = ModelTraits<M>::NV, N = CHAR ? 2 * NV : 4 * NV;
};

// State of cell i of the line with base point pb.
template <int M, int DIR>
__device__ __forceinline__ void line_state(const double* __restrict__ U, long long pb, int i, const DevGeom& geo,
                                           double* u) {
  constexpr int NV = ModelTraits<M>::NV;
  const double* src =
      U + (pb + (long long)fold_index(i, geo.dim[DIR], geo.bclo[DIR], geo.bchi[DIR]) * geo.stride[DIR]) * NV;
#pragma unroll
  for (int v = 0; v < NV; v++) u[v] = src[v];
}

template <int M, int UPW, int DIR>
__device__ __forceinline__ CellAux<M> cell_aux(const double* u, const PhysParams& pp) {
  const Prim<M> q = to_prim<M>(u, pp);
  CellAux<M> a;
  a.rs = roe_side<M>(q);
  a.c = 0.0;
  if (UPW == UPW_RUS) a.c = rusanov_speed<M, DIR>(q, pp);
  else if (M == MODEL_EULER1D && UPW != UPW_ROE) a.c = sound_speed<M>(q, pp);
  return a;
}

template <int M, bool CHAR, int UPW, int DIR, bool ALTW>
__device__ __forceinline__ void fp64_task(const double* __restrict__ U, long long pb, int i, const DevGeom& geo,
                                          const double* sf, int S, int w, int task, const PhysParams& pp,
                                          double* scr) {
  constexpr int NV = ModelTraits<M>::NV;
  const double eps4 = 4.0 * pp.eps;
  if (!CHAR) {
    const int v = task >> 2, isu = (task >> 1) & 1, right = task & 1;
    double x[6], m[5];
#pragma unroll
    for (int p = 0; p < 6; p++) {
      const int c = i - 2 + p;
      const double uv = U[(pb + (long long)fold_index(c, geo.dim[DIR], geo.bclo[DIR], geo.bchi[DIR]) * geo.stride[DIR]) *
                              NV + v];
      x[p] = isu ? uv : sf[v * S + w - 2 + p];
    }
#pragma unroll
    for (int p = 0; p < 5; p++) m[p] = (right ? x[5 - p] : x[p]) - x[2];
    scr[task] = weno5_one_side<ALTW>(m, eps4, pp.wtype);
  } else {
    const int v = task >> 1, isu = task & 1;
    double u[NV], u2[NV];
    line_state<M, DIR>(U, pb, i, geo, u2);
    line_state<M, DIR>(U, pb, i + 1, geo, u);
    const Eig E = roe_eig<M, DIR>(roe_side<M>(to_prim<M>(u2, pp)), roe_side<M>(to_prim<M>(u, pp)), pp);
    double x[6];
#pragma unroll
    for (int p = 0; p < 6; p++) {
      if (p == 2) {
        x[p] = 0.0;
        continue;
      }
      double d[NV], y[NV];
      line_state<M, DIR>(U, pb, i - 2 + p, geo, u);
#pragma unroll
      for (int e = 0; e < NV; e++) d[e] = isu ? u[e] - u2[e] : sf[e * S + w - 2 + p] - sf[e * S + w];
      projL<M, DIR>(E, pp, d, y);
      x[p] = y[0];
#pragma unroll
      for (int e = 1; e < NV; e++) x[p] = v == e ? y[e] : x[p];
    }
    double oL, oR;
    wpair<ALTW, true>(x, x, eps4, pp.wtype, oL, oR);
    scr[2 * task] = oL;
    scr[2 * task + 1] = oR;
  }
}

// The same for every field of one quantity (characteristic): a block with many flagged
// interfaces takes these, which project a cell once instead of once per field (half the FP64
// operations; noise of 20 % on 512^2, Euler2D: 7.1 -> 4.8 ms per step).  The operations on a
// value are the same, and its bits.
template <int M, int DIR, bool ALTW>
__device__ __forceinline__ void fp64_fields(const double* su, const double* sf, int S, int w, int isu,
                                            const PhysParams& pp, double* scr) {
  constexpr int NV = ModelTraits<M>::NV;
  double u2[NV], u3[NV], x[NV][6];
#pragma unroll
  for (int v = 0; v < NV; v++) {
    u2[v] = su[v * S + w];
    u3[v] = su[v * S + w + 1];
  }
  const Eig E = roe_eig<M, DIR>(roe_side<M>(to_prim<M>(u2, pp)), roe_side<M>(to_prim<M>(u3, pp)), pp);
  const double* q = isu ? su : sf;
#pragma unroll
  for (int p = 0; p < 6; p++) {
    double d[NV], y[NV];
#pragma unroll
    for (int e = 0; e < NV; e++) d[e] = q[e * S + w - 2 + p] - q[e * S + w];
    if (p != 2) projL<M, DIR>(E, pp, d, y);
#pragma unroll
    for (int v = 0; v < NV; v++) x[v][p] = p == 2 ? 0.0 : y[v];
  }
#pragma unroll
  for (int v = 0; v < NV; v++) {
    double oL, oR;
    wpair<ALTW, true>(x[v], x[v], 4.0 * pp.eps, pp.wtype, oL, oR);
    scr[4 * v + 2 * isu] = oL;
    scr[4 * v + 2 * isu + 1] = oR;
  }
}

template <int M, bool CHAR, int UPW, int DIR>
__device__ __forceinline__ void fp64_upwind(const double* __restrict__ U, long long pb, int i, const DevGeom& geo,
                                            const double* sf, int S, int w, const PhysParams& pp, const double* scr,
                                            double* G) {
  constexpr int NV = ModelTraits<M>::NV;
  double fL[NV], fR[NV], uL[NV], uR[NV], u2[NV], u3[NV], f2[NV], fI[NV];
#pragma unroll
  for (int v = 0; v < NV; v++) {
    fL[v] = scr[4 * v];
    fR[v] = scr[4 * v + 1];
    uL[v] = scr[4 * v + 2];
    uR[v] = scr[4 * v + 3];
    f2[v] = sf[v * S + w];
  }
  line_state<M, DIR>(U, pb, i, geo, u2);
  line_state<M, DIR>(U, pb, i + 1, geo, u3);
  const CellAux<M> cl = cell_aux<M, UPW, DIR>(u2, pp), cr = cell_aux<M, UPW, DIR>(u3, pp);
  Eig E;
  if (NeedCC<M, CHAR, UPW>::value) E = roe_eig<M, DIR>(cl.rs, cr.rs, pp);
  if (CHAR) upwind_char<M, UPW, DIR>(fL, fR, uL, uR, E, cl, cr, pp, fI, 1.0, u2, f2);
  else upwind_iface<M, false, UPW, DIR>(fL, fR, uL, uR, E, cl, cr, pp, fI, 1.0, u2, f2);
#pragma unroll
  for (int v = 0; v < NV; v++) G[v * S] = fI[v];
}

// The fourth-order central value of the interface to the right of slot f[0], less f[0].
__device__ __forceinline__ double central_rel(const double* f) {
  const double d1 = f[0] - f[-1], d2 = f[1] - f[0], d3 = f[2] - f[1];
  return fma(6.0, d2, d1 - d3) * (1.0 / 12.0);
}

// stage_epilogue of NB values at once: all reads are issued before the first write, so
// that their latencies overlap.
template <int NB>
__device__ __forceinline__ void stage_epilogue_batch(const StageEpi& ep, double* __restrict__ H, const long long* off,
                                                     const double* h, const bool* on) {
  const bool finish = ep.last && ep.mode != EPI_HYP, rk = finish && ep.mode != EPI_RHS;
  double x[NB], par[NB], u[NB], a[NB], p[NB][4];
#pragma unroll
  for (int k = 0; k < NB; k++) {
    if (!on[k]) continue;
    x[k] = ep.first ? 0.0 : H[off[k]];
    par[k] = (finish && ep.par) ? ep.par[off[k]] : 0.0;
    u[k] = (rk && ep.need_u) ? ep.u[off[k]] : 0.0;
    a[k] = (rk && ep.stage != 0) ? ep.acc[off[k]] : u[k];
#pragma unroll
    for (int t = 1; t < 4; t++)
      p[k][t] = (rk && t > ep.stage && t < ep.nstages && ep.ca[t] != 0.0 && ep.touched[t]) ? ep.P[t][off[k]] : u[k];
  }
#pragma unroll
  for (int k = 0; k < NB; k++) {
    if (!on[k]) continue;
    const double hyp = ep.first ? h[k] : x[k] + h[k];
    if (!finish) {
      H[off[k]] = hyp;
      continue;
    }
    const double kv = par[k] - hyp;
    if (!rk) {
      ep.rhs[off[k]] = kv;
      continue;
    }
    const double av = fma(ep.cb, kv, a[k]);
    if (ep.stage == ep.nstages - 1) ep.uout[off[k]] = av;
    else ep.acc[off[k]] = av;
#pragma unroll
    for (int t = 1; t < 4; t++)
      if (t > ep.stage && t < ep.nstages && ep.ca[t] != 0.0) ep.P[t][off[k]] = fma(ep.ca[t], kv, p[k][t]);
  }
}

// Shared memory of a block of T threads (slots S = T + 4), in 8-byte words per slot:
//   f (doubles);
//   the right differences of f and u (pairs; with gravity also of the modified solution
//   and of g); component-wise, a component's two rows take its results once its
//   sub-stencils are done;
//   the cells' ingredients;
//   u (doubles) and, component-wise, the sub-stencils of one component of f and u, which
//   take u's place unless the mean states are still formed from it;
//   characteristic: the fields' results; mean states and RF's differences where needed;
//   with gravity the hydrostatic fields.
template <int M, bool CHAR, int UPW, bool ALTW, bool GRAV>
struct PairLayout {
  static constexpr int NV = ModelTraits<M>::NV, ND = ModelTraits<M>::ND;
  static constexpr bool CC = NeedCC<M, CHAR, UPW>::value;
  static constexpr bool NEEDC = UPW == UPW_RUS || (M == MODEL_EULER1D && UPW != UPW_ROE);
  static constexpr bool STATES = (UPW == UPW_ROE && M == MODEL_EULER2D) ||
                                 ((UPW == UPW_LLF || UPW == UPW_RF) && M != MODEL_EULER1D);
  static constexpr int NA = (CC ? ND + 2 : 0) + (NEEDC ? 1 : 0);
  static constexpr int NR = ALTW ? 6 : 4;  // pairs of a sub-stencil row
  static constexpr int NDIF = 2 * NV + (GRAV ? NV + 1 : 0);
  static constexpr bool KEEP_U = CHAR || STATES;
  static constexpr int NROW = CHAR ? 0 : 2 * NR;
  static constexpr int NU = KEEP_U ? NV + NROW : (NV > NROW ? NV : NROW);
  static constexpr int NRES = (CHAR ? 2 * NV : 0) + (STATES ? NV : 0) + (UPW == UPW_RF ? NV : 0);
  static constexpr int WORDS = NV + NDIF + NA + NU + NRES + (GRAV ? 2 : 0);
  static size_t bytes(int T) { return (size_t)WORDS * (T + 4) * 8; }
};

// One block: XL neighbouring grid lines times L cells of each, LL = L + 6 slots per line,
// one thread per slot.  A thread owns a cell and the interface to its right.  sm is not
// __restrict__: the barriers order other threads' accesses to it, and a pointer that is
// said to have no alias lets the compiler move its loads and stores across them.
template <int M, bool CHAR, int UPW, int DIR, bool ALTW, bool GRAV = false>
__device__ __forceinline__ void pair_body(const double* __restrict__ U, double* __restrict__ H,
                                          const double* __restrict__ dxinv, const DevGeom& G, const PhysParams& pp,
                                          const StageEpi& ep, long long ntrans, int L, int XL, long long blk,
                                          double* sm) {
  using LY = PairLayout<M, CHAR, UPW, ALTW, GRAV>;
  constexpr int NV = LY::NV, ND = LY::ND, NR = LY::NR;
  constexpr bool CC = LY::CC, NEEDC = LY::NEEDC, STATES = LY::STATES;
  // a block evaluates its flagged interfaces together, else each thread its own
  constexpr bool COOP = !GRAV && !(M == MODEL_NS3D && CHAR);
  constexpr float BOUND = pair_bound(M, CHAR);
  constexpr bool PROJ = M != MODEL_NS3D;
  const int T = blockDim.x, S = T + 4, t = threadIdx.x;
  double* sf = sm;
  ff* sd = (ff*)(sf + NV * S);  // rows 0..NV-1: f, NV..2NV-1: u, then the modified solution and g
  ff* sa = sd + LY::NDIF * S;
  double* su = (double*)(sa + LY::NA * S);
  ff* sr = (ff*)su + (LY::KEEP_U ? NV * S : 0);  // rows of f's component, then of u's
  ff* sx = (ff*)su + LY::NU * S;                 // characteristic: 2 NV results; mean states; RF's differences
  ff* sum = sx + (CHAR ? 2 * NV * S : 0);
  ff* sfd = sum + (STATES ? NV * S : 0);
  double* sgf = (double*)(sx + LY::NRES * S);
  double* sgg = sgf + S;
  const bool grav_dir = GRAV && pp.grav[DIR] != 0.0;
  const bool src_dir = grav_dir && (ep.mode != EPI_HYP || ep.with_source);
  const int N = G.dim[DIR], LL = L + 6;
  const long long sdir = G.stride[DIR];
  const int lo = G.bclo[DIR], hi = G.bchi[DIR];
  const unsigned ngrp = (unsigned)((ntrans + XL - 1) / XL), tile = (unsigned)blk / ngrp;
  const long long l0 = (long long)((unsigned)blk - tile * ngrp) * XL;
  const int a0 = (int)tile * L;
  const int nl = (int)(ntrans - l0 < XL ? ntrans - l0 : XL), Lc = N - a0 < L ? N - a0 : L;
  auto line_base = [&](long long tr) {
    long long pb = (long long)G.g * sdir;
#pragma unroll
    for (int e = 0; e < ND; e++) {
      if (e == DIR) continue;
      const int ie = (int)(tr % G.dim[e]);
      tr /= G.dim[e];
      pb += (long long)(ie + G.g) * G.stride[e];
    }
    return pb;
  };
  int* cnt = (int*)(sf + T + 3);  // interfaces that leave the pairs' bound (a padding slot)
  if (t == 0) *cnt = 0;
  // Cells a0-3 .. a0+Lc+2 of the lines, consecutive threads on consecutive doubles: along a
  // line for DIR 0, else across the lines.
  if (DIR == 0) {
    for (int l = 0; l < nl; l++) {
      const long long pb = line_base(l0 + l);
#pragma unroll 4
      for (int i = t; i < (Lc + 6) * NV; i += T) {
        const int c = i / NV, v = i - c * NV;
        su[v * S + l * LL + c] = U[(pb + (long long)fold_index(a0 - 3 + c, N, lo, hi) * sdir) * NV + v];
      }
    }
  } else {
    const int R = nl * NV, c0 = t / R, r = t - c0 * R, l = r / NV, v = r - l * NV, step = T / R;
    if (c0 < step) {
      const long long pb = line_base(l0 + l);
#pragma unroll 4
      for (int c = c0; c < Lc + 6; c += step)
        su[v * S + l * LL + c] = U[(pb + (long long)fold_index(a0 - 3 + c, N, lo, hi) * sdir) * NV + v];
    }
  }
  __syncthreads();
  const int line = t / LL, q = t - line * LL, w = t;
  double term[2] = {0.0, 0.0};  // gravity's source per unit difference of g: momentum, energy
  // Every thread computes, also those whose slot holds no cell or no interface (their
  // values, from whatever the slots hold, are not used): the warps stay converged from
  // barrier to barrier, and the slots' padding keeps all indexes inside the arrays.
  PParams P;
  P.gm1 = to_pair(pp.gm1);
  P.gamma = to_pair(pp.gamma);
  P.eps4 = to_pair(4.0 * pp.eps);
  {
    double uu[NV], fv[NV];
#pragma unroll
    for (int v = 0; v < NV; v++) uu[v] = su[v * S + w];
    const Prim<M> pr = to_prim<M>(uu, pp);
    cell_flux<M, DIR>(pr, fv);
    fv[0] = uu[1 + DIR];
#pragma unroll
    for (int v = 0; v < NV; v++) sf[v * S + w] = fv[v];
    if (GRAV) {
      const int i = a0 - 3 + q;
      double f = 1.0, g = 1.0;
      if (line < nl && i <= N + 2) {
        const long long pt = line_base(l0 + line) + (long long)fold_index(i, N, lo, hi) * sdir;
        f = pp.gf[pt];
        g = pp.gg[pt];
      }
      sgf[w] = f;
      sgg[w] = g;
      // the modified solution, in the place its differences take
      double* sc = (double*)(sd + 2 * NV * S);
#pragma unroll
      for (int v = 0; v < NV - 1; v++) sc[v * S + w] = uu[v] * f;
      sc[(NV - 1) * S + w] = modified_energy<M>(pr, uu[NV - 1], f, g, pp);
      // [0, rho RT e_DIR, rho RT v_DIR] f (NavierStokes3DSource.c:92-97)
      const double rRT = pr.rho * pp.RT;
      term[0] = rRT * f;
      term[1] = (rRT * (pr.rho == 0.0 ? 0.0 : uu[1 + DIR] * pr.rinv)) * f;
    }
    if (CC) {
      const ff r = to_pair(uu[0]);
      sa[w] = r * rsqrt(r);
#pragma unroll
      for (int k = 0; k < ND; k++) sa[(1 + k) * S + w] = to_pair(pr.vel[k]);
      sa[(1 + ND) * S + w] = to_pair((pr.e + pr.P) * pr.rinv);
    }
    if (NEEDC) {
      const ff c2 = P.gamma * to_pair(pr.P * pr.rinv);
      ff c = (UPW == UPW_RUS && M == MODEL_EULER1D) ? c2 : c2 * rsqrt(c2);
      if (UPW == UPW_RUS) c = c + ffabs(to_pair(pr.vel[DIR]));
      sa[(CC ? ND + 2 : 0) * S + w] = c;
    }
  }
  __syncthreads();
  if (GRAV) {
    const double* sc = (const double*)(sd + 2 * NV * S);
    ff dc[NV];
#pragma unroll
    for (int v = 0; v < NV; v++) dc[v] = to_pair(sc[v * S + w + 1] - sc[v * S + w]);
    __syncthreads();
#pragma unroll
    for (int v = 0; v < NV; v++) sd[(2 * NV + v) * S + w] = dc[v];
    sd[3 * NV * S + w] = to_pair(sgg[w + 1] - sgg[w]);
  }
#pragma unroll
  for (int v = 0; v < NV; v++) {
    sd[v * S + w] = to_pair(sf[v * S + w + 1] - sf[v * S + w]);
    sd[(NV + v) * S + w] = to_pair(su[v * S + w + 1] - su[v * S + w]);
  }
  __syncthreads();
  const bool iface = line < nl && q >= 2 && q <= Lc + 2;
  const bool own = line < nl && q >= 3 && q <= Lc + 2;
  bool ok = true;
  ff g12[NV];
  float lam, rho, Hs, alm;
  auto cell_of = [&](int x) {
    PCell<M> c;
    c.t = c.H = c.c = ff{1.0f, 0.0f};
#pragma unroll
    for (int k = 0; k < 3; k++) c.vel[k] = ff{0.0f, 0.0f};
    if (CC) {
      c.t = sa[x];
#pragma unroll
      for (int k = 0; k < ND; k++) c.vel[k] = sa[(1 + k) * S + x];
      c.H = sa[(1 + ND) * S + x];
    }
    if (NEEDC) c.c = sa[(CC ? ND + 2 : 0) * S + x];
    return c;
  };
  // gravity: the source function's corrections (momentum, energy), the dissipation's factor
  ff gsm = {0.0f, 0.0f}, gse = {0.0f, 0.0f}, tg1, tg2, tg3, kap;
  if (GRAV) {
    const ff* dd = sd + 3 * NV * S + w;
    const ff dl[5] = {dd[-2], dd[-1], dd[0], dd[1], dd[2]};
    third_differences(dl, tg1, tg2, tg3);
    kap = to_pair(fmax(sgg[w], sgg[w + 1]));
  }
  if (!CHAR) {
    // 6 x the terms of density, the momenta (largest), energy: of f, of u
    float m0 = 0.0f, mm = 0.0f, mE = 0.0f, u0 = 0.0f, um = 0.0f, uE = 0.0f, magsm = 0.0f, magse = 0.0f;
#pragma unroll 1
    for (int v = 0; v < NV; v++) {
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const ff* dd = sd + (h * NV + v) * S;
        const PRow r = weno_row<ALTW>(dd[w - 1], dd[w], P.eps4, pp.wtype == PW_NONE);
        ff* o = sr + h * NR * S + w;
        o[0] = r.d;
        o[S] = r.l;
        o[2 * S] = r.c;
        o[3 * S] = r.r;
        if (ALTW) {
          o[4 * S] = r.bl;
          o[5 * S] = r.br;
        }
      }
      __syncthreads();
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const ff* o = sr + h * NR * S + w;
        ff bl1, br3, br4, bl2;
        bl1 = br3 = br4 = bl2 = ff{0.0f, 0.0f};
        if (ALTW) {
          bl1 = o[4 * S - 1];
          bl2 = o[4 * S];
          br3 = o[5 * S + 1];
          br4 = o[5 * S + 2];
        }
        const ff d2 = o[0], d3 = o[1];
        ff t1 = d2 - o[-1], t2 = d3 - d2, t3 = o[2] - d3;
        PWeights W;
        ok = weno_pair_weights<ALTW>(t1, t2, t3, o[S - 1], o[2 * S], o[3 * S + 1], o[3 * S + 2], o[2 * S + 1], o[S],
                                     bl1, br3, br4, bl2, pp.wtype, W) & ok;
        ff* res = sd + (h * NV + v) * S + w;  // this component's differences are read no more
        float mag;
        if (h == 0) {
          mag = weno_mag6(W, t1, t2, t3);
          ok = ok & (mag <= 3.0e38f);  // (the maxima below drop a NaN)
          if (UPW == UPW_RF) sfd[v * S + w] = weno_dif6(W, t1, t2, t3);
          if (GRAV && (v == 1 + DIR || v == NV - 1)) {
            const ff g = weno_sum6(W, tg1, tg2, tg3);
            const float mg = weno_mag6(W, tg1, tg2, tg3);
            if (v == NV - 1) {
              gse = g;
              magse = mg;
            } else {
              gsm = g;
              magsm = mg;
            }
          }
          *res = weno_sum6(W, t1, t2, t3);
          m0 = v == 0 ? mag : m0;
          mm = (v > 0 && v < NV - 1) ? fmaxf(mm, mag) : mm;
          mE = v == NV - 1 ? mag : mE;
        } else {
          if (STATES) sum[v * S + w] = pmean(to_pair(su[v * S + w]), *res, d2, d3, weno_sum6(W, t1, t2, t3));
          if (GRAV) {  // weights of u, values of the modified solution
            const ff* dd = sd + (2 * NV + v) * S + w;
            const ff dl[5] = {dd[-2], dd[-1], dd[0], dd[1], dd[2]};
            third_differences(dl, t1, t2, t3);
          }
          mag = weno_mag6(W, t1, t2, t3);
          ok = ok & (mag <= 3.0e38f);
          *res = weno_dif6(W, t1, t2, t3);
          u0 = v == 0 ? mag : u0;
          um = (v > 0 && v < NV - 1) ? fmaxf(um, mag) : um;
          uE = v == NV - 1 ? mag : uE;
        }
      }
      __syncthreads();
    }
    ff fs6[NV], fd6[NV], ud6[NV], us[NV];
#pragma unroll
    for (int v = 0; v < NV; v++) {
      fs6[v] = sd[v * S + w];
      ud6[v] = sd[(NV + v) * S + w];
      if (UPW == UPW_RF) fd6[v] = sfd[v * S + w];
      if (STATES) us[v] = sum[v * S + w];
    }
    PCell<M> cl, cr;
    PEig Ecc;
    if (CC || NEEDC) {
      cl = cell_of(w);
      cr = cell_of(w + 1);
    }
    if (CC) Ecc = peig<M, DIR>(cl, cr, P);
    pupwind<M, UPW, DIR>(fs6, fd6, ud6, us, Ecc, cl, cr, P, g12, lam, rho, Hs, alm, GRAV ? &kap : nullptr);
    const float s0 = rho * lam, sm1 = s0 * lam, sE = s0 * Hs;
    ok = ok & (ffma(alm, u0, m0) <= BOUND * s0) & (ffma(alm, um, mm) <= BOUND * sm1) &
         (ffma(alm, uE, mE) <= BOUND * sE);
    ok = ok & scales_in_range(rho, lam, Hs, GRAV ? kap.h : 1.0f);
    if (grav_dir) {  // asked for or not, so that both evaluations take the same form
      const float rt = (float)term[0];
      ok = ok & (magsm * rt <= BOUND * sm1) & (magse * rt * lam <= BOUND * sE) & source_in_range(rt, lam, sm1, sE);
    }
  } else {
    PCell<M> cl = cell_of(w), cr = cell_of(w + 1);
    PEig Ecc = peig<M, DIR>(cl, cr, P);
    ff lcol[NV], sch[NV];  // L (e_{1+DIR} + e_E): the source function's projection per unit of g
    if (GRAV) {
      ff ev[NV];
#pragma unroll
      for (int v = 0; v < NV; v++) ev[v] = ff{(v == 1 + DIR || v == NV - 1) ? 1.0f : 0.0f, 0.0f};
      pprojL<M, DIR>(Ecc, P, ev, lcol);
    }
    // Per unit of g, the source function's terms; 6 x the terms of fields 0-2, of the shear
    // fields, of f, of u (the largest of each).
    float ma = 0.0f, ms = 0.0f, ua = 0.0f, us = 0.0f, magg = 0.0f, pf = 0.0f, pu = 0.0f;
    const float sc01 = M == MODEL_EULER1D ? Ecc.rs.h : 1.0f;
    const ff gh = P.gm1 * Ecc.hac, ah = Ecc.a * Ecc.hac;
    // The magnitude of what a face's projections add up, in densities: a field may cancel out of
    // it (an entropy jump leaves no sound), its rounding does not.
    const float i2a = ah.h * sc01;
    auto terms = [&](const ff* y) {
      float s = ffma(Ecc.ek.h, fabsf(y[0].h), fabsf(y[(NV - 1) * S].h)), m = 0.0f;
#pragma unroll
      for (int e = 0; e < ND; e++) {
        const float ve = fabsf(Ecc.vel[e].h), ye = fabsf(y[(1 + e) * S].h);
        s = ffma(ve, ye, s);
        m = fadd(ffma(ve, fabsf(y[0].h), ye), m);
      }
      return ffma(i2a, m, ffma(Ecc.gi.h, s, fabsf(y[0].h)));
    };
#pragma unroll 1
    for (int h = 0; h < 2; h++) {
      // the projections' common parts at the five faces: s/(gamma-1) times (gamma-1) hac, t hac
      const ff* x = sd + h * NV * S + w - 2;
      const ff* xc = sd + 2 * NV * S + w - 2;  // gravity: the modified solution
      ff gs[5], th[5], gc[GRAV ? 5 : 1], tc[GRAV ? 5 : 1];
      auto parts = [&](const ff* y, ff& a, ff& b) {
        FAcc acc = acc_mul(Ecc.ek, y[0]);
#pragma unroll
        for (int e = 0; e < ND; e++) acc_fma(acc, neg(Ecc.vel[e]), y[(1 + e) * S]);
        acc_add(acc, y[(NV - 1) * S]);
        a = acc_get(acc);
        b = mulu(ah, mulu(Ecc.un, y[0]) - y[(1 + DIR) * S]);
      };
      // field v of the difference at one face, from its common parts
      auto field = [&](const ff* y, int v, ff a, ff b) {
        if (v < 2) return mulu(gh, a) + (v == 0 ? b : neg(b));
        if (v == 2) return y[0] - mulu(Ecc.gi, a);
        const int e = (v - 3) + ((v - 3) >= DIR ? 1 : 0);  // the shear fields: transverse directions ascending
        return mulu(e == 0 ? Ecc.vel[0] : (e == 1 || ND < 3 ? Ecc.vel[ND > 1 ? 1 : 0] : Ecc.vel[ND - 1]), y[0]) -
               y[(1 + e) * S];
      };
#pragma unroll
      for (int k = 0; k < 5; k++) {
        parts(x + k, gs[k], th[k]);
        if (GRAV) {
          if (h) parts(xc + k, gc[GRAV ? k : 0], tc[GRAV ? k : 0]);
        }
      }
      float p1 = 0.0f, p2 = 0.0f, p3 = 0.0f;  // of the third differences
      if (PROJ) {
        const ff* y = GRAV && h ? xc : x;
        const float q0 = terms(y), q1 = terms(y + 1), q2 = terms(y + 2), q3 = terms(y + 3), q4 = terms(y + 4);
        p1 = q0 + 2.0f * q1 + q2;
        p2 = q1 + 2.0f * q2 + q3;
        p3 = q2 + 2.0f * q3 + q4;
      }
      // one field at a time (unrolled only with gravity, which keeps values per field): the
      // unrolled loop's code does not fit the instruction cache
#pragma unroll(GRAV ? NV : 1)
      for (int v = 0; v < NV; v++) {
        const ff dl[5] = {field(x, v, gs[0], th[0]), field(x + 1, v, gs[1], th[1]), field(x + 2, v, gs[2], th[2]),
                          field(x + 3, v, gs[3], th[3]), field(x + 4, v, gs[4], th[4])};
        PWeights W;
        ff t1, t2, t3;
        ok = weno_window_weights<ALTW>(dl, P.eps4, pp.wtype, W, t1, t2, t3) & ok;
        if (GRAV) {
          if (h) {
            const ff dc[5] = {field(xc, v, gc[0], tc[0]), field(xc + 1, v, gc[GRAV ? 1 : 0], tc[GRAV ? 1 : 0]),
                              field(xc + 2, v, gc[GRAV ? 2 : 0], tc[GRAV ? 2 : 0]),
                              field(xc + 3, v, gc[GRAV ? 3 : 0], tc[GRAV ? 3 : 0]),
                              field(xc + 4, v, gc[GRAV ? 4 : 0], tc[GRAV ? 4 : 0])};
            third_differences(dc, t1, t2, t3);
          } else {
            sch[v] = weno_sum6(W, tg1, tg2, tg3) * lcol[v];
            const float mg = weno_mag6(W, tg1, tg2, tg3) * fabsf(lcol[v].h) * (v < 2 ? sc01 : 1.0f);
            ok = ok & (mg <= 3.0e38f);
            magg = fmaxf(magg, mg);
          }
        }
        float mag = weno_mag6(W, t1, t2, t3);
        if (v < 2) mag = mag * sc01;
        ok = ok & (mag <= 3.0e38f);  // (the maxima below drop a NaN)
        const float w2 = h == 0 ? W.r3.h - W.l3.h : W.r3.h + W.l3.h - 1.0f;
        const float proj = PROJ ? ffma(W.r1.h, p3, ffma(W.l1.h, p1, fabsf(w2) * p2)) : 0.0f;
        if (h == 0) {
          pf = fmaxf(pf, proj);
          sx[v * S + w] = weno_sum6(W, t1, t2, t3);
          if (UPW == UPW_RF) sfd[v * S + w] = weno_dif6(W, t1, t2, t3);
          if (v < 3) ma = fmaxf(ma, mag);
          else ms = fmaxf(ms, mag);
        } else {
          pu = fmaxf(pu, proj);
          sx[(NV + v) * S + w] = weno_dif6(W, t1, t2, t3);
          if (STATES) sum[v * S + w] = weno_sum6(W, t1, t2, t3);
          if (v < 3) ua = fmaxf(ua, mag);
          else us = fmaxf(us, mag);
        }
      }
    }
    ff xs[NV], xd[NV], ud[NV];
#pragma unroll
    for (int v = 0; v < NV; v++) {
      xs[v] = sx[v * S + w];
      ud[v] = sx[(NV + v) * S + w];
      if (UPW == UPW_RF) xd[v] = sfd[v * S + w];
    }
    constexpr bool SAME_BASIS = UPW == UPW_RUS || M == MODEL_EULER1D || (M == MODEL_NS3D && UPW == UPW_ROE);
    if (SAME_BASIS) {
      rho = cl.t.h * cr.t.h;
      lam = fadd(fabsf(Ecc.un.h), Ecc.a.h);
      Hs = Ecc.H.h;
      ff lm[3] = {Ecc.un - Ecc.a, Ecc.un + Ecc.a, Ecc.un};
      float sg[3] = {0.0f, 0.0f, 0.0f};
      if (UPW == UPW_RUS) {
        const ff avg = (M == MODEL_EULER1D ? sqr(Ecc.a) : Ecc.a) + ffabs(Ecc.un);
        lm[0] = lm[1] = lm[2] = ffmax(ffmax(cl.c, cr.c), avg);
        if (GRAV) lm[0] = lm[1] = lm[2] = lm[0] * kap;
      } else if (UPW == UPW_ROE) {
#pragma unroll
        for (int k = 0; k < 3; k++) {
          lm[k] = M == MODEL_EULER1D ? ffabs(lm[k]) : pharten(lm[k]);
          if (GRAV) lm[k] = lm[k] * kap;
        }
      } else {
        const ff cv = cl.vel[DIR], rv = cr.vel[DIR];
        pfield<UPW>(cv - cl.c, lm[0], rv - cr.c, lm[0], sg[0]);
        pfield<UPW>(cv + cl.c, lm[1], rv + cr.c, lm[1], sg[1]);
        pfield<UPW>(cv, lm[2], rv, lm[2], sg[2]);
        if (GRAV) {
#pragma unroll
          for (int k = 0; k < 3; k++) lm[k] = lm[k] * kap;
        }
      }
      alm = fmaxf(lm[0].h, fmaxf(lm[1].h, lm[2].h));
      if (UPW == UPW_RF) alm = fmaxf(alm, lam);  // fields taken from one side count f's terms twice
#pragma unroll
      for (int k = 0; k < NV; k++) {
        const int m = k < 2 ? k : 2;
        FAcc r = acc_mul(neg(lm[m]), ud[k]);
        acc_add(r, xs[k]);
        if (UPW == UPW_RF) acc_add(r, mul2(xd[k], -sg[m]));
        xs[k] = acc_get(r);
      }
      pprojR<M, DIR>(Ecc, xs, g12);
      if (GRAV) {
        ff y[NV];
        pprojR<M, DIR>(Ecc, sch, y);
        gsm = y[1 + DIR];
        gse = y[NV - 1];
      }
    } else {
      ff fs6[NV], fd6[NV], us6[NV], ud6[NV], um[NV];
      pprojR<M, DIR>(Ecc, xs, fs6);
      pprojR<M, DIR>(Ecc, ud, ud6);
      if (UPW == UPW_RF) pprojR<M, DIR>(Ecc, xd, fd6);
#pragma unroll
      for (int v = 0; v < NV; v++) xs[v] = STATES ? sum[v * S + w] : xs[v];
      pprojR<M, DIR>(Ecc, xs, us6);
#pragma unroll
      for (int v = 0; v < NV; v++) {
        const ff* dd = sd + (NV + v) * S + w;
        um[v] = pmean(to_pair(su[v * S + w]), dd[0], dd[0] - dd[-1], dd[1] - dd[0], us6[v]);
      }
      pupwind<M, UPW, DIR>(fs6, fd6, ud6, um, Ecc, cl, cr, P, g12, lam, rho, Hs, alm);
    }
    // the fields' strengths are densities (shear: momenta) times a speed for f
    const float s0 = rho * lam, sm1 = s0 * lam;
    ok = ok & scales_in_range(rho, lam, Hs, GRAV ? kap.h : 1.0f) & (ffma(alm, ua, ma) <= BOUND * s0) &
         (ffma(alm, us, ms) <= BOUND * sm1);
    if (PROJ) ok = ok & (ffma(alm, pu, pf) <= PROJ_BOUND * s0);
    if (grav_dir) {
      const float rt = (float)term[0];
      ok = ok & (magg * rt <= BOUND * s0) & source_in_range(rt, lam, sm1, s0 * Hs);
    }
  }
  // What entered from a term that overflowed or was not finite is NaN here (every result is a
  // normalised pair).
#pragma unroll
  for (int v = 0; v < NV; v++) ok = ok & is_finite(g12[v]);
  if (grav_dir) ok = ok & is_finite(gsm) & is_finite(gse);
  // The differences are read no more: their place takes G and the cells' sums.
  const int pos = (COOP && iface && !ok) ? atomicAdd(cnt, 1) : 0;
  __syncthreads();
  double* sg = sf + NV * S;
  double* sh = sg + NV * S;
  double* ss = sh + NV * S;  // gravity: the source function's corrections, momentum and energy
  int* list = CHAR ? (int*)sx : (int*)sr;  // the slots evaluated in FP64 (in a free place)
  int* fp64 = list + 2 * S;                // per slot: whether its interface is
  fp64[w] = iface && !ok;
  if (iface && ok) {
#pragma unroll
    for (int v = 0; v < NV; v++) sg[v * S + w] = to_double(mulu(ffc(1.0 / 12.0), g12[v]));
    if (GRAV && src_dir) {
      ss[w] = to_double(ffc(1.0 / 12.0) * gsm);
      ss[S + w] = to_double(ffc(1.0 / 12.0) * gse);
    }
  }
  if (!COOP) {
    if (iface && !ok)
      iface_fp64<M, CHAR, UPW, DIR, ALTW, GRAV>(U, line_base(l0 + line), a0 - 3 + q, G, sf, sgf, sgg, S, w, pp, src_dir,
                                                sg + w, ss + w);
  } else if (const int nbad = *cnt) {
    if (iface && !ok) list[pos] = w;
    __syncthreads();
    constexpr int NT = Fp64Tasks<M, CHAR>::N;
    const int batch = S / 4;  // NV S values of scratch
    for (int base = 0; base < nbad; base += batch) {
      const int m = nbad - base < batch ? nbad - base : batch;
      // characteristic: whole quantities where the single fields would take more than two rounds
      const bool whole = CHAR && m * NT > 2 * T;
      if constexpr (CHAR) {
        for (int k = t; whole && k < m * 2; k += T)
          fp64_fields<M, DIR, ALTW>(su, sf, S, list[base + (k >> 1)], k & 1, pp, sh + (k >> 1) * 4 * NV);
      }
      for (int k = t; !whole && k < m * NT; k += T) {
        const int it = k / NT, x = list[base + it], l = x / LL;
        fp64_task<M, CHAR, UPW, DIR, ALTW>(U, line_base(l0 + l), a0 - 3 + x - l * LL, G, sf, S, x, k - it * NT, pp,
                                           sh + it * 4 * NV);
      }
      __syncthreads();
      for (int it = t; it < m; it += T) {
        const int x = list[base + it], l = x / LL;
        fp64_upwind<M, CHAR, UPW, DIR>(U, line_base(l0 + l), a0 - 3 + x - l * LL, G, sf, S, x, pp, sh + it * 4 * NV,
                                       sg + x);
      }
      __syncthreads();
    }
  }
  if (iface) {
    const int i = a0 - 3 + q;  // the own cell
    const int I = i + 1;  // the interface to its right
    if (ep.bnd && (I == 0 || I == N)) {
      double Fb[NV];
#pragma unroll
      for (int v = 0; v < NV; v++) {
        const double* f = sf + v * S + w;
        Fb[v] = (ok ? fma(7.0, f[0] + f[1], -(f[-1] + f[2])) * (1.0 / 12.0) : f[0]) + sg[v * S + w];
      }
      boundary_flux<NV>(ep, I, N, l0 + line, ntrans, Fb);
    }
  }
  __syncthreads();
  if (own) {
    const double dxi = dxinv[G.g + a0 - 3 + q], c1 = dxi * (2.0 / 3.0), c2 = dxi * (-1.0 / 12.0);
    const bool fr = fp64[w], fl = fp64[w - 1];
#pragma unroll
    for (int v = 0; v < NV; v++) {
      const double* f = sf + v * S + w;
      const double g1 = sg[v * S + w], g0 = sg[v * S + w - 1];
      double h;
      if (fr | fl) {
        // beside an interface evaluated in FP64 the fluxes may jump: both relative to their left
        // cells, as in the FP64 kernels, where the central difference would round the jump
        const double D1 = fr ? g1 : central_rel(f) + g1, D0 = fl ? g0 : central_rel(f - 1) + g0;
        h = dxi * ((f[0] - f[-1]) + (D1 - D0));
      } else {
        const double c4 = fma(c1, f[1] - f[-1], (f[2] - f[-2]) * c2);
        h = fma(dxi, g1 - g0, c4);
      }
      if (GRAV && src_dir && (v == 1 + DIR || v == NV - 1)) {
        const int k = v == 1 + DIR ? 0 : 1;
        const double* g = sgg + w;
        const double g4 = fma(2.0 / 3.0, g[1] - g[-1], (g[2] - g[-2]) * (-1.0 / 12.0));
        h = fma(-term[k] * (g4 + (ss[k * S + w] - ss[k * S + w - 1])), dxi, h);  // rhs = -hyp + source
      }
      sh[v * S + w] = h;
    }
  }
  __syncthreads();
  // Stage epilogue, value by value in the order of memory.
  constexpr int NB = 3;
  long long off[NB];
  double hv[NB];
  bool on[NB];
  if (DIR == 0) {
    for (int l = 0; l < nl; l++) {
      const long long ob = (line_base(l0 + l) + (long long)a0 * sdir) * NV;
      for (int i0 = t; i0 < Lc * NV; i0 += NB * T) {
#pragma unroll
        for (int k = 0; k < NB; k++) {
          const int i = i0 + k * T, c = i / NV, v = i - c * NV;
          on[k] = i < Lc * NV;
          off[k] = ob + i;
          hv[k] = on[k] ? sh[v * S + l * LL + c + 3] : 0.0;
        }
        stage_epilogue_batch<NB>(ep, H, off, hv, on);
      }
    }
  } else {
    const int R = nl * NV, c0 = t / R, r = t - c0 * R, l = r / NV, v = r - l * NV, step = T / R;
    if (c0 < step) {
      const long long ob = (line_base(l0 + l) + (long long)a0 * sdir) * NV + v;
      for (int cc = c0; cc < Lc; cc += NB * step) {
#pragma unroll
        for (int k = 0; k < NB; k++) {
          const int c = cc + k * step;
          on[k] = c < Lc;
          off[k] = ob + (long long)c * sdir * NV;
          hv[k] = on[k] ? sh[v * S + l * LL + c + 3] : 0.0;
        }
        stage_epilogue_batch<NB>(ep, H, off, hv, on);
      }
    }
  }
}

// Blocks (pair_threads) per SM the kernels are held to.  Bound by issue slots and latency
// (6,000 to 10,000 mostly FP32 instructions per thread against 60-150 FP64 ones): two blocks
// (128 registers) left the schedulers idle half of the time; three (80 registers; spills in
// the FP64 evaluation only) took the 1024^2 vortex from 3.12 to 2.56 ms per step when they were
// brought in, four (64 registers) were no faster (2.54 ms; shared memory allows three).
constexpr int PAIR_MINB = 3;
template <int M, bool CHAR, int UPW, int DIR, bool ALTW, bool GRAV>
__global__ void __launch_bounds__((M == MODEL_NS3D && !CHAR ? 224 : 256), PAIR_MINB)
hyp_pair_kernel(const double* __restrict__ U, double* __restrict__ H, const double* __restrict__ dxinv, DevGeom G,
                PhysParams pp, StageEpi ep, long long ntrans, int L, int XL) {
  extern __shared__ double pair_smem[];
  pdl_wait();
  pair_body<M, CHAR, UPW, DIR, ALTW, GRAV>(U, H, dxinv, G, pp, ep, ntrans, L, XL, blockIdx.x, pair_smem);
}

template <int M, bool CHAR, int UPW, int DIR, bool ALTW, bool GRAV>
cudaError_t launch_pair(const double* U, double* H, const double* dxinv_dir, const DevGeom& G, const PhysParams& pp,
                        const StageEpi& ep, long long ntrans, int cap, cudaStream_t s) {
  const int N = G.dim[DIR];
  const int most = pair_threads(M == MODEL_NS3D, CHAR);
  cap = cap > 0 ? cap : pair_cap(ntrans * N);
  const PairPlan p = pair_plan(N, ntrans, DIR, cap < most ? cap : most);
  const long long nblk = (ntrans + p.XL - 1) / p.XL * ((N + p.L - 1) / p.L);
  if (nblk > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
  auto k = hyp_pair_kernel<M, CHAR, UPW, DIR, ALTW, GRAV>;
  const size_t sm = PairLayout<M, CHAR, UPW, ALTW, GRAV>::bytes(p.T);
  if (sm > 48 * 1024)
    if (cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm)) return e;
  return launch_pdl(k, (unsigned)nblk, p.T, sm, s, U, H, dxinv_dir, G, pp, ep, ntrans, p.L, p.XL);
}

// Ensemble: the blocks of all members in one launch.
template <int M, bool CHAR, int UPW, int DIR>
__global__ void __launch_bounds__((M == MODEL_NS3D && !CHAR ? 224 : 256), PAIR_MINB)
hyp_batched_pair_kernel(const MemberDev* __restrict__ mem, int nmem, const double* __restrict__ U,
                        double* __restrict__ H, const double* __restrict__ dxinv, PhysParams pp, StageEpi ep) {
  extern __shared__ double pair_smem[];
  pdl_wait();
  StageEpi e = ep;
  const long long b = blockIdx.x;
  const MemberDev& m = batched_member<DIR>(mem, nmem, b, e);
  const long long o = m.off;
  pair_body<M, CHAR, UPW, DIR, false>(U + o, H ? H + o : nullptr, dxinv + m.dx_off[DIR], m.G, pp, e, m.ntrans[DIR],
                                      m.L[DIR], m.XL[DIR], b - m.start[DIR], pair_smem);
}

template <int M, bool CHAR, int UPW, int DIR>
cudaError_t launch_batched_pair(const MemberDev* mem, int nmem, long long nblk, int T, const double* U, double* H,
                                const double* dxinv, const PhysParams& pp, const StageEpi& ep, cudaStream_t s) {
  if (nblk <= 0) return cudaSuccess;
  if (nblk > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
  auto k = hyp_batched_pair_kernel<M, CHAR, UPW, DIR>;
  const size_t sm = PairLayout<M, CHAR, UPW, false, false>::bytes(T);
  if (sm > 48 * 1024)
    if (cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm)) return e;
  return launch_pdl(k, (unsigned)nblk, T, sm, s, mem, nmem, U, H, dxinv, pp, ep);
}

}  // namespace gbh
