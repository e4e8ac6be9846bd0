// gbh_visc.cu -- NavierStokes3D viscous term and the boundary / pointwise kernels.
//
// The viscous term follows NavierStokes3DParabolicFunction
// (src/PhysicalModels/NavierStokes3D/NavierStokes3DParabolicFunction.c:50-325)
// with the fourth-order central first derivative of
// FirstDerivativeFourthOrderCentral (src/FirstDerivative/FirstDerivativeFourthOrder.c:36-129),
// including its single-rank behaviour: a derivative along d is formed only on
// lines whose other indices are interior, so at a ghost point the derivatives
// across the ghost direction are zero.  Three passes over arrays of one component each
// (consecutive threads, consecutive addresses):
//   visc_q    : velocity and T = gamma P / rho at every point
//   visc_flux : the scaled derivatives of velocity and temperature, with the rule above,
//               and from them and mu = T^0.76 the stress tensor (6) and the energy fluxes (3)
//   visc_div  : par = sum over d of dxinv_d d/dx_d (flux along d) at interior points.
//
// All three are bound by arithmetic, the FP64 pipe above all (2 operations per clock and
// SM), so the passes share what the three directions have in common (some 150 FP64
// operations per point against the 310 of one flux pass per direction) and, where the viscous flux is
// small against the convective one, work in pairs of FP32 numbers (gbh_pair.cuh): the
// derivatives of the velocity, the stresses, the energy flux and their divergence.
// Velocities hold 48 bits as pairs, so their derivatives are off by 2^-50 |v| / h and the
// stress by 2^-50 mu |v| / (Re h); where mu / (Re h) is at most rho a / 32 at every point
// that is below a quarter of the rounding of the convective flux (rho a^2) it is added to.
// visc_q checks this, and any point that fails (or leaves the pairs' range, or is not
// finite) turns the whole evaluation to FP64.  Temperature derivatives stay in FP64.
// 256^3: 8.30 -> 2.6 ms per evaluation.
#include "gbh_internal.h"
#include "gbh_pair.cuh"

namespace gbh {

__device__ __forceinline__ int fold1(int i, int N, int lo, int hi) {
  if (i < 0) return lo == FOLD_PERIODIC ? i + N : (lo == FOLD_MIRROR ? -1 - i : i);
  if (i >= N) return hi == FOLD_PERIODIC ? i - N : (hi == FOLD_MIRROR ? 2 * N - 1 - i : i);
  return i;
}


// T^0.76 (raiseto, include/math_ops.h:37).  y = T^(19/25) from an FP32 estimate y0 and
// z = y0^25 / T^19 = (y0 / T)^19 y0^6: y = y0 z^(-1/25) = y0 (1 + e/25 + 13 e^2/625 + ...),
// e = 1 - z.  The estimate's error of some 1e-6 leaves 1e-17 after these terms, and the
// rounding of z (some ten units) counts a 25th: 18 FP64 operations against about 90 of
// exp(0.76 log T), at its accuracy.
__device__ __forceinline__ double pow076(double T) {
  const float t = d2f_mag(T);
  if (!(T > 0.0) || !(t > 1e-8f) || !(t < 1e8f)) return exp(0.76 * log(T));
  const double y = (double)exp2f(0.76f * log2f(t)), k = y * nr_rcp(T);
  const double k2 = k * k, k4 = k2 * k2, k8 = k4 * k4, k16 = k8 * k8, y2 = y * y;
  const double e = fma(-((k16 * k2) * k), (y2 * y2) * y2, 1.0);
  return fma(y * e, fma(13.0 / 625.0, e, 0.04), y);
}
// The same as a pair: z in pairs, to 2^-44 or so, whose 25th is the pair's own precision.
// (Beyond 1e-4 .. 1e4 the powers' second words leave the FP32 range: FP64.)
__device__ __forceinline__ ff pow076_pair(double T) {
  const float t = d2f_mag(T);
  if (!(T > 0.0) || !(t > 1e-4f) || !(t < 1e4f)) return to_pair(pow076(T));
  const float y = exp2f(0.76f * log2f(t));
  const ff k = mulf(rcp(to_pair(T)), y), k2 = sqr(k), k16 = sqr(sqr(sqr(k2)));
  const ff y2 = {fmul(y, y), ffma(y, y, -fmul(y, y))};
  const ff z = ((k16 * k2) * k) * (sqr(y2) * y2);
  const ff e = ff{1.0f, 0.0f} - z;
  return ff{y, 0.0f} + mulf(e * (ffc(0.04) + ff{fmul(0.0208f, e.h), 0.0f}), y);
}

// Arrays of one component each, n points: doubles u, v, w, T, then pairs u, v, w.
enum { VQ_T = 3, VQ_PAIR = 4 };

// At all points including ghosts; ghost points read through the fold.  flag[0] is set where the
// pairs' bound fails; visc_flux copies it to flag[1], which visc_div reads while it clears
// flag[0] for the next evaluation: no kernel reads what another thread of it writes, every
// evaluation starts from its own points alone, and a captured one does so at each replay.
__global__ void __launch_bounds__(256)
visc_q_kernel(const double* __restrict__ u, double* __restrict__ Q, const double* __restrict__ dxinv, DevGeom G,
              ViscParams vp, int* __restrict__ flag) {
  pdl_wait();
  const int ng0 = G.dim[0] + 2 * G.g, ng1 = G.dim[1] + 2 * G.g, ng2 = G.dim[2] + 2 * G.g;
  const long long n = (long long)ng0 * ng1 * ng2;
  long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  int i = (int)(p % ng0) - G.g;
  int j = (int)((p / ng0) % ng1) - G.g;
  int k = (int)(p / ((long long)ng0 * ng1)) - G.g;
  int si = fold1(i, G.dim[0], G.bclo[0], G.bchi[0]);
  int sj = fold1(j, G.dim[1], G.bclo[1], G.bchi[1]);
  int sk = fold1(k, G.dim[2], G.bclo[2], G.bchi[2]);
  long long q = (long long)(si + G.g) * G.stride[0] + (long long)(sj + G.g) * G.stride[1] +
                (long long)(sk + G.g) * G.stride[2];
  const double* uu = u + q * 5;
  double rho = uu[0];
  double ri = nr_rcp(rho);
  double v[3];
#pragma unroll
  for (int d = 0; d < 3; d++) v[d] = rho == 0.0 ? 0.0 : uu[1 + d] * ri;
  const double mv = fma(uu[1], v[0], fma(uu[2], v[1], uu[3] * v[2]));  // rho |v|^2
  const double T = vp.gamma * (fma(-0.5, mv, uu[4]) * vp.gm1) * ri;
#pragma unroll
  for (int d = 0; d < 3; d++) Q[d * n + p] = v[d];
  Q[VQ_T * n + p] = T;
  if (!flag) return;
  ff* R = (ff*)(Q + VQ_PAIR * n);
  float vm = 0.0f;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const ff pv = to_pair(v[d]);
    R[d * n + p] = pv;
    vm = fadd(vm, fabsf(pv.h));
  }
  const float h0 = d2f_mag(dxinv[G.g + i]), h1 = d2f_mag(dxinv[ng0 + G.g + j]), h2 = d2f_mag(dxinv[ng0 + ng1 + G.g + k]);
  const float h = fmaxf(h0, fmaxf(h1, h2)), hmin = fminf(h0, fminf(h1, h2));
  const float t = d2f_mag(T), r = d2f_mag(rho), ire = d2f_mag(vp.inv_Re), mu = exp2f(0.76f * log2f(t));
  // rho and 1/h in 2^-24 .. 2^24, a^2 in 2^-20 .. 2^40, |v| up to 2^24: the divergence of the
  // energy flux, up to rho a |v|^2 / h / 4, stays below 2^120, and 2^-59 of rho a^3 / h above
  // 2^-149, where second words end
  const bool ok = (T > 0.0) & (mu * ire * h <= 0.03125f * r * sqrtf(t)) & (t >= 9.5367432e-7f) &
                  (t <= 1.0995116e12f) & (r >= 5.9604645e-8f) & (r <= 1.6777216e7f) & (vm <= 1.6777216e7f) &
                  (hmin >= 5.9604645e-8f) & (h <= 1.6777216e7f) & (ire >= 8.6736174e-19f);
  // points off the interior in two directions enter no derivative (visc_flux), and boundaries
  // applied in memory leave them unset
  const int outside = (i < 0 || i >= G.dim[0]) + (j < 0 || j >= G.dim[1]) + (k < 0 || k >= G.dim[2]);
  if (!ok && outside < 2) flag[0] = 1;
}

// Fourth-order first derivative of one Q component at position i of a line of
// length N with g ghost points on each side, f(k) = value at position i+k.
template <class F>
__device__ __forceinline__ double d4(int i, int N, int g, F f) {
  const double one_twelve = 1.0 / 12.0;
  if (i == -g) return (-25.0 * f(0) + 48.0 * f(1) - 36.0 * f(2) + 16.0 * f(3) - 3.0 * f(4)) * one_twelve;
  if (i == -g + 1) return (-3.0 * f(-1) - 10.0 * f(0) + 18.0 * f(1) - 6.0 * f(2) + f(3)) * one_twelve;
  if (i < N + g - 2) return (f(-2) - 8.0 * f(-1) + 8.0 * f(1) - f(2)) * one_twelve;
  if (i == N + g - 2) return (-f(-3) + 6.0 * f(-2) - 18.0 * f(-1) + 10.0 * f(0) + 3.0 * f(1)) * one_twelve;
  return (3.0 * f(-4) - 16.0 * f(-3) + 36.0 * f(-2) - 48.0 * f(-1) + 25.0 * f(0)) * one_twelve;
}

// First-order one-sided first derivative (FirstDerivativeFirstOrder.c:50-84): bias 1
// forward, -1 backward in the interior of the ghost-extended line, forward at its first
// point and backward at its last, in the reference's expression
// max(bias,0) f(1) - bias f(0) + min(bias,0) f(-1).
template <class F>
__device__ __forceinline__ double d1(int i, int N, int g, int bias, F f) {
  if (i == -g) return f(1) - f(0);
  if (i == N + g - 1) return f(0) - f(-1);
  return (bias > 0) ? __dadd_rn(__dsub_rn(f(1), f(0)), __dmul_rn(0.0, f(-1)))
                    : __dsub_rn(__dadd_rn(__dmul_rn(0.0, f(1)), f(0)), f(-1));
}

// The numbers the passes work in.
__device__ __forceinline__ double vadd(double a, double b) { return a + b; }
__device__ __forceinline__ double vsub(double a, double b) { return a - b; }
__device__ __forceinline__ double vmul(double a, double b) { return a * b; }
__device__ __forceinline__ double vtwo(double a) { return 2.0 * a; }
__device__ __forceinline__ double veight(double a, double b) { return fma(8.0, a, b); }  // 8 a + b
__device__ __forceinline__ double vdot(double a, double x, double b, double y, double c, double z, double q) {
  return fma(a, x, fma(b, y, fma(c, z, q)));
}
__device__ __forceinline__ ff vadd(ff a, ff b) { return a + b; }
__device__ __forceinline__ ff vsub(ff a, ff b) { return a - b; }
__device__ __forceinline__ ff vmul(ff a, ff b) { return a * b; }
__device__ __forceinline__ ff vtwo(ff a) { return mul2(a, 2.0f); }
__device__ __forceinline__ ff veight(ff a, ff b) { return mul2(a, 8.0f) + b; }
__device__ __forceinline__ ff vdot(ff a, ff x, ff b, ff y, ff c, ff z, ff q) {
  FAcc s = acc_mul(a, x);
  acc_fma(s, b, y);
  acc_fma(s, c, z);
  acc_add(s, q);
  return acc_get(s);
}
template <class T> __device__ __forceinline__ T vnum(double x);
template <> __device__ __forceinline__ double vnum<double>(double x) { return x; }
template <> __device__ __forceinline__ ff vnum<ff>(double x) { return to_pair(x); }
__device__ __forceinline__ double vout(double x) { return x; }
__device__ __forceinline__ double vout(ff x) { return to_double(x); }

template <class T> __device__ __forceinline__ T vmu(double t);
template <> __device__ __forceinline__ double vmu<double>(double t) { return pow076(t); }
template <> __device__ __forceinline__ ff vmu<ff>(double t) { return pow076_pair(t); }

// The stress tensor (xx, yy, zz, xy, xz, yz) and energy fluxes (x, y, z) at one point
// (NavierStokes3DParabolicFunction.c:151-314) from the derivatives along the lines whose
// other indices are interior (on[e]; the rest are zero).
template <class T>
__device__ __forceinline__ void visc_flux_at(const double* __restrict__ Q, double* __restrict__ F, const DevGeom& G,
                                             const ViscParams& vp, const double* di, long long n, long long p,
                                             const int* idx, const bool* on) {
  const T* V = (const T*)(sizeof(T) == sizeof(double) && __is_same(T, double) ? Q : Q + VQ_PAIR * n);
  const double* TT = Q + VQ_T * n;
  T D[3][3], H[3];  // D[e][c] = d v_c / dx_e, H[e] = dT/dx_e
#pragma unroll
  for (int e = 0; e < 3; e++) {
    const long long sd = G.stride[e];
    const int i = idx[e], N = G.dim[e];
    if (!on[e]) {
#pragma unroll
      for (int c = 0; c < 3; c++) D[e][c] = vnum<T>(0.0);
      H[e] = vnum<T>(0.0);
      continue;
    }
    const bool central = vp.order != 2 && i > -G.g + 1 && i < N + G.g - 2;
    const double d12 = di[e] * (1.0 / 12.0);
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const T* f = V + c * n + p;
      if (central) {
        D[e][c] = vmul(veight(vsub(f[sd], f[-sd]), vsub(f[-2 * sd], f[2 * sd])), vnum<T>(d12));
      } else {  // the ends of the ghost-extended line (and the first-order scheme): FP64
        const double* b = Q + c * n + p;
        auto fk = [&](int k) { return b[k * sd]; };
        D[e][c] = vnum<T>((vp.order == 2 ? d1(i, N, G.g, 1, fk) : d4(i, N, G.g, fk)) * di[e]);
      }
    }
    const double* b = TT + p;
    auto fk = [&](int k) { return b[k * sd]; };
    if (central) H[e] = vnum<T>(fma(8.0, b[sd] - b[-sd], b[-2 * sd] - b[2 * sd]) * d12);
    else H[e] = vnum<T>((vp.order == 2 ? d1(i, N, G.g, 1, fk) : d4(i, N, G.g, fk)) * di[e]);
  }
  const T mr = vmul(vmu<T>(TT[p]), vnum<T>(vp.inv_Re)), kq = vmul(mr, vnum<T>(vp.inv_gm1 * vp.inv_Pr));
  const T third = vmul(vadd(vadd(D[0][0], D[1][1]), D[2][2]), vnum<T>(2.0 / 3.0));
  T s[6];
#pragma unroll
  for (int d = 0; d < 3; d++) s[d] = vmul(mr, vsub(vtwo(D[d][d]), third));
  s[3] = vmul(mr, vadd(D[1][0], D[0][1]));
  s[4] = vmul(mr, vadd(D[2][0], D[0][2]));
  s[5] = vmul(mr, vadd(D[2][1], D[1][2]));
  const T a = V[p], b = V[n + p], c = V[2 * n + p];
  T* out = (T*)F + p;
#pragma unroll
  for (int k = 0; k < 6; k++) out[k * n] = s[k];
  out[6 * n] = vdot(a, s[0], b, s[3], c, s[4], vmul(kq, H[0]));
  out[7 * n] = vdot(a, s[3], b, s[1], c, s[5], vmul(kq, H[1]));
  out[8 * n] = vdot(a, s[4], b, s[5], c, s[2], vmul(kq, H[2]));
}

// Points off the interior in one direction carry the flux along it only, two deep.
__global__ void __launch_bounds__(256)
visc_flux_kernel(const double* __restrict__ Q, double* __restrict__ F, const double* __restrict__ dxinv, DevGeom G,
                 ViscParams vp, int* flag) {
  pdl_wait();
  const bool refused = !flag || flag[0];
  if (flag && blockIdx.x == 0 && threadIdx.x == 0) flag[1] = refused;
  const int ng[3] = {G.dim[0] + 2 * G.g, G.dim[1] + 2 * G.g, G.dim[2] + 2 * G.g};
  const long long n = (long long)ng[0] * ng[1] * ng[2];
  const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const int idx[3] = {(int)(p % ng[0]) - G.g, (int)((p / ng[0]) % ng[1]) - G.g,
                      (int)(p / ((long long)ng[0] * ng[1])) - G.g};
  int outside = 0;
  bool reach = true, in[3];
#pragma unroll
  for (int e = 0; e < 3; e++) {
    in[e] = idx[e] >= 0 && idx[e] < G.dim[e];
    outside += !in[e];
    reach = reach && idx[e] >= -2 && idx[e] < G.dim[e] + 2;
  }
  if (outside > 1 || !reach) return;
  const bool on[3] = {in[1] && in[2], in[0] && in[2], in[0] && in[1]};
  const double di[3] = {dxinv[G.g + idx[0]], dxinv[ng[0] + G.g + idx[1]], dxinv[ng[0] + ng[1] + G.g + idx[2]]};
  if (!refused) visc_flux_at<ff>(Q, F, G, vp, di, n, p, idx, on);
  else visc_flux_at<double>(Q, F, G, vp, di, n, p, idx, on);
}

template <class T>
__device__ __forceinline__ void visc_div_at(const double* __restrict__ F0, double* out, const DevGeom& G,
                                            const ViscParams& vp, const double* di, long long n, long long p) {
  const T* F = (const T*)F0 + p;
  const int comp[3][4] = {{0, 3, 4, 6}, {3, 1, 5, 7}, {4, 5, 2, 8}};
#pragma unroll
  for (int v = 0; v < 4; v++) {
    T sum = vnum<T>(0.0);
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const T* f = F + comp[d][v] * n;
      const long long sd = G.stride[d];
      T term;
      // interior points: the central fourth-order difference, or the backward
      // first-order one of the second-order scheme
      if (__is_same(T, double) && vp.order == 2) {
        const double* b = (const double*)f;
        term = vnum<T>(di[d] * __dsub_rn(__dadd_rn(__dmul_rn(0.0, b[sd]), b[0]), b[-sd]));
      } else {
        term = vmul(veight(vsub(f[sd], f[-sd]), vsub(f[-2 * sd], f[2 * sd])), vnum<T>(di[d] * (1.0 / 12.0)));
      }
      sum = d == 0 ? term : vadd(sum, term);
    }
    out[1 + v] = vout(sum);
  }
}

__global__ void __launch_bounds__(256)
visc_div_kernel(const double* __restrict__ F, double* __restrict__ par, const double* __restrict__ dxinv, DevGeom G,
                ViscParams vp, int* flag) {
  pdl_wait();
  const bool refused = !flag || flag[1];
  if (flag && blockIdx.x == 0 && threadIdx.x == 0) flag[0] = 0;
  const long long m = (long long)G.dim[0] * G.dim[1] * G.dim[2];
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= m) return;
  const int i = (int)(t % G.dim[0]), j = (int)((t / G.dim[0]) % G.dim[1]), k = (int)(t / ((long long)G.dim[0] * G.dim[1]));
  const int ng0 = G.dim[0] + 2 * G.g, ng1 = G.dim[1] + 2 * G.g, ng2 = G.dim[2] + 2 * G.g;
  const long long n = (long long)ng0 * ng1 * ng2;
  const long long p = (long long)(i + G.g) * G.stride[0] + (long long)(j + G.g) * G.stride[1] +
                      (long long)(k + G.g) * G.stride[2];
  const double di[3] = {dxinv[G.g + i], dxinv[ng0 + G.g + j], dxinv[ng0 + ng1 + G.g + k]};
  double out[5];
  out[0] = 0.0;
  if (!refused) visc_div_at<ff>(F, out, G, vp, di, n, p);
  else visc_div_at<double>(F, out, G, vp, di, n, p);
#pragma unroll
  for (int v = 0; v < 5; v++) par[p * 5 + v] = out[v];
}

// flag: where the pairs may be used, two device integers, the first one 0; nullptr: FP64
// throughout.
cudaError_t launch_visc(const double* u, double* Q, double* F, double* par, const double* dxinv, const DevGeom& G,
                        const ViscParams& vp, int* flag, cudaStream_t s) {
  const long long n = (long long)(G.dim[0] + 2 * G.g) * (G.dim[1] + 2 * G.g) * (G.dim[2] + 2 * G.g);
  const long long m = (long long)G.dim[0] * G.dim[1] * G.dim[2];
  if (vp.order == 2) flag = nullptr;
  const unsigned gn = (unsigned)((n + 255) / 256), gm = (unsigned)((m + 255) / 256);
  if (cudaError_t e = launch_pdl(visc_q_kernel, gn, 256, 0, s, u, Q, dxinv, G, vp, flag)) return e;
  if (cudaError_t e = launch_pdl(visc_flux_kernel, gn, 256, 0, s, Q, F, dxinv, G, vp, flag)) return e;
  return launch_pdl(visc_div_kernel, gm, 256, 0, s, F, par, dxinv, G, vp, flag);
}

// ---------------------------------------------------------------------------
// Boundary zones applied to the array in memory (ApplyBoundaryConditions ->
// BCPeriodicU / BCExtrapolateU, src/BoundaryConditions/BCPeriodic.c:36-56,
// BCExtrapolate.c:29-46) for faces whose zone does not cover the whole face.
// ---------------------------------------------------------------------------
struct ZoneDev {
  int type, dim, face, is[3], ie[3];
  double data[8];
  double gamma;
  // thermal walls: the wall temperature field (all time levels) and the level in use;
  // turbulent inflow: the inflow data (all slices), their number and the slice in use
  const double* tfield;
  int tn, it;
};

// Ghost state from the mirror interior state w, for the wall and inflow /
// outflow types (BCSlipWall.c, BCNoslipWall.c, BCSubsonicInflow.c,
// BCSubsonicOutflow.c, BCSupersonicInflow.c, BCSupersonicOutflow.c; 2-D and 3-D
// branches), in their operation order without contraction.
template <int ND>
__device__ __forceinline__ void bc_ghost(const ZoneDev& z, const double* w, double* out, bool inflow = false,
                                         double Tb = 0.0, const double* fluct = nullptr) {
  constexpr int NV = ND + 2;
  const double gm1 = z.gamma - 1.0;
  const double inv_gm1 = __ddiv_rn(1.0, gm1);
  double rho = 0.0, vel[3] = {0.0, 0.0, 0.0}, P = 0.0;
  if (z.type != GB_BC_SUPERSONIC_INFLOW && z.type != GB_BC_TURBULENT_INFLOW) {
    rho = w[0];
    for (int d = 0; d < ND; d++) vel[d] = (ND == 3 && rho == 0.0) ? 0.0 : __ddiv_rn(w[1 + d], rho);
    double vsq = __dadd_rn(__dmul_rn(vel[0], vel[0]), __dmul_rn(vel[1], vel[1]));
    if (ND == 3) vsq = __dadd_rn(vsq, __dmul_rn(vel[2], vel[2]));
    P = __dmul_rn(__dsub_rn(w[NV - 1], __dmul_rn(__dmul_rn(0.5, rho), vsq)), gm1);
  }
  double rg = rho, vg[3] = {vel[0], vel[1], vel[2]}, Pg = P;
  switch (z.type) {
    case GB_BC_SLIP_WALL: vg[z.dim] = __dsub_rn(__dmul_rn(2.0, z.data[z.dim]), vel[z.dim]); break;
    case GB_BC_NOSLIP_WALL:
      for (int d = 0; d < ND; d++) vg[d] = __dsub_rn(__dmul_rn(2.0, z.data[d]), vel[d]);
      break;
    case GB_BC_SUBSONIC_INFLOW:
      rg = z.data[0];
      for (int d = 0; d < ND; d++) vg[d] = z.data[1 + d];
      break;
    case GB_BC_SUBSONIC_OUTFLOW: Pg = z.data[0]; break;
    case GB_BC_SUPERSONIC_INFLOW:
      rg = z.data[0];
      for (int d = 0; d < ND; d++) vg[d] = z.data[1 + d];
      Pg = z.data[1 + ND];
      break;
    case GB_BC_THERMAL_SLIP_WALL:
      // BCThermalSlipWall.c:86-105: the normal velocity mirrored about the wall's, the
      // pressure from the extrapolated density and the wall temperature
      vg[z.dim] = __dsub_rn(__dmul_rn(2.0, z.data[z.dim]), vel[z.dim]);
      Pg = __dmul_rn(rg, Tb);
      break;
    case GB_BC_THERMAL_NOSLIP_WALL:
      // BCThermalNoslipWall.c:86-105: every velocity component mirrored
      for (int d = 0; d < ND; d++) vg[d] = __dsub_rn(__dmul_rn(2.0, z.data[d]), vel[d]);
      Pg = __dmul_rn(rg, Tb);
      break;
    case GB_BC_TURBULENT_INFLOW:
      // BCTurbulentSupersonicInflow.c:54-85: the supersonic inflow state with the data's
      // velocity fluctuations added
      rg = z.data[0];
      for (int d = 0; d < ND; d++) vg[d] = __dadd_rn(z.data[1 + d], fluct[d]);
      Pg = z.data[1 + ND];
      break;
    case GB_BC_SUBSONIC_AMBIVALENT:
      // BCSubsonicAmbivalent.c:105-117: inflow's rule (density, velocity given) or
      // outflow's (pressure given) by the sign of the extrapolated face velocity
      if (inflow) {
        rg = z.data[0];
        for (int d = 0; d < ND; d++) vg[d] = z.data[1 + d];
      } else {
        Pg = z.data[1 + ND];
      }
      break;
    default: break;  // supersonic outflow: the interior state, energy recomputed
  }
  double vsq = __dadd_rn(__dmul_rn(vg[0], vg[0]), __dmul_rn(vg[1], vg[1]));
  if (ND == 3) vsq = __dadd_rn(vsq, __dmul_rn(vg[2], vg[2]));
  out[0] = rg;
  for (int d = 0; d < ND; d++) out[1 + d] = __dmul_rn(rg, vg[d]);
  out[NV - 1] = __dadd_rn(__dmul_rn(inv_gm1, Pg), __dmul_rn(__dmul_rn(0.5, rg), vsq));
}

__global__ void bc_zone_kernel(double* u, DevGeom G, int nv, ZoneDev z) {
  pdl_wait();
  pdl_launch();
  int b[3] = {1, 1, 1};
  for (int d = 0; d < G.nd; d++) b[d] = z.ie[d] - z.is[d];
  long long n = (long long)b[0] * b[1] * b[2];
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  int ib[3] = {(int)(t % b[0]), (int)((t / b[0]) % b[1]), (int)(t / ((long long)b[0] * b[1]))};
  int ig[3] = {0, 0, 0}, is[3] = {0, 0, 0};
  for (int d = 0; d < G.nd; d++) {
    ig[d] = ib[d] + z.is[d];
    is[d] = ig[d];
  }
  int dd = z.dim, N = G.dim[dd];
  if (z.type == GB_BC_PERIODIC) is[dd] = (z.face == 1) ? ib[dd] + N - G.g : ib[dd];
  else is[dd] = (z.face == 1) ? G.g - 1 - ib[dd] : N - ib[dd] - 1;  // the mirror interior point
  long long p1 = 0, p2 = 0;
  for (int d = 0; d < G.nd; d++) {
    p1 += (long long)(ig[d] + G.g) * G.stride[d];
    p2 += (long long)(is[d] + G.g) * G.stride[d];
  }
  if (z.type == GB_BC_PERIODIC || z.type == GB_BC_EXTRAPOLATE) {
    for (int v = 0; v < nv; v++) u[p1 * nv + v] = u[p2 * nv + v];
  } else if (z.type == GB_BC_REFLECT) {
    for (int v = 0; v < nv; v++) u[p1 * nv + v] = -u[p2 * nv + v];
  } else if (z.type == GB_BC_DIRICHLET) {
    for (int v = 0; v < nv; v++) u[p1 * nv + v] = z.data[v];
  } else {
    bool inflow = false;
    if (z.type == GB_BC_SUBSONIC_AMBIVALENT) {
      // BCSubsonicAmbivalent.c:70-92: the face velocity extrapolated from the boundary
      // cell and its neighbour at this transverse position, 1.5 v_1 - 0.5 v_2, on the
      // inward normal face * e_dim (only interior points are read: no ordering with the
      // ghost writes of other threads)
      long long q1 = 0, q2 = 0;
      for (int d = 0; d < G.nd; d++) {
        const int i1 = d == dd ? (z.face == 1 ? 0 : N - 1) : ig[d];
        const int i2 = d == dd ? (z.face == 1 ? 1 : N - 2) : ig[d];
        q1 += (long long)(i1 + G.g) * G.stride[d];
        q2 += (long long)(i2 + G.g) * G.stride[d];
      }
      const double *w1 = u + q1 * nv, *w2 = u + q2 * nv;
      const double r1 = w1[0], r2 = w2[0];
      const double m1 = w1[1 + dd], m2 = w2[1 + dd];
      const double v1 = (G.nd == 3 && r1 == 0.0) ? 0.0 : __ddiv_rn(m1, r1);
      const double v2 = (G.nd == 3 && r2 == 0.0) ? 0.0 : __ddiv_rn(m2, r2);
      const double vb = __dsub_rn(__dmul_rn(1.5, v1), __dmul_rn(0.5, v2));
      inflow = (z.face == 1) ? vb > 0.0 : vb < 0.0;
    }
    double Tb = 0.0;
    if (z.type == GB_BC_THERMAL_SLIP_WALL || z.type == GB_BC_THERMAL_NOSLIP_WALL) {
      // the temperature at this point: zone-relative index, the time level along dim
      // (BCThermalNoslipWall.c:80-84)
      long long q = 0, stride = 1;
      for (int d = 0; d < G.nd; d++) {
        q += stride * (d == dd ? z.it : ib[d]);
        stride *= (d == dd ? z.tn : b[d]);
      }
      Tb = z.tfield[q];
    }
    const double* fl = nullptr;
    if (z.type == GB_BC_TURBULENT_INFLOW) {
      // the slice in use along dim, the zone-relative indices across it (the data spans
      // the grid across, BCTurbulentSupersonicInflow.c:66-72)
      long long q = 0, stride = 1;
      for (int d = 0; d < G.nd; d++) {
        q += stride * (d == dd ? z.it : ib[d]);
        stride *= (d == dd ? z.tn : G.dim[d]);
      }
      fl = z.tfield + q * nv + 1;
    }
    double g[5];
    if (G.nd == 1) {
      // BCSlipWall.c:38-76 (Euler1D, the one wall type with a 1-D branch): density and
      // pressure extrapolated, the velocity mirrored about the wall's, in the 1-D flow
      // variables' operation order
      const double* w = u + p2 * nv;
      const double gm1 = z.gamma - 1.0, inv_gm1 = __ddiv_rn(1.0, gm1);
      const double rho = w[0], vel = __ddiv_rn(w[1], rho);
      const double P = __dmul_rn(__dsub_rn(w[2], __dmul_rn(__dmul_rn(__dmul_rn(0.5, rho), vel), vel)), gm1);
      const double vg = __dsub_rn(__dmul_rn(2.0, z.data[0]), vel);
      g[0] = rho;
      g[1] = __dmul_rn(rho, vg);
      g[2] = __dadd_rn(__dmul_rn(inv_gm1, P), __dmul_rn(__dmul_rn(__dmul_rn(0.5, rho), vg), vg));
    } else if (G.nd == 2) {
      bc_ghost<2>(z, u + p2 * nv, g, inflow, Tb, fl);
    } else {
      bc_ghost<3>(z, u + p2 * nv, g, inflow, Tb, fl);
    }
    for (int v = 0; v < nv; v++) u[p1 * nv + v] = g[v];
  }
}

cudaError_t launch_bc_zone_t(double* u, const DevGeom& G, int nv, const int* zone9, const double* data8,
                             double gamma, const double* tfield, int tn, int it, cudaStream_t s);

cudaError_t launch_bc_zone(double* u, const DevGeom& G, int nv, const int* zone9, const double* data8, double gamma,
                           cudaStream_t s) {
  return launch_bc_zone_t(u, G, nv, zone9, data8, gamma, nullptr, 0, 0, s);
}

// As launch_bc_zone, with a thermal wall's temperature field (tn time levels, device
// array) and the level `it` in use.
cudaError_t launch_bc_zone_t(double* u, const DevGeom& G, int nv, const int* zone9, const double* data8,
                             double gamma, const double* tfield, int tn, int it, cudaStream_t s) {
  if (zone9[0] == GB_BC_SPONGE) return cudaSuccess;  // a source term, no ghost points (BCSpongeUDummy)
  ZoneDev z;
  z.tfield = tfield;
  z.tn = tn;
  z.it = it;
  if ((zone9[0] == GB_BC_THERMAL_SLIP_WALL || zone9[0] == GB_BC_THERMAL_NOSLIP_WALL ||
       zone9[0] == GB_BC_TURBULENT_INFLOW) && (!tfield || tn < 1 || it < 0 || it >= tn))
    return cudaErrorInvalidValue;  // a thermal wall or turbulent inflow without its field
  z.type = zone9[0];
  z.dim = zone9[1];
  z.face = zone9[2];
  z.gamma = gamma;
  for (int k = 0; k < 8; k++) z.data[k] = data8 ? data8[k] : 0.0;
  long long n = 1;
  for (int d = 0; d < 3; d++) {
    z.is[d] = zone9[3 + d];
    z.ie[d] = zone9[6 + d];
    if (d < G.nd) n *= (z.ie[d] - z.is[d] > 0 ? z.ie[d] - z.is[d] : 0);
  }
  if (n <= 0) return cudaSuccess;
  return launch_pdl(bc_zone_kernel, (unsigned)((n + 255) / 256), 256, 0, s, u, G, nv, z);
}

// The sponge zone's source (BCSponge.c:34-61): src -= sigma_i (u - u_ref) at every
// interior point of the zone's extent, sigma indexed along the zone's dimension.  The
// three roundings of the reference's expression are kept (no contraction).  Zones may
// overlap: one launch per zone, in zone order, on one stream.
__global__ void sponge_kernel(double* __restrict__ src, const double* __restrict__ u, DevGeom G, int nv,
                              ZoneDev z, const double* __restrict__ sigma) {
  int b[3] = {1, 1, 1};
  for (int d = 0; d < G.nd; d++) b[d] = z.ie[d] - z.is[d];
  const long long n = (long long)b[0] * b[1] * b[2];
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const int ib[3] = {(int)(t % b[0]), (int)((t / b[0]) % b[1]), (int)(t / ((long long)b[0] * b[1]))};
  long long p = 0;
  for (int d = 0; d < G.nd; d++) p += (long long)(ib[d] + z.is[d] + G.g) * G.stride[d];
  const double sg = sigma[ib[z.dim]];
  for (int v = 0; v < nv; v++)
    src[p * nv + v] = __dsub_rn(src[p * nv + v], __dmul_rn(sg, __dsub_rn(u[p * nv + v], z.data[v])));
}

cudaError_t launch_sponge(double* src, const double* u, const DevGeom& G, int nv, const int* zone9,
                          const double* uref8, const double* sigma, cudaStream_t s) {
  if (zone9[0] != GB_BC_SPONGE) return cudaErrorInvalidValue;
  ZoneDev z;
  z.tfield = nullptr;
  z.tn = z.it = 0;
  z.type = zone9[0];
  z.dim = zone9[1];
  z.face = zone9[2];
  z.gamma = 0.0;
  for (int k = 0; k < 8; k++) z.data[k] = uref8[k];
  long long n = 1;
  for (int d = 0; d < 3; d++) {
    z.is[d] = zone9[3 + d];
    z.ie[d] = zone9[6 + d];
    if (d < G.nd) n *= (z.ie[d] - z.is[d] > 0 ? z.ie[d] - z.is[d] : 0);
  }
  if (n <= 0) return cudaSuccess;
  if (!sigma) return cudaErrorInvalidValue;
  sponge_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(src, u, G, nv, z, sigma);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Layout copies between interior-only and ghosted arrays, and a finite check.
// ---------------------------------------------------------------------------
__global__ void pack_kernel(double* dst, const double* src, DevGeom G, int nv, int to_interior) {
  long long n = (long long)G.dim[0] * G.dim[1] * G.dim[2];
  long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  int i = (int)(p % G.dim[0]);
  int j = (int)((p / G.dim[0]) % G.dim[1]);
  int k = (int)(p / ((long long)G.dim[0] * G.dim[1]));
  long long q = (long long)(i + G.g) * G.stride[0];
  if (G.nd > 1) q += (long long)(j + G.g) * G.stride[1];
  if (G.nd > 2) q += (long long)(k + G.g) * G.stride[2];
  for (int v = 0; v < nv; v++) {
    if (to_interior) dst[p * nv + v] = src[q * nv + v];
    else dst[q * nv + v] = src[p * nv + v];
  }
}

cudaError_t launch_pack(double* dst, const double* src, const DevGeom& G, int nv, int to_interior, cudaStream_t s) {
  long long n = (long long)G.dim[0] * G.dim[1] * G.dim[2];
  pack_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(dst, src, G, nv, to_interior);
  return cudaGetLastError();
}

__global__ void finite_kernel(const double* u, DevGeom G, int nv, int* flag) {
  long long n = (long long)G.dim[0] * G.dim[1] * G.dim[2];
  long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  int i = (int)(p % G.dim[0]);
  int j = (int)((p / G.dim[0]) % G.dim[1]);
  int k = (int)(p / ((long long)G.dim[0] * G.dim[1]));
  long long q = (long long)(i + G.g) * G.stride[0];
  if (G.nd > 1) q += (long long)(j + G.g) * G.stride[1];
  if (G.nd > 2) q += (long long)(k + G.g) * G.stride[2];
  bool bad = false;
  for (int v = 0; v < nv; v++) bad |= !isfinite(u[q * nv + v]);
  if (bad) atomicOr(flag, 1);
}

cudaError_t launch_finite_check(const double* u, const DevGeom& G, int nv, int* flag, cudaStream_t s) {
  long long n = (long long)G.dim[0] * G.dim[1] * G.dim[2];
  finite_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(u, G, nv, flag);
  return cudaGetLastError();
}

}  // namespace gbh
