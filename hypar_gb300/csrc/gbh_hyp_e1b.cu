// EULER1D instantiation of the batched (ensemble) kernels.
#include "gbh_hyp_impl.cuh"
namespace gbh {
cudaError_t launch_batched_euler1d(int dir, int chr, int upw, const MemberDev* mem, int nmem, long long total, int T,
                                   const double* U, double* H, const double* dxinv, const PhysParams& pp,
                                   const StageEpi& ep, const HypLaunch& L, unsigned long long* counter, cudaStream_t s) {
  return launch_batched_model<MODEL_EULER1D>(dir, chr, upw, mem, nmem, total, T, U, H, dxinv, pp, ep, L, counter, s);
}
}  // namespace gbh
