// mf_face_fma.cu - face fluxes of the fast FP64 path, plasma and neutrals in
// kernels of their own: the parity path's routines with fused multiply-adds.
// With divisions and roots off the FP64 pipe their quotients cost less than
// products with shared reciprocals would.  Built with -fmad=false: every
// fusion is written out, so all kernels of this path round alike.
#define MF_PHYS fused
#define MF_RIEMANN_NS fused
#include "mf_riemann_exact.cuh"
#include "mf_face_kernel.cuh"

namespace mf {

cudaError_t launch_plasma_fast(const DevParams& P, const double* w, const double* const* fv,
                               void* const f[3], void* const bn[3], const Batch& b,
                               const StepState* state, cudaStream_t s) {
  return launch_plasma_t(P, w, fv, f, bn, b, state, s);
}

cudaError_t launch_neutral_fast(const DevParams& P, const double* w, const double* const* fv,
                                void* const f[3], const Batch& b, cudaStream_t s) {
  return launch_neutral_t(P, w, fv, f, b, s);
}

}  // namespace mf
