// mf_face_exact.cu - face fluxes of the FP64 parity path (built with -fmad=false),
// plasma and neutrals in kernels of their own.
#define MF_PHYS exact
#include "mf_riemann_exact.cuh"
#include "mf_face_kernel.cuh"

namespace mf {

cudaError_t launch_plasma_exact(const DevParams& P, const double* w, const double* const* fv,
                               void* const f[3], void* const bn[3], const Batch& b,
                               const StepState* state, cudaStream_t s) {
  return launch_plasma_t(P, w, fv, f, bn, b, state, s);
}

cudaError_t launch_neutral_exact(const DevParams& P, const double* w, const double* const* fv,
                                void* const f[3], const Batch& b, cudaStream_t s) {
  return launch_neutral_t(P, w, fv, f, b, s);
}

}  // namespace mf
