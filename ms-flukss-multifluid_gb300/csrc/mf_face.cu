// mf_face.cu - face fluxes of the fast FP64 path,
// plasma and neutrals in kernels of their own.
#define MF_PHYS fast
#include "mf_riemann.cuh"
#include "mf_face_kernel.cuh"

namespace mf {

cudaError_t launch_plasma_fast(const DevParams& P, const double* w, void* const f[3],
                              void* const bn[3], const Batch& b, const StepState* state,
                              cudaStream_t s) {
  return launch_plasma_t(P, w, f, bn, b, state, s);
}

cudaError_t launch_neutral_fast(const DevParams& P, const double* w, void* const f[3],
                               const Batch& b, cudaStream_t s) {
  return launch_neutral_t(P, w, f, b, s);
}

}  // namespace mf
