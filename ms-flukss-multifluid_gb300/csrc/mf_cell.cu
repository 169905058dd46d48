// mf_cell.cu - the update of the fast FP64 path and of the mixed-precision
// paths, one thread per cell and fluid.
#define MF_PHYS fast
#include "mf_sources.cuh"
#include "mf_cell_kernel.cuh"

namespace mf {

template <typename R>
cudaError_t launch_cells_fast(const DevParams& P, const StageBuffers& B, const Batch& b,
                              int flags, double dt_scale, StepState* state,
                              DtPartial* partials, int* nblocks_v, cudaStream_t s) {
  if constexpr (sizeof(R) == 4) {
    // charge-exchange rates: FP64, or FP32 in the opt-in MF_PREC_MIXED_CE32 form
    if (P.ce32)
      return launch_cells_t<R, float>(P, B, b, flags, dt_scale, state, partials, nblocks_v, s);
  }
  return launch_cells_t<R, double>(P, B, b, flags, dt_scale, state, partials, nblocks_v, s);
}

template cudaError_t launch_cells_fast<double>(const DevParams&, const StageBuffers&, const Batch&,
                                               int, double, StepState*, DtPartial*, int*,
                                               cudaStream_t);
template cudaError_t launch_cells_fast<float>(const DevParams&, const StageBuffers&, const Batch&,
                                              int, double, StepState*, DtPartial*, int*,
                                              cudaStream_t);

}  // namespace mf
