// mf_cell_exact.cu - the update of the FP64 parity path (built with
// -fmad=false), one thread per cell and fluid.
#define MF_PHYS exact
#define MF_CELL_REGS 128
#include "mf_sources_exact.cuh"
#include "mf_cell_kernel.cuh"

namespace mf {

cudaError_t launch_cells_exact(const DevParams& P, const StageBuffers& B, const Batch& b,
                               int flags, double dt_scale, StepState* state,
                               DtPartial* partials, int* nblocks_v, cudaStream_t s) {
  return launch_cells_t<double>(P, B, b, flags, dt_scale, state, partials, nblocks_v, s);
}

}  // namespace mf
