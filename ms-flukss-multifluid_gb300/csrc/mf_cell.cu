// mf_cell.cu - the update of the fast FP64 path and of the mixed-precision
// paths, one thread per cell and fluid.
#define MF_PHYS fast
// 64 registers a thread (4 blocks of 4 fluids per SM), a few spilled: the FP64
// work left per thread hides less latency than the parity update's, and more
// warps pay (mixed 128^3: 5.32 ms a step at 128 registers, 4.86 at 80, 4.54 at
// 64; fast FP64 6.01, 5.63, 5.61; the parity update 8.51, 8.92, 8.84)
#define MF_CELL_REGS 64
#include "mf_sources.cuh"
#include "mf_cell_kernel.cuh"

namespace mf {

template <typename R>
cudaError_t launch_cells_fast(const DevParams& P, const StageBuffers& B, const Batch& b,
                              int flags, double dt_scale, StepState* state,
                              DtPartial* partials, int* nblocks_v, cudaStream_t s) {
  return launch_cells_t<R>(P, B, b, flags, dt_scale, state, partials, nblocks_v, s);
}

template cudaError_t launch_cells_fast<double>(const DevParams&, const StageBuffers&, const Batch&,
                                               int, double, StepState*, DtPartial*, int*,
                                               cudaStream_t);
template cudaError_t launch_cells_fast<float>(const DevParams&, const StageBuffers&, const Batch&,
                                              int, double, StepState*, DtPartial*, int*,
                                              cudaStream_t);

}  // namespace mf
