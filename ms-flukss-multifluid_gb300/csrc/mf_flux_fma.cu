// mf_flux_fma.cu - face-flux kernels of the fast FP64 path for the options
// that mf_face_fma.cu does not take, by lines, from the Hancock corrector's
// face values and from given face states: the parity path's Riemann routines
// with fused multiply-adds (built with -fmad=false, see mf_face_fma.cu).
#define MF_PHYS fused
#define MF_RIEMANN_NS fused
#include "mf_riemann_exact.cuh"
#include "mf_flux_kernel.cuh"

namespace mf {

template <>
cudaError_t launch_flux_fast<double>(const DevParams& P, int dir, const double* w, void* f,
                                     void* bn, const Batch& b, const StepState* state,
                                     cudaStream_t s, const float*, int first, int end) {
  if (end < 0) end = b.tot_f[dir];
  if (end - first <= 0) return cudaSuccess;
  const int nt = b.nt[1];
  const unsigned nb = flat_blocks(end - first, nt);
  const dim3 gf(nb, helio_parts<double>(P, nb));
  double* F = (double*)f;
  double* Bn = (double*)bn;
  if (dir == 0)
    k_flux<double, 0, 0><<<gf, nt, 0, s>>>(P, w, nullptr, F, Bn, b.desc, b.ndesc, first, end,
                                            b.runs, state);
  if (dir == 1)
    k_flux<double, 1, 0><<<gf, nt, 0, s>>>(P, w, nullptr, F, Bn, b.desc, b.ndesc, first, end,
                                            b.runs, state);
  if (dir == 2)
    k_flux<double, 2, 0><<<gf, nt, 0, s>>>(P, w, nullptr, F, Bn, b.desc, b.ndesc, first, end,
                                            b.runs, state);
  return cudaGetLastError();
}

cudaError_t launch_flux_lines_fast(const DevParams& P, int dir, const double* w, void* f,
                                   void* bn, const Batch& b, const LinePlan& lp,
                                   const StepState* state, cudaStream_t s) {
  return launch_lflux_t<double>(P, dir, w, f, bn, b, lp, state, s);
}

cudaError_t lines_prepare_fma() { return lflux_allow_t<double>(); }

template <>
cudaError_t launch_face_flux_fast<double>(const DevParams& P, int dir, const double* wl,
                                          const double* wr, double* f, int n, double ch,
                                          cudaStream_t s) {
  return launch_face_flux_t<double>(P, dir, wl, wr, f, n, ch, s);
}

template <>
cudaError_t launch_hflux_fast<double>(const DevParams& P, int dir, const double* w,
                                      const double* fv, void* f, void* bn, const Batch& b,
                                      const StepState* state, cudaStream_t s) {
  return launch_hflux_t<double>(P, dir, w, fv, f, bn, b, state, s);
}

}  // namespace mf
