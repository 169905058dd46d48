// mf_prim_exact.cu - conserved -> primitive variables on valueBox.grow(2), and
// the neutral pass-through at the sun after a level step.
//
// Built with -fmad=false: the primitive state feeds the limiter sign tests
// and the region thresholds, so it is rounded exactly as in the CPU
// restatement of the reference (EqSysMHDMF::stateToPrim).  The FP32 copy of
// W (mixed precision) is rounded to nearest by fp64::d2f, which gives the
// conversion instruction's bits with integer instructions (the kernel is
// bound by the FP64 pipe, where the conversion instruction issues).
#include "mf_internal.h"
#include "mf_fp64.cuh"
#include "mf_kernels.cuh"

namespace mf {
namespace {
// Store N primitive components of a cell to W and to its FP32 copy (each
// where not null).
template <int N>
__device__ __forceinline__ void store_prim(double* __restrict__ W, float* __restrict__ Wf,
                                           long long o, long long cs, const double* w) {
  if (W) {
#pragma unroll
    for (int q = 0; q < N; ++q) W[o + q * cs] = w[q];
  }
  if (Wf) {  // the FP32 copy the mixed-precision flux kernels read
#pragma unroll
    for (int q = 0; q < N; ++q) Wf[o + q * cs] = fp64::d2f(w[q]);
  }
}

// Far-field ghost state of the plasma (HELIOGS, swlism/HeliosphericF.ChF:
// 978-1140), psi 0 and the tracking surfaces: the region tracer +1 (:996-1000),
// the others, which HELIOGS leaves unassigned, keep U's ghost value.
__device__ __forceinline__ void far_plasma(const DevParams& P, const RunParams& R,
                                           const double* __restrict__ U, double* __restrict__ W,
                                           float* __restrict__ Wf, long long base, long long cs) {
  double w[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) w[q] = R.bc_plasma[q];
  store_prim<8>(W, Wf, base, cs, w);
  const double zero = 0.0;
  if (P.glm) store_prim<1>(W, Wf, base + 8 * cs, cs, &zero);
  for (int q = P.ils; q < P.nc; ++q) {
    const double v = (P.reg_tracer && q == P.nc - 1) ? 1.0 : U[base + q * cs];
    store_prim<1>(W, Wf, base + q * cs, cs, &v);
  }
}

// One thread per cell and fluid (blockIdx.y: 0 the plasma, psi and the
// tracking surfaces, else a neutral population): the kernel moves data, and a
// thread with a whole cell held 100 registers, too few warps to keep loads in
// flight.
__global__ void __launch_bounds__(kMaxBlock)
    k_prim(const __grid_constant__ DevParams P, const double* __restrict__ U, double* __restrict__ W,
           float* __restrict__ Wf, const StageDesc* __restrict__ descs, int ndesc, int total,
           const RunParams* __restrict__ runs, StepState* __restrict__ states, double dt_scale) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= total) return;
  const int f = blockIdx.y;
  const StageDesc& D = descs[find_desc(descs, ndesc, kRegW, g)];
  const int lin = g - D.g0[kRegW];
  const RunParams& R = runs[D.run];
  int x[3];
  decode(lin, D.wlo, D.wn, x[0], x[1], x[2]);
  const long long cs = (long long)D.fn[0] * D.fn[1] * D.fn[2];
  const long long base = D.u_off + loc(D.flo, D.fn, x[0], x[1], x[2]);
  int od = -1;
  if (P.bc_kind == MF_BC_FARFIELD) {
    for (int d = 0; d < P.sd; ++d)
      if (!P.periodic[d] && (x[d] < R.dlo[d] || x[d] > R.dhi[d])) od = d;
  }
  if (f == 0) {
    // GLM damping factor exp(-dt Ch^2 / Cp^2) of PSIPARABOLIC (src/DednerF.ChF:
    // 65-87) of the stage, once per patch (all of a run write the same value)
    // instead of in every warp of the update
    if (P.glm && states && lin == 0) {
      StepState& S = states[D.run];
      const double dt = S.dt * dt_scale;
      S.damp = exp(-dt * S.ch * S.ch / (S.cp * S.cp));
    }
    if (od >= 0) {
      far_plasma(P, R, U, W, Wf, base, cs);
      return;
    }
    double u[8], w[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) u[q] = U[base + q * cs];
    cons_to_prim_plasma(P, u, w);
    store_prim<8>(W, Wf, base, cs, w);
    // psi and the tracking surfaces: copied (EqSysMHDMF::stateToPrim,
    // srcIdeal/EqSysMHDMF.cpp:198-201, 207-210)
    if (P.glm) store_prim<1>(W, Wf, base + 8 * cs, cs, U + base + 8 * cs);
    for (int q = P.ils; q < P.nc; ++q)
      store_prim<1>(W, Wf, base + q * cs, cs, U + base + q * cs);
    return;
  }
  // far-field ghost: neutral fluid 1 from the boundary state, the others the
  // primitive state of the nearest domain cell along the boundary normal
  const int s = P.irhon + (f - 1) * 5;
  double u[5], w[5];
  if (od >= 0 && f == 1) {
#pragma unroll
    for (int q = 0; q < 5; ++q) w[q] = R.bc_n1[q];
  } else {
    long long from = base;
    if (od >= 0) {
      x[od] = (x[od] < R.dlo[od]) ? R.dlo[od] : R.dhi[od];
      from = D.u_off + loc(D.flo, D.fn, x[0], x[1], x[2]);
    }
#pragma unroll
    for (int q = 0; q < 5; ++q) u[q] = U[from + (s + q) * cs];
    cons_to_prim_euler(P, u, w);
  }
  store_prim<5>(W, Wf, base + s * cs, cs, w);
}

// Far-field ghosts of the primitive state, exactly as k_prim's far-field
// branch fills them, for the levels whose valid-cell primitives and ghost
// copies come first: plasma and neutral fluid 1 from the boundary state, the
// other neutral fluids from the primitive state of the nearest cell along the
// boundary normal: a valid cell of the patch or, one cell off the boundary, a
// ghost that the sibling copy filled (in the FP32 copy alone where the FP64
// state is not exchanged).  One block per box, fluid and 256 cells, or more
// cells where the box has over 2^24: a grid holds 65535 blocks along z.
__global__ void __launch_bounds__(256)
    k_farfield(const __grid_constant__ DevParams P, const double* __restrict__ U, double* W,
               float* __restrict__ Wf, const FarReg* __restrict__ regs,
               const RunParams* __restrict__ runs, int write_w) {
  const FarReg& F = regs[blockIdx.x];
  const RunParams& R = runs[F.run];
  const int f = blockIdx.y;
  const int n = F.ext[0] * F.ext[1] * F.ext[2];
  const long long cs = (long long)F.fn[0] * F.fn[1] * F.fn[2];
  double* Ww = write_w ? W : nullptr;  // (else only the FP32 ghosts are filled and read)
  const int s = P.irhon + (f - 1) * 5;
  for (int t = blockIdx.z * blockDim.x + threadIdx.x; t < n; t += gridDim.z * blockDim.x) {
    int x[3];
    decode(t, F.lo, F.ext, x[0], x[1], x[2]);
    const long long base = F.off + loc(F.flo, F.fn, x[0], x[1], x[2]);
    if (f == 0) {
      far_plasma(P, R, U, Ww, Wf, base, cs);
      continue;
    }
    double w[5];
    if (f == 1) {
#pragma unroll
      for (int q = 0; q < 5; ++q) w[q] = R.bc_n1[q];
    } else {
      for (int d = 0; d < P.sd; ++d)
        if (!P.periodic[d]) x[d] = min(max(x[d], R.dlo[d]), R.dhi[d]);
      const long long from = F.off + loc(F.flo, F.fn, x[0], x[1], x[2]) + s * cs;
      if (!write_w) {  // the FP64 ghosts were not copied: the FP32 copy of both
#pragma unroll
        for (int q = 0; q < 5; ++q) Wf[base + (s + q) * cs] = Wf[from + q * cs];
        continue;
      }
#pragma unroll
      for (int q = 0; q < 5; ++q) w[q] = W[from + q * cs];
    }
    store_prim<5>(Ww, Wf, base + s * cs, cs, w);
  }
}

// ---------------------------------------------------------------------------
// face fluxes in direction DIR
}  // namespace

cudaError_t launch_farfield(const DevParams& P, const double* u, double* w, float* wf,
                            const FarReg* far, int nfar, int most, const RunParams* runs,
                            int write_w, cudaStream_t s) {
  if (nfar <= 0) return cudaSuccess;
  const int blocks = (most + 255) / 256;
  const dim3 grid(nfar, P.nf, blocks < 65535 ? blocks : 65535);
  k_farfield<<<grid, 256, 0, s>>>(P, u, w, wf, far, runs, write_w);
  return cudaGetLastError();
}

cudaError_t launch_prim(const DevParams& P, const double* uin, double* w, const Batch& b,
                        cudaStream_t s, float* wf, StepState* state, double dt_scale) {
  if (b.tot_w <= 0) return cudaSuccess;
  const int nt = b.nt[0];
  const dim3 grid(flat_blocks(b.tot_w, nt), P.nf);
  k_prim<<<grid, nt, 0, s>>>(P, uin, w, wf, b.desc, b.ndesc, b.tot_w, b.runs, state, dt_scale);
  return cudaGetLastError();
}

}  // namespace mf

namespace mf {
namespace {
// NEUTRALS_SUNBC (swlism/SWLISMF.ChF:1555-1598): neutral fluid 1 (and 4)
// from the mirror cell, y and z momenta reversed.
__global__ void k_sun_copy(double* __restrict__ U, const SunPair* __restrict__ pairs, int n,
                           int irhon, int nf) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const SunPair sp = pairs[t];
  const double sg[5] = {1.0, 1.0, -1.0, -1.0, 1.0};
  for (int f = 1; f < nf; f += 3) {  // fluids 1 and 4
    const int s0 = irhon + (f - 1) * 5;
#pragma unroll
    for (int m = 0; m < 5; ++m)
      U[sp.to + (long long)(s0 + m) * sp.cs_to] =
          sg[m] * U[sp.from + (long long)(s0 + m) * sp.cs_from];
  }
}
}  // namespace

cudaError_t launch_sun_copy(double* U, const SunPair* pairs, int n, int irhon, int nf,
                            cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_sun_copy<<<(n + 127) / 128, 128, 0, s>>>(U, pairs, n, irhon, nf);
  return cudaGetLastError();
}
}  // namespace mf
