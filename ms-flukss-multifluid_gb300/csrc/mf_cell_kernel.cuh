// mf_cell_kernel.cuh - the update kernel with one thread per cell and fluid.
// Included by mf_cell_exact.cu (parity physics) and mf_cell.cu (fast physics);
// MF_PHYS names the physics namespace, MF_CELL_REGS the registers per thread.
//
// Bound by the FP64 pipe while enough warps are resident.  With one thread
// per cell a whole cell's state, its sources and their temporaries took 222
// registers: 2 warps per scheduler, the pipe 60 % busy.  Here a block of 64
// cells has two warps for the plasma and two for each neutral population; a
// thread holds one fluid, and the populations' charge-exchange terms reach
// the plasma (and the population that receives the new neutrals) through
// shared memory, summed there in the reference's order.  Parity update of a
// 64^3 heliosphere step: 1.45 -> 1.09 ms (96 to 168 registers measured the
// same, 80 2 % slower).
#pragma once

#include <cfloat>
#include <climits>

#include "mf_update_kernel.cuh"

namespace mf {
namespace {
using namespace MF_PHYS;

constexpr int kCells = kCellBlock;

constexpr int cell_blocks(int nf) { return 65536 / (MF_CELL_REGS * kCells * nf); }

// R: type of the face fluxes and wave speeds.
template <int NF, typename R>
__global__ void __launch_bounds__(kCells* NF, cell_blocks(NF))
    k_cells(const __grid_constant__ DevParams P, const __grid_constant__ StageBuffers B,
            const StageDesc* __restrict__ descs, int ndesc, int total, int flags,
            const RunParams* __restrict__ runs, StepState* __restrict__ states,
            const double dt_scale, DtPartial* __restrict__ partials) {
  constexpr int NN = NF - 1;
  __shared__ double terms[NN > 0 ? NN : 1][CeTerms::kShared][kCells];
  __shared__ R speed[NF][kCells];
  __shared__ int region[kCells];
  const int role = threadIdx.x / kCells, lane = threadIdx.x % kCells;  // role 0: the plasma
  const bool plasma = NN == 0 || role == 0;
  const bool ce = NN > 0 && P.ce;
  const int g = blockIdx.x * kCells + lane;
  const StageDesc* Dp = nullptr;
  int lin = 0;
  if (g < total) {
    Dp = &descs[find_desc(descs, ndesc, kRegV, g)];
    lin = g - Dp->g0[kRegV];
    if (lin >= Dp->vn[0] * Dp->vn[1] * Dp->vn[2]) Dp = nullptr;  // run-alignment gap
  }
  const int s = plasma ? 0 : P.irhon + (role - 1) * 5;  // first component of the thread's fluid
  int i = 0, j = 0, k = 0;
  long long cs = 0, base = 0;
  double dt = 0.0, r2 = -1.0, u[9];
  CeTerms t;
  if (Dp) {
    const StageDesc& D = *Dp;
    const RunParams& RP = runs[D.run];
    decode(lin, D.vlo, D.vn, i, j, k);
    cs = (long long)D.fn[0] * D.fn[1] * D.fn[2];
    base = D.u_off + loc(D.flo, D.fn, i, j, k);
    dt = dt_scale == 1.0 ? states[D.run].dt : states[D.run].dt * dt_scale;
    const double dtinv = dt * RP.invdx;
    const WColumn w{B.w + base, cs};
#pragma unroll
    for (int q = 0; q < 9; ++q)
      if (q < 5 || (plasma && (q < 8 || P.glm))) u[q] = B.uin[base + (s + q) * cs];
    // UPDATECONS (src/PatchMHDAMF.ChF:542-587), one direction after another
    // (FP32 fluxes: the differences of the directions are summed in FP32 and
    // enter the FP64 state once, as in update_cells)
    double divB = 0.0;
    R sum[sizeof(R) == 4 ? 9 : 1];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      if (d < P.sd) {
        int n[3] = {D.vn[0], D.vn[1], D.vn[2]};
        n[d] += 1;
        const long long fcs = (long long)n[0] * n[1] * n[2];
        const long long sf = (d == 0) ? 1 : (d == 1) ? (long long)n[0] : (long long)n[0] * n[1];
        const long long fo = loc(D.vlo, n, i, j, k);
        const R* __restrict__ F = (const R*)B.f[d] + D.f_off[d] + fo + s * fcs;
#pragma unroll
        for (int q = 0; q < 9; ++q) {
          if (q < 5 || (plasma && (q < 8 || P.glm))) {
            const R diff = F[q * fcs + sf] - F[q * fcs];
            if constexpr (sizeof(R) == 4)
              sum[q] = (d == 0) ? diff : sum[q] + diff;
            else
              u[q] = u[q] - dtinv * diff;
          }
        }
        if (plasma && P.use8) {  // COMPUTEDIVB
          const R* __restrict__ b = (const R*)B.bn[d] + D.bn_off[d] + fo;
          if constexpr (sizeof(R) == 4)
            divB = divB + fp64::f2d(b[sf] - b[0]);
          else
            divB = divB + b[sf] - b[0];
        }
      }
    }
    if constexpr (sizeof(R) == 4) {
#pragma unroll
      for (int q = 0; q < 9; ++q)
        if (q < 5 || (plasma && (q < 8 || P.glm))) u[q] = fma(-dtinv, fp64::f2d(sum[q]), u[q]);
    }
    if (plasma) {
      if (P.use8) {
        source_8wave(w, divB, ieee64::div(dt, RP.dx), u);
        if ((flags & kStageDt) && B.divb) B.divb[loc(B.divb_lo, B.divb_n, i, j, k)] = divB;
      }
      if (P.glm) u[8] = states[D.run].damp * u[8];  // PSIPARABOLIC (src/DednerF.ChF:65-87)
      if (ce) region[lane] = region_cell(P, RP.dx, i, j, k, w, 0.0, r2);
    } else if (ce) {
      charge_exchange_terms(P, w, s, t);
#pragma unroll
      for (int q = 0; q < CeTerms::kShared; ++q) terms[role - 1][q][lane] = t.shared[q];
    }
  }
  if (ce) __syncthreads();
  if (Dp) {
    const auto at = [&](int f, int q) { return terms[f][q][lane]; };
    bool finite = true;
    // charge exchange, then problem post-processing and positivity
    // (src/PatchMHDAM.cpp:705-707); with constrained transport these follow
    // the recalculation of B
    if (plasma) {
      if constexpr (NN > 0) {
        if (ce) charge_exchange_plasma<NN>(dt, u, at);
      }
      if (!P.ct) {
        if (P.reinit) reinit_plasma(P, runs[Dp->run].dx, i, j, k, stage_time(states[Dp->run], dt), r2, u);
        positivity_plasma(P, u);
      }
    } else {
      if constexpr (NN > 0) {
        if (ce) {
          const bool rec = ce_recipient(NN, region[lane]) == role;
          charge_exchange_neutral<NN>(rec, role - 1, WColumn{B.w + base, cs}, t, dt, u, at);
        }
      }
      if (!P.ct) positivity_neutral(P, role, u);
    }
    // AVERAGESTATE (src/PatchMHDAMF.ChF:289-316): half the difference is
    // exact, so the fused form rounds once, like the sum
#pragma unroll
    for (int q = 0; q < 9; ++q) {
      if (q < 5 || (plasma && (q < 8 || P.glm))) {
        const long long o = base + (s + q) * cs;
        if (flags & kStageAverage) u[q] = fma(0.5, B.uold[o] - B.uin[o], u[q]);
        finite = finite && ((__double2hiint(u[q]) & 0x7ff00000) != 0x7ff00000);
        B.uout[o] = u[q];
      }
    }
    if (!finite) atomicOr(&states[Dp->run].flags, kFlagNonFinite);
    if (flags & kStageDt)
      speed[role][lane] = plasma ? wave_speed_plasma<R>(P, u) : wave_speed_neutral<R>(P, u);
  }
  if (flags & kStageDt) {
    __syncthreads();
    double dtc = DBL_MAX;
    int idx = INT_MAX;
    if (plasma && Dp) {
      double cmax = 0.0;
#pragma unroll
      for (int f = 0; f < NF; ++f) cmax = ieee64::maxnum((double)speed[f][lane], cmax);
      dtc = ieee64::div(runs[Dp->run].dx, cmax);
      idx = g;
    }
    block_dt_min(dtc, idx, descs, ndesc, partials, blockIdx.x);
  }
}

template <typename R>
cudaError_t launch_cells_t(const DevParams& P, const StageBuffers& B, const Batch& b,
                                  int flags, double dt_scale, StepState* state,
                                  DtPartial* partials, int* nblocks_v, cudaStream_t s) {
  const unsigned nb = flat_blocks(b.tot_v, kCells);
  if (nblocks_v) *nblocks_v = (int)nb;
  if (b.tot_v <= 0) return cudaSuccess;
#define MF_CELLS(NF)                                                                             \
  k_cells<NF, R><<<nb, kCells * NF, 0, s>>>(P, B, b.desc, b.ndesc, b.tot_v, flags, b.runs, \
                                               state, dt_scale, partials)
  switch (P.nf) {
    case 1: MF_CELLS(1); break;
    case 2: MF_CELLS(2); break;
    case 3: MF_CELLS(3); break;
    case 4: MF_CELLS(4); break;
    default: MF_CELLS(5); break;
  }
#undef MF_CELLS
  return cudaGetLastError();
}

}  // namespace
}  // namespace mf
