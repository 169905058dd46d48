// mf_face_kernel.cuh - face fluxes of the FP64 paths, plasma and neutral
// populations in kernels of their own, all directions in one launch.
// Included by mf_face_exact.cu (parity path) and mf_face_fma.cu (fast FP64
// path); MF_PHYS names the physics namespace of the including unit.
//
// Bound by the FP64 pipe while enough warps are resident, else by the
// latency of each warp's chain of FP64 and integer instructions (with both
// parts in one kernel, 200 registers, 2 warps per scheduler: pipe 53 % busy).
// The parts share nothing but the face, so the neutral populations run one
// per thread with a third of the registers, and the plasma solver alone fits
// eight blocks of 64 per SM.  The state is loaded in the face's
// frame (normal, then the two transverse components), which makes the code
// the same for the three directions: one kernel instead of three, a third of
// the instruction cache.  Fluxes of a 64^3 heliosphere step: 3.68 -> 2.33 ms
// (pipe 75 % busy).  The plasma kernel takes 8 blocks per SM (128 registers;
// 128^3, plasma fluxes of a stage in ms, 6 / 8 / 10 blocks: parity 6.08 / 5.98 /
// 6.13, fast FP64 5.27 / 4.68 / 4.75).  The neutral kernel takes 8 blocks (64 registers): its
// products run on the integer pipes (vanleer_euler), whose latency more warps
// hide (128^3, three populations: 6.04 ms a step with the products on the
// FP64 pipe and 4 blocks, 5.67 with both changed).
#pragma once

#include "mf_kernels.cuh"

namespace mf {
namespace {
using namespace MF_PHYS;

constexpr int kPlasmaThreads = 64, kNeutralThreads = 128;
constexpr int kPlasmaBlocks = 8, kNeutralBlocks = 8;  // per SM

// The faces of a batch in every direction: the launch's blocks cover those of
// direction 0, then 1, then 2 (nb blocks each).  w: the primitive state whose
// cells the face states are limited from; fv: the Hancock corrector's face
// values instead (low, then high face of every component per cell of the
// slope box, nc components).
struct FaceBatch {
  const double* w;
  const double* fv[3];
  int nc;
  double* f[3];
  double* bn[3];
  int tot[3], nb[3];
};

// One face: its patch, position, and where its stencil and fluxes lie.
struct Face {
  const StageDesc* D;
  int dir, pos;          // direction, index along it
  const double* w;       // component 0 of the cell on the face's high side
  long long cs, st;      // component and stencil strides of w
  const double* fr;      // Hancock: component 0 of the high cell's low-face value
  const double* fl;      // and of the low cell's high-face value
  long long scs;         // their component stride
  double* f;             // component 0 of the face's flux
  double* bn;
  long long fcs;         // component stride of f
};

template <bool HANCOCK>
__device__ __forceinline__ bool find_face(const FaceBatch& A, const StageDesc* __restrict__ descs,
                                          int ndesc, Face& F) {
  int blk = blockIdx.x, dir = 0;
  if (blk >= A.nb[0]) {
    blk -= A.nb[0];
    dir = 1;
    if (blk >= A.nb[1]) {
      blk -= A.nb[1];
      dir = 2;
    }
  }
  const int gi = blk * blockDim.x + threadIdx.x;
  if (gi >= A.tot[dir]) return false;
  const StageDesc& D = descs[find_desc(descs, ndesc, kRegF + dir, gi)];
  int n[3] = {D.vn[0], D.vn[1], D.vn[2]};
  n[0] += (dir == 0);
  n[1] += (dir == 1);
  n[2] += (dir == 2);
  int i, j, k;
  decode(gi - D.g0[kRegF + dir], D.vlo, n, i, j, k);
  F.D = &D;
  F.dir = dir;
  F.pos = (dir == 0) ? i : (dir == 1) ? j : k;
  F.cs = (long long)D.fn[0] * D.fn[1] * D.fn[2];
  F.st = (dir == 0) ? 1 : (dir == 1) ? (long long)D.fn[0] : (long long)D.fn[0] * D.fn[1];
  F.w = A.w + D.u_off + loc(D.flo, D.fn, i, j, k);
  const long long fo = loc(D.vlo, n, i, j, k);
  F.f = A.f[dir] + D.f_off[dir] + fo;
  F.bn = A.bn[dir] + D.bn_off[dir] + fo;
  F.fcs = (long long)n[0] * n[1] * n[2];
  if (HANCOCK) {
    F.scs = (long long)D.sn[0] * D.sn[1] * D.sn[2];
    const long long ss = (dir == 0) ? 1 : (dir == 1) ? (long long)D.sn[0]
                                                     : (long long)D.sn[0] * D.sn[1];
    F.fr = A.fv[dir] + D.fv_off[dir] + loc(D.slo, D.sn, i, j, k);
    F.fl = F.fr + A.nc * F.scs - ss;
  }
  return true;
}

// Offset of the v-th component of a vector in the frame of direction dir
// (v = 0: normal).
__device__ __forceinline__ int axis(int dir, int v) {
  const int a = dir + v;
  return a >= 3 ? a - 3 : a;
}

// Limiters other than minmod: out of line, so that their twelve forms stand
// in the kernel once.
struct Pair {
  double lo, hi;
};
__device__ __noinline__ Pair limited(int lim, double a, double b, double c) {
  Pair p;
  face_values<double>(lim, a, b, c, p.lo, p.hi);
  return p;
}

// Face states of component c: the high-face value of the low cell (l) and the
// low-face value of the high cell (r); flat cells keep their own value.
template <bool HANCOCK>
__device__ __forceinline__ void face_pair(const Face& F, int c, int lim, bool flatL, bool flatR,
                                          double& l, double& r) {
  if (HANCOCK) {
    l = __ldg(F.fl + c * F.scs);
    r = __ldg(F.fr + c * F.scs);
    return;
  }
  const double* __restrict__ w = F.w + c * F.cs;
  const double wa = __ldg(w - 2 * F.st), wb = __ldg(w - F.st), wc = __ldg(w), wd = __ldg(w + F.st);
  if (lim == MF_LIM_MINMOD) {
    double lo, hi;
    face_values<double>(MF_LIM_MINMOD, wa, wb, wc, lo, l);
    face_values<double>(MF_LIM_MINMOD, wb, wc, wd, r, hi);
  } else {
    l = limited(lim, wa, wb, wc).hi;
    r = limited(lim, wb, wc, wd).lo;
  }
  l = flatL ? wb : l;
  r = flatR ? wc : r;
}

// CHECKPOSITIVITY (src/reconstructionF.ChF:1023-1054): cells whose rho or p
// face values are not positive fall back to first order.
__device__ __forceinline__ void flat_cells(const DevParams& P, const Face& F, bool& flatL,
                                           bool& flatR) {
  flatL = flatR = false;
  if (!P.check_pos) return;
  for (int c = 0; c <= 4; c += 4) {
    const double* __restrict__ w = F.w + c * F.cs;
    const double wa = w[-2 * F.st], wb = w[-F.st], wc = w[0], wd = w[F.st];
    const Pair a = limited(P.lim[c], wa, wb, wc), b = limited(P.lim[c], wb, wc, wd);
    flatL |= a.lo <= 0.0 || a.hi <= 0.0;
    flatR |= b.lo <= 0.0 || b.hi <= 0.0;
  }
}

// Plasma (and psi) fluxes and Bn of every face, the operations of k_flux (or,
// HANCOCK, of k_hflux: the face values were limited before the predictor).
template <int RS, bool HANCOCK>
__global__ void __launch_bounds__(kPlasmaThreads, kPlasmaBlocks)
    k_plasma(const __grid_constant__ DevParams P, const __grid_constant__ FaceBatch A,
             const StageDesc* __restrict__ descs, int ndesc, const RunParams* __restrict__ runs,
             const StepState* __restrict__ states) {
  Face F;
  if (!find_face<HANCOCK>(A, descs, ndesc, F)) return;
  bool flatL = false, flatR = false;
  if (!HANCOCK) flat_cells(P, F, flatL, flatR);
  double wl[9], wr[9], g[9];
#pragma unroll
  for (int v = 0; v < 8; ++v) {
    const int c = (v == 0 || v == 4) ? v : (v < 4) ? 1 + axis(F.dir, v - 1) : 5 + axis(F.dir, v - 5);
    face_pair<HANCOCK>(F, c, P.lim[c], flatL, flatR, wl[v], wr[v]);
  }
  wl[8] = wr[8] = 0.0;
  if (P.glm) face_pair<HANCOCK>(F, 8, MF_LIM_MINMOD, flatL, flatR, wl[8], wr[8]);
  if (RS == kRusanov)
    rusanov_mhd<double, 0>(P, wl, wr, g);
  else if (RS == kVFRoe)
    vfroe_mhd<double, 0>(P, wl, wr, g);
  else
    roe_mhd<double, 0, RS == kRoe7>(P, wl, wr, g);
  if (P.glm) {
    double fbn, fpsi;
    dedner_2x2<double>(states[F.D->run].ch, wl[5], wl[8], wr[5], wr[8], fbn, fpsi);
    g[5] = fbn;
    F.f[8 * F.fcs] = fpsi;
  }
#pragma unroll
  for (int v = 0; v < 8; ++v) {
    const int c = (v == 0 || v == 4) ? v : (v < 4) ? 1 + axis(F.dir, v - 1) : 5 + axis(F.dir, v - 5);
    F.f[c * F.fcs] = g[v];
  }
  // face-normal B (PatchMHDMF::computeBn, srcIdeal/PatchMHDMF.cpp:509-620)
  double bn = 0.0;
  if (P.divb_method == 1) {
    bn = half_r<double>(wl[5] + wr[5]);
    if (!P.periodic[F.dir]) {
      const RunParams& RP = runs[F.D->run];
      if (F.pos == RP.dlo[F.dir]) bn = wr[5];
      if (F.pos == RP.dhi[F.dir] + 1) bn = wl[5];
    }
  } else if (P.divb_method == 2) {
    const double* wv = F.w + (5 + F.dir) * F.cs;
    bn = 0.5 * (wv[-F.st] + wv[0]);
  }
  *F.bn = bn;
}

// Van Leer fluxes of one neutral population (blockIdx.y) of every face.
template <bool HANCOCK>
__global__ void __launch_bounds__(kNeutralThreads, kNeutralBlocks)
    k_neutral(const __grid_constant__ DevParams P, const __grid_constant__ FaceBatch A,
              const StageDesc* __restrict__ descs, int ndesc) {
  Face F;
  if (!find_face<HANCOCK>(A, descs, ndesc, F)) return;
  bool flatL = false, flatR = false;
  if (!HANCOCK) flat_cells(P, F, flatL, flatR);
  const int s = P.irhon + (int)blockIdx.y * 5;
  double nl[5], nr[5], g[5];
#pragma unroll
  for (int v = 0; v < 5; ++v) {
    const int c = s + ((v == 0 || v == 4) ? v : 1 + axis(F.dir, v - 1));
    face_pair<HANCOCK>(F, c, MF_LIM_MINMOD, flatL, flatR, nl[v], nr[v]);
  }
  vanleer_euler<double, 0>(P, nl, nr, g);
#pragma unroll
  for (int v = 0; v < 5; ++v) {
    const int c = s + ((v == 0 || v == 4) ? v : 1 + axis(F.dir, v - 1));
    F.f[c * F.fcs] = g[v];
  }
}

inline FaceBatch face_batch(const DevParams& P, const double* w, const double* const* fv,
                            void* const f[3], void* const bn[3], const Batch& b, int nt) {
  FaceBatch A;
  A.w = w;
  A.nc = P.nc;
  for (int d = 0; d < 3; ++d) {
    A.fv[d] = fv ? fv[d] : nullptr;
    A.f[d] = (double*)f[d];
    A.bn[d] = (double*)bn[d];
    A.tot[d] = d < P.sd ? b.tot_f[d] : 0;
    A.nb[d] = (A.tot[d] + nt - 1) / nt;
  }
  return A;
}

template <bool HANCOCK>
cudaError_t launch_plasma_t(const DevParams& P, const FaceBatch& A, const Batch& b,
                            const StepState* state, cudaStream_t s) {
  const int nb = A.nb[0] + A.nb[1] + A.nb[2];
  if (nb <= 0) return cudaSuccess;
#define MF_PLASMA(RS) \
  k_plasma<RS, HANCOCK><<<nb, kPlasmaThreads, 0, s>>>(P, A, b.desc, b.ndesc, b.runs, state)
  if (P.rs == kRusanov) MF_PLASMA(kRusanov);
  else if (P.rs == kVFRoe) MF_PLASMA(kVFRoe);
  else if (P.rs == kRoe8) MF_PLASMA(kRoe8);
  else MF_PLASMA(kRoe7);
#undef MF_PLASMA
  return cudaGetLastError();
}

inline cudaError_t launch_plasma_t(const DevParams& P, const double* w, const double* const* fv,
                                   void* const f[3], void* const bn[3], const Batch& b,
                                   const StepState* state, cudaStream_t s) {
  const FaceBatch A = face_batch(P, w, fv, f, bn, b, kPlasmaThreads);
  return fv ? launch_plasma_t<true>(P, A, b, state, s) : launch_plasma_t<false>(P, A, b, state, s);
}

inline cudaError_t launch_neutral_t(const DevParams& P, const double* w, const double* const* fv,
                                    void* const f[3], const Batch& b, cudaStream_t s) {
  void* const none[3] = {nullptr, nullptr, nullptr};
  const FaceBatch A = face_batch(P, w, fv, f, none, b, kNeutralThreads);
  const int nb = A.nb[0] + A.nb[1] + A.nb[2];
  if (nb <= 0 || P.nf < 2) return cudaSuccess;
  const dim3 grid(nb, P.nf - 1);
  if (fv)
    k_neutral<true><<<grid, kNeutralThreads, 0, s>>>(P, A, b.desc, b.ndesc);
  else
    k_neutral<false><<<grid, kNeutralThreads, 0, s>>>(P, A, b.desc, b.ndesc);
  return cudaGetLastError();
}

}  // namespace
}  // namespace mf
