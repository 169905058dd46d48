// mf_sources.cuh - cell sources and cell-wise post-processing (always FP64):
// region classification, charge exchange, inner-sphere reset, positivity and
// the CFL wave speed.
//
// The region and sphere tests are thresholds on the primitive state; they use
// intrinsics that never fuse into multiply-adds so that each cell lands on the
// same side of every threshold as in the CPU restatement.
#pragma once

#include "mf_device.cuh"
#include "mf_fp64.cuh"

namespace mf {
namespace fast {

constexpr double kInvPi = 0.318309886183790671537767526745028724;

// DEFINE_REGIONS_TRACER_4F (swlism/SWLISMF.ChF:839-1016), Cartesian: regtr
// is the region tracer of the cell (negative: solar wind).  The thresholds
// are the routine's literals.  Its x > 650 test reads the x of the last
// solar-wind cell the routine visited (x is assigned in that branch only);
// here the cell's own x, the same on every domain within x <= 650.
template <typename WA>
__device__ __forceinline__ int region_tracer_cell(const DevParams& P, double dx, int i, int j,
                                                  int k, const WA& w, double regtr) {
  const double x = __dadd_rn(__dmul_rn(i + 0.5, dx), -P.sun_c[0]);
  const double ux = w[1], uy = w[2], uz = w[3];
  int reg;
  if (regtr < 0.0) {
    const double y = __dadd_rn(__dmul_rn(j + 0.5, dx), -P.sun_c[1]);
    double z = 0.0, r2, invr, ur;
    if (P.sd == 3) {
      z = __dadd_rn(__dmul_rn(k + 0.5, dx), -P.sun_c[2]);
      r2 = __dadd_rn(__dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)), __dmul_rn(z, z));
      invr = __ddiv_rn(1.0, __dsqrt_rn(r2));
      ur = __dadd_rn(__dadd_rn(__dmul_rn(ux, __dmul_rn(x, invr)), __dmul_rn(uy, __dmul_rn(y, invr))),
                     __dmul_rn(uz, __dmul_rn(z, invr)));
    } else {
      r2 = __dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y));
      invr = __ddiv_rn(1.0, __dsqrt_rn(r2));
      ur = __dadd_rn(__dmul_rn(ux, __dmul_rn(x, invr)), __dmul_rn(uy, __dmul_rn(y, invr)));
    }
    if (fabs(ur) >= __dmul_rn(0.6, P.sun_v)) {
      const double TEMP = __ddiv_rn(__dmul_rn(P.t_coeff, w[4]), w[0]);
      reg = ((TEMP >= 1.0e6) && (r2 > __dmul_rn(P.sun_r, P.sun_r))) ? 2 : 3;
    } else {
      reg = 2;
    }
    if (P.sd == 3 && ((z < P.zbot) || (z > P.ztop))) reg = 4;
  } else {
    reg = 1;
    double vel = __dadd_rn(__dmul_rn(ux, ux), __dmul_rn(uy, uy));
    if (P.sd == 3) vel = __dadd_rn(vel, __dmul_rn(uz, uz));
    vel = __dsqrt_rn(vel);
    const double ang = __ddiv_rn(
        __dadd_rn(__dadd_rn(__dmul_rn(ux, P.lism_u[0]), __dmul_rn(uy, P.lism_u[1])),
                  __dmul_rn(uz, P.lism_u[2])),
        vel);
    const double TEMP = __ddiv_rn(__dmul_rn(P.t_coeff, w[4]), w[0]);
    if (w[0] > 1.2) reg = 4;
    if (vel < 0.8) reg = 4;
    if (ang < 0.95) reg = 4;
    if (TEMP > 9000.0) reg = 4;
    if (x > 650.0) reg = 1;
  }
  return reg;
}

// DEFINE_REGIONS_2F (swlism/SWLISMF.ChF:654-742), Cartesian branch, or the
// tracer variant above (HeliosphericProblem::defineRegions,
// swlism/HeliosphericProblem.cpp:2538-2575).
// r2: receives the squared distance to the sun.
template <typename WA>
__device__ __forceinline__ int region_cell(const DevParams& P, double dx, int i, int j, int k,
                                           const WA& w, double regtr, double& r2) {
  using namespace ieee64;
  const double x = __dadd_rn(__dmul_rn(cell_centre(i), dx), -P.sun_c[0]);
  const double y = __dadd_rn(__dmul_rn(cell_centre(j), dx), -P.sun_c[1]);
  double z = 0.0;
  r2 = __dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y));
  if (P.sd == 3) {
    z = __dadd_rn(__dmul_rn(cell_centre(k), dx), -P.sun_c[2]);
    r2 = __dadd_rn(r2, __dmul_rn(z, z));
  }
  if (P.reg_tracer) return region_tracer_cell(P, dx, i, j, k, w, regtr);
  const double invr = div(1.0, root(r2));
  double ur = __dadd_rn(__dmul_rn(w[1], __dmul_rn(x, invr)), __dmul_rn(w[2], __dmul_rn(y, invr)));
  if (P.sd == 3) ur = __dadd_rn(ur, __dmul_rn(w[3], __dmul_rn(z, invr)));
  const double TEMP = div(__dmul_rn(P.t_coeff, w[4]), w[0]);
  const bool zout = (P.sd == 3) && (lt(z, P.zbot) || lt(P.ztop, z));
  int reg;
  if (le(P.lim_sun, absval(ur))) {
    reg = (le(1.0e6, TEMP) && lt(P.sun_r2, r2)) ? 2 : 3;
    if (zout) reg = 1;
  } else if (le(P.tmlim, TEMP)) {
    reg = zout ? 1 : 2;
  } else {
    reg = 1;
  }
  return reg;
}
template <typename WA>
__device__ __forceinline__ int region_cell(const DevParams& P, double dx, int i, int j, int k,
                                           const WA& w, double regtr) {
  double r2;
  return region_cell(P, dx, i, j, k, w, regtr, r2);
}

// Recipient of newly created neutrals: CHARGE_EXCHANGE_2F/3F/4F/MF
// (swlism/ChargeExchange2F.ChF:294-1149).
__device__ __forceinline__ int ce_recipient(int nN, int reg) {
  if (nN == 1) return (reg == 1 || reg == 4) ? 1 : 0;
  if (nN == 2) return (reg == 1) ? 1 : (reg == 2) ? 2 : 0;
  if (nN == 3) return (reg == 1 || reg == 4) ? 1 : (reg == 2) ? 2 : (reg == 3) ? 3 : 0;
  return (reg >= 1 && reg <= nN) ? reg : 0;
}

// Arithmetic type of the charge-exchange rates and wave speeds: FP64, or FP32
// (the rates in the opt-in MF_PREC_MIXED_CE32 mode, the wave speeds in every
// mixed mode; both scale what is a small fraction of the state per step).
// The FP64 forms take division and square root from the integer pipes
// (mf_ieee64.cuh) and the logarithm of mf_fp64.cuh.  Products and sums are
// written as fused operations (mad), or the product by prod() where it must
// not fuse, so that every kernel that inlines these routines rounds alike.
// The state update itself is FP64 either way.
__device__ __forceinline__ double mad(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float mad(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double prod(double a, double b) { return __dmul_rn(a, b); }
template <int K>
__device__ __forceinline__ double pow2(double x) { return ieee64::scale<K>(x); }
template <int K>
__device__ __forceinline__ float pow2(float x) {
  return x * (K < 0 ? 1.0f / (1 << (K < 0 ? -K : 0)) : (float)(1 << (K < 0 ? 0 : K)));
}
__device__ __forceinline__ double ce_log(double x) { return fp64::log64(x); }
__device__ __forceinline__ float ce_log(float x) { return logf(x); }
__device__ __forceinline__ double ce_exp(double x) { return exp(x); }
__device__ __forceinline__ float ce_exp(float x) { return expf(x); }
__device__ __forceinline__ double ce_pow(double x, double y) { return pow(x, y); }
__device__ __forceinline__ float ce_pow(float x, float y) { return powf(x, y); }
// conversions between the FP64 state and the type T of the rates, off the
// FP64 pipe (identities for T = double)
template <typename T>
__device__ __forceinline__ T to_t(double x);
template <> __device__ __forceinline__ double to_t<double>(double x) { return x; }
template <> __device__ __forceinline__ float to_t<float>(double x) { return fp64::d2f(x); }
__device__ __forceinline__ double to_d(float x) { return fp64::f2d(x); }
__device__ __forceinline__ double to_d(double x) { return x; }

// Pauls & Zank charge exchange of the plasma with one neutral population
// (HeliosphericProblem::explicitSource, swlism/HeliosphericProblem.cpp:1394-1539,
// CHARGE_EXCHANGE_4F swlism/ChargeExchange2F.ChF:673-993 and _MF :995-1149).
// FP64 rates.  The products ARR UD, ARR VVTHU and ARR VP_UHM that several
// terms share are formed once; the plasma's terms that carry a cell factor
// (ux, U2/2) are summed without it and scaled after the sum: the reference's
// H in another order.  The products stay on the FP64 pipe: on the integer
// pipes (ieee64::mul) the mixed update takes 4.18 instead of 4.00 ms a step at
// 128^3.
struct CeTerms {
  static constexpr int kShared = 9;
  // what the plasma sums over the populations: h2..h4, the S of PPLUX..Z,
  // ARR UD (-DENPLU), G (in the energy source and the recipient's energy
  // gain) and the rest of h5
  double shared[kShared];
  double own[4];  // PMIX, PMIY, PMIZ, ENMI
};

// w: the stage-start primitive state; o: the population's first component
template <typename WA>
__device__ __forceinline__ void charge_exchange_terms(const DevParams& P, const WA& w, int o,
                                                      CeTerms& c) {
  using namespace ieee64;
  constexpr double c4p = 4.0 * kInvPi, c16p = 16.0 * kInvPi, c94pi = 2.25 * kPi;
  constexpr double c649ip = 64.0 / 9.0 * kInvPi;
  const double rho = w[0], ux = w[1], uy = w[2], uz = w[3];
  const double rhoN = w[o], uxN = w[o + 1], uyN = w[o + 2], uzN = w[o + 3];
  const double VVTP = div(w[4], rho);
  const double VVTH = div(scale<1>(w[o + 4]), rhoN);
  const double dx_ = ux - uxN, dy_ = uy - uyN, dz_ = uz - uzN;
  const double hUH2 = half(mad(uzN, uzN, mad(uyN, uyN, uxN * uxN)));
  const double DU2 = mad(dz_, dz_, mad(dy_, dy_, dx_ * dx_)), DU24 = scale<2>(DU2);
  const double VPHH = mad(dz_, uzN, mad(dy_, uyN, dx_ * uxN));
  const double VPHP = mad(dz_, uz, mad(dy_, uy, dx_ * ux));
  // thermal + relative speeds; every radicand is > 0
  const double UD = root(mad(c4p, VVTH, mad(c4p, VVTP, DU2)));
  const double VVTHU = div(VVTH, root(mad(c94pi, VVTH, mad(c16p, VVTP, DU24))));
  const double VP_UHM = div(VVTP, root(mad(c16p, VVTH, mad(c94pi, VVTP, DU24))));
  const double UPE = root(mad(c649ip, VVTH, mad(c4p, VVTP, DU2)));
  const double UHE = root(mad(c4p, VVTH, mad(c649ip, VVTP, DU2)));
  const double UDS = P.ce_scale_vel * UD;
  const double t = mad(-P.ce_b, ce_log(UDS), P.ce_a);
  double SIG = t * t;
  const double damp_c = P.ce_damp_c;
  if (damp_c > 0.0) SIG = SIG * ce_pow(1.0 - ce_exp(-damp_c / UDS), P.ce_damp_pow);
  const double ARR = SIG * (rhoN * (P.ce_sigma_scale * rho));
  const double aU = prod(ARR, UD), aT = prod(ARR, VVTHU), aV = prod(ARR, VP_UHM);
  const double Y = 0.75 * ((ARR * UPE) * VVTH);
  const double hv = aU + aT + aV;
  c.shared[0] = prod(hv, dx_);
  c.shared[1] = prod(hv, dy_);
  c.shared[2] = prod(hv, dz_);
  c.shared[3] = prod(aV, dx_);
  c.shared[4] = prod(aV, dy_);
  c.shared[5] = prod(aV, dz_);
  c.shared[6] = aU;
  c.shared[7] = mad(aV, VPHP, (0.75 * VVTP) * (ARR * UHE));
  // (U2 - UH2) / 2 = (VPHP + VPHH) / 2, without the cancellation
  c.shared[8] = mad(aT, VPHH, mad(aU, half(VPHP + VPHH), -Y));
  c.own[0] = mad(uxN, aU, -(dx_ * aT));
  c.own[1] = mad(uyN, aU, -(dy_ * aT));
  c.own[2] = mad(uzN, aU, -(dz_ * aT));
  c.own[3] = mad(hUH2, aU, mad(-VPHH, aT, Y));
}

// S = -dt H of the plasma (momentum and energy; the magnetic field's and
// psi's S is zero) from the sums over the populations, sum[q] of shared[q].
__device__ __forceinline__ void charge_exchange_plasma(double dt, double* u, const double* sum) {
#pragma unroll
  for (int q = 0; q < 3; ++q) u[1 + q] = fma(-dt, sum[q], u[1 + q]);
  u[4] = fma(-dt, sum[7] + sum[8], u[4]);
}

// S = -dt H of a population's own loss and gain
__device__ __forceinline__ void charge_exchange_own(const CeTerms& c, double dt, double* un) {
  un[0] = fma(-dt, c.shared[6], un[0]);
#pragma unroll
  for (int q = 0; q < 4; ++q) un[1 + q] = fma(-dt, c.own[q], un[1 + q]);
}

// The newly created neutrals that the recipient gains (its own loss, already
// applied, cancels): from the sums; w: the plasma's primitive state.
template <typename WA>
__device__ __forceinline__ void charge_exchange_gain(const WA& w, const double* sum, double dt,
                                                     double* un) {
  const double ux = w[1], uy = w[2], uz = w[3], D = sum[6];
  const double hU2 = ieee64::half(mad(uz, uz, mad(uy, uy, ux * ux)));
  un[0] = fma(dt, D, un[0]);
  un[1] = fma(dt, mad(ux, D, sum[3]), un[1]);
  un[2] = fma(dt, mad(uy, D, sum[4]), un[2]);
  un[3] = fma(dt, mad(uz, D, sum[5]), un[3]);
  un[4] = fma(dt, mad(hU2, D, sum[7]), un[4]);
}

// The same for a thread per fluid; at(f, q): shared[q] of population f (from 0)
template <int NN, typename AT>
__device__ __forceinline__ void charge_exchange_sums(double* sum, const AT& at) {
#pragma unroll
  for (int q = 0; q < CeTerms::kShared; ++q) {
    sum[q] = at(0, q);
#pragma unroll
    for (int f = 1; f < NN; ++f) sum[q] = sum[q] + at(f, q);
  }
}
template <int NN, typename AT>
__device__ __forceinline__ void charge_exchange_plasma(double dt, double* u, const AT& at) {
  double sum[CeTerms::kShared];
  charge_exchange_sums<NN>(sum, at);
  charge_exchange_plasma(dt, u, sum);
}
template <int NN, typename WA, typename AT>
__device__ __forceinline__ void charge_exchange_neutral(bool rec, int f, const WA& w,
                                                        const CeTerms& c, double dt,
                                                        double* un, const AT& at) {
  charge_exchange_own(c, dt, un);
  if (!rec) return;
  double sum[CeTerms::kShared];
  charge_exchange_sums<NN>(sum, at);
  charge_exchange_gain(w, sum, dt, un);
}

// All populations of one cell by one thread with FP32 rates
// (MF_PREC_MIXED_CE32).  The update stays with one thread per cell there
// (update_by_fluid): the sums over the populations fuse into running totals,
// which a thread per population would round otherwise, and FP32 rounding of
// the rates moves the state by more than any FP64 order of the sums does.
template <int IRHON, typename WA, int NN>
__device__ __forceinline__ void charge_exchange_add_32(const DevParams& P, const WA& w, int reg,
                                                    double dt, double* u) {
  using T = float;
  const int nN = NN > 0 ? NN : P.nf - 1;
  constexpr T c4p = T(4.0 * kInvPi), c16p = T(16.0 * kInvPi), c94pi = T(2.25 * kPi);
  constexpr T c4ip = T(4.0 * kInvPi), c649ip = T(64.0 / 9.0 * kInvPi);
  const T rho = to_t<T>(w[0]), ux = to_t<T>(w[1]), uy = to_t<T>(w[2]), uz = to_t<T>(w[3]);
  const T U2 = ux * ux + uy * uy + uz * uz, hU2 = T(0.5) * U2;
  const T VVTP = to_t<T>(w[4]) * (T(1) / rho);
  // plasma thermal-speed terms of the five speed arguments
  const T aUDp = c4p * VVTP, aUPMp = c16p * VVTP, aUHMp = c94pi * VVTP;
  const T aPEp = c4ip * VVTP, aHEp = c649ip * VVTP, q75VP = T(0.75) * VVTP;
  const T scale_vel = to_t<T>(P.ce_scale_vel), ce_a = to_t<T>(P.ce_a), ce_b = to_t<T>(P.ce_b);
  const T damp_c = to_t<T>(P.ce_damp_c), damp_pow = to_t<T>(P.ce_damp_pow);
  const T srho = to_t<T>(P.ce_sigma_scale) * rho;
  // Each population's own loss / gain is applied inside the loop; the
  // recipient of the newly created neutrals (region-dependent) then also
  // receives the plasma's totals.  The products ARR*UD, ARR*VVTHU and
  // ARR*VP_UHM that several terms share are formed once, and the plasma's
  // terms that carry a cell factor (ux, U2/2, 3 VVTP/4) are summed without it
  // and scaled after the loop: the reference's H, summed in another order.
  // G: the sum of ARR (VPHP VP_UHM + 3 VVTP UHE / 4), which both the energy
  // source and the recipient's energy gain hold; H5: the rest of h5.
  T h2 = 0, h3 = 0, h4 = 0, DSUM = 0, S1x = 0, S1y = 0, S1z = 0, G = 0, H5 = 0;
#pragma unroll
  for (int f = 1; f < MF_MAX_FLUIDS; ++f) {
    if (f > nN) break;
    const int o = IRHON + (f - 1) * 5;
    const T rhoN = to_t<T>(w[o]), uxN = to_t<T>(w[o + 1]), uyN = to_t<T>(w[o + 2]), uzN = to_t<T>(w[o + 3]);
    const T dx_ = ux - uxN, dy_ = uy - uyN, dz_ = uz - uzN;
    const T UH2 = uxN * uxN + uyN * uyN + uzN * uzN;
    const T DU2 = dx_ * dx_ + dy_ * dy_ + dz_ * dz_, DU2x4 = T(4) * DU2;
    const T VPHH = dx_ * uxN + dy_ * uyN + dz_ * uzN;
    const T VPHP = dx_ * ux + dy_ * uy + dz_ * uz;
    const T VVTH = T(2) * (to_t<T>(w[o + 4]) * (T(1) / rhoN));
    // thermal + relative speeds; every argument is > 0, so sqrt(a) = a*rsqrt(a)
    const T aUD = (aUDp + c4p * VVTH) + DU2;
    const T UD = aUD * rsqrtf(aUD);
    const T iUPM = rsqrtf((aUPMp + c94pi * VVTH) + DU2x4);
    const T iUHM = rsqrtf((aUHMp + c16p * VVTH) + DU2x4);
    const T aPE = (aPEp + c649ip * VVTH) + DU2;
    const T UPE = aPE * rsqrtf(aPE);
    const T aHE = (aHEp + c4ip * VVTH) + DU2;
    const T UHE = aHE * rsqrtf(aHE);
    const T UDS = scale_vel * UD;
    const T t = ce_a - ce_b * ce_log(UDS);
    T SIG = t * t;
    if (damp_c > T(0)) SIG = SIG * ce_pow(T(1) - ce_exp(-damp_c / UDS), damp_pow);
    const T ARR = SIG * (rhoN * srho);
    const T aU = ARR * UD;                  // -DENPLU
    const T aT = ARR * (VVTH * iUPM);       // ARR*VVTHU
    const T aV = ARR * (VVTP * iUHM);       // ARR*VP_UHM
    const T Y = (ARR * UPE) * VVTH;
    const T hv = aU + aT + aV;
    h2 = h2 + hv * dx_;
    h3 = h3 + hv * dy_;
    h4 = h4 + hv * dz_;
    S1x = S1x + aV * dx_;
    S1y = S1y + aV * dy_;
    S1z = S1z + aV * dz_;
    DSUM = DSUM - aU;
    G = G + aV * VPHP + q75VP * (ARR * UHE);
    H5 = H5 + aT * VPHH + aU * (hU2 - T(0.5) * UH2) - T(0.75) * Y;
    double* un = u + IRHON + (f - 1) * 5;
    un[0] = un[0] - dt * to_d(aU);
    un[1] = un[1] - dt * to_d(uxN * aU - dx_ * aT);
    un[2] = un[2] - dt * to_d(uyN * aU - dy_ * aT);
    un[3] = un[3] - dt * to_d(uzN * aU - dz_ * aT);
    un[4] = un[4] - dt * to_d((T(0.5) * UH2) * aU - VPHH * aT + T(0.75) * Y);
  }
  const T h5 = G + H5;
  const T PPLUX = ux * DSUM - S1x, PPLUY = uy * DSUM - S1y, PPLUZ = uz * DSUM - S1z;
  const T ENPLU = hU2 * DSUM - G;
  u[1] = u[1] - dt * to_d(h2);
  u[2] = u[2] - dt * to_d(h3);
  u[3] = u[3] - dt * to_d(h4);
  u[4] = u[4] - dt * to_d(h5);
  // S of the magnetic field (and of psi) is zero; the recipient gets the
  // other populations' lost density (DSUM less its own, already applied)
  const int rk = ce_recipient(nN, reg);
#pragma unroll
  for (int f = 1; f < MF_MAX_FLUIDS; ++f) {
    if (f > nN) break;
    const bool rec = (f == rk);
    double* un = u + IRHON + (f - 1) * 5;
    un[0] = rec ? un[0] - dt * to_d(DSUM) : un[0];
    un[1] = rec ? un[1] - dt * to_d(PPLUX) : un[1];
    un[2] = rec ? un[2] - dt * to_d(PPLUY) : un[2];
    un[3] = rec ? un[3] - dt * to_d(PPLUZ) : un[3];
    un[4] = rec ? un[4] - dt * to_d(ENPLU) : un[4];
  }
}

// All populations of one cell by one thread.  w: the stage-start primitive
// state (an array, or a column view that loads each component where it is
// used).  NN > 0: the number of populations fixed at compile time (their
// independent chains can be scheduled together); 0: P.nf - 1 at run time.
template <int IRHON, typename T = double, typename WA = const double*, int NN = 0>
__device__ __forceinline__ void charge_exchange_add(const DevParams& P, const WA& w, int reg,
                                                    double dt, double* u) {
  if constexpr (sizeof(T) == 4) {
    charge_exchange_add_32<IRHON, WA, NN>(P, w, reg, dt, u);
  } else {
    const int nN = NN > 0 ? NN : P.nf - 1;
    double sum[CeTerms::kShared];
#pragma unroll
    for (int f = 0; f < MF_MAX_FLUIDS - 1; ++f) {
      if (f < nN) {
        CeTerms c;
        charge_exchange_terms(P, w, IRHON + f * 5, c);
        charge_exchange_own(c, dt, u + IRHON + f * 5);
#pragma unroll
        for (int q = 0; q < CeTerms::kShared; ++q)
          sum[q] = (f == 0) ? c.shared[q] : sum[q] + c.shared[q];
      }
    }
    charge_exchange_plasma(dt, u, sum);
    const int rk = ce_recipient(nN, reg);
#pragma unroll
    for (int f = 0; f < MF_MAX_FLUIDS - 1; ++f)
      if (f < nN && f + 1 == rk) charge_exchange_gain(w, sum, dt, u + IRHON + f * 5);
  }
}

// SOURCE8WAVES (srcIdeal/PatchIdealMHDF.ChF:681-722) + ADDSOURCES
template <typename WA>
__device__ __forceinline__ void source_8wave(const WA& w, double divB, double dtbydx, double* u) {
  const double dB = -divB * dtbydx;
  const double Ux = w[1], Uy = w[2], Uz = w[3];
  const double Bx = kInv4Pi * w[5], By = kInv4Pi * w[6], Bz = kInv4Pi * w[7];
  u[1] = mad(dB, Bx, u[1]);
  u[2] = mad(dB, By, u[2]);
  u[3] = mad(dB, Bz, u[3]);
  u[4] = mad(dB, mad(Bz, Uz, mad(By, Uy, Bx * Ux)), u[4]);
  u[5] = mad(dB, Ux, u[5]);
  u[6] = mad(dB, Uy, u[6]);
  u[7] = mad(dB, Uz, u[7]);
}

// HELIOREINIT_DEFAULT (swlism/HeliosphericPlasmaBCF.ChF:1435-1566): the
// plasma in r <= Rinit becomes the radial wind at time t (the stage's start
// time plus its dt); bipolar field: B flips where the colatitude is not
// below the current sheet's, and the current-sheet surface takes +1 / -1.
// The wind state of a cell inside the sphere.  Inlined: a call out of line
// would cost the whole calling kernel local-memory traffic.
static __device__ __host__ __forceinline__ void reinit_state(const ReinitIn P, double x,
                                                          double y, double z, double r2,
                                                          double t, ReinitState& o) {
  o.hcs = 0.0;
  const double r = sqrt(r2);
  const double rr = r / P.rint;
  const double xy = sqrt(x * x + y * y);
  const double cosT = z / r;
  const double sinT = sqrt(fmax(0.0, 1.0 - cosT * cosT));
  const double cosF = x / xy;
  const double sinF = y / xy;
  const double rho = P.sun_rho / (rr * rr);
  const double ux = P.sun_v * sinT * cosF;
  const double uy = P.sun_v * sinT * sinF;
  const double uz = P.sun_v * cosT;
  const double pr = P.sun_p / pow(rr, 2.0 * P.gamma);
  const double br = P.dir_br * P.sun_b / (rr * rr);
  const double bp = -P.sun_beta * br * r * sinT;
  double bx = br * sinT * cosF - bp * sinF;
  double by = br * sinT * sinF + bp * cosF;
  double bz = br * cosT;
  const double b = bx * bx + by * by + bz * bz;
  const double e0 = pr / P.hgamma + 0.5 * (rho * P.sun_v * P.sun_v + kInv4Pi * b);
  if (!P.monopolar) {
    const double theta = acos(cosT);
    double sinBr, cosBr;
    reinit_sincos(P.sun_beta * (r - P.sun_v * t), sinBr, cosBr);
    const double sinB = sinF * cosBr + cosF * sinBr;
    const double cosB = cosF * cosBr - sinF * sinBr;
    const double ct = P.cos_tilt * cosB;
    const double thetaS = asin(P.sin_tilt * sinB / sqrt(ct * ct + sinB * sinB)) + 0.5 * kPi;
    const bool keep = theta < thetaS;
    if (!keep) {
      bx = -bx;
      by = -by;
      bz = -bz;
    }
    o.hcs = keep ? 1.0 : -1.0;
  }
  o.u[0] = rho;
  o.u[1] = rho * ux;
  o.u[2] = rho * uy;
  o.u[3] = rho * uz;
  o.u[4] = e0;
  o.u[5] = bx;
  o.u[6] = by;
  o.u[7] = bz;
}

// The reset of one cell: the membership test in non-fused arithmetic (host
// and device agree exactly), then the wind state.
__device__ __host__ __forceinline__ bool reinit_wind(const DevParams& P, double dx, int i, int j,
                                                     int k, double t, ReinitState& o) {
#ifdef __CUDA_ARCH__
  const double x = __dadd_rn(__dmul_rn(i + 0.5, dx), -P.sun_c[0]);
  const double y = __dadd_rn(__dmul_rn(j + 0.5, dx), -P.sun_c[1]);
  const double z = (P.sd == 3) ? __dadd_rn(__dmul_rn(k + 0.5, dx), -P.sun_c[2]) : 0.0;
  const double r2 = (P.sd == 3)
                        ? __dadd_rn(__dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)), __dmul_rn(z, z))
                        : __dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y));
  if (!(r2 <= __dmul_rn(P.r0, P.r0))) return false;
#else
  const double x = (i + 0.5) * dx - P.sun_c[0];
  const double y = (j + 0.5) * dx - P.sun_c[1];
  const double z = (P.sd == 3) ? (k + 0.5) * dx - P.sun_c[2] : 0.0;
  const double r2 = (P.sd == 3) ? (x * x + y * y + z * z) : (x * x + y * y);
  if (!(r2 <= P.r0 * P.r0)) return false;
#endif
  reinit_state(reinit_in(P), x, y, z, r2, t, o);
  return true;
}

__device__ __host__ __forceinline__ void reinit_cell(const DevParams& P, double dx, int i, int j, int k,
                                            double t, double* u) {
  ReinitState o;
  if (!reinit_wind(P, dx, i, j, k, t, o)) return;
#pragma unroll
  for (int q = 0; q < 8; ++q) u[q] = o.u[q];
  if (!P.monopolar) {
    // a select per component keeps u in registers (ihcs is -1 or a surface
    // component; conditional stores would be merged into one indexed store,
    // which puts u in local memory)
#pragma unroll
    for (int q = 8; q < MF_MAX_COMP; ++q) u[q] = (q == P.ihcs) ? o.hcs : u[q];
  }
}

// The plasma alone (no tracking surfaces).  r2: the squared distance to the
// sun of region_cell, or < 0 where that did not run.
__device__ __forceinline__ void reinit_plasma(const DevParams& P, double dx, int i, int j, int k,
                                              double t, double r2, double* u) {
  ReinitState o;
  if (ieee64::lt(P.r0_2, r2) || !reinit_wind(P, dx, i, j, k, t, o)) return;
#pragma unroll
  for (int q = 0; q < 8; ++q) u[q] = o.u[q];
}

// POSTPROCESSING (srcIdeal/PatchIdealMHDF.ChF:1019-1070) and POSTPROCESSING_MF
// (srcIdeal/PatchMHDMFF.ChF:301-511).
__device__ __forceinline__ void positivity_plasma(const DevParams& P, double* u) {
  using namespace ieee64;
  const double hg = P.hgamma, ihg = P.invhgamma, smallR = P.smallr, smallP = P.smallp;
  double Rho = u[0];
  bool was = lt(Rho, smallR);
  if (P.nf == 1 && was) Rho = smallR;  // one fluid: the velocities of the floored density
  // kinetic energy from the momenta; the velocities only where a floor acts
  const double ke = half(div(mad(u[3], u[3], mad(u[2], u[2], u[1] * u[1])), Rho));
  const double Rho0 = Rho;
  const double BxB = prod(kInv8Pi, mad(u[7], u[7], mad(u[6], u[6], u[5] * u[5])));
  double Pr = hg * ((u[4] - BxB) - ke);
  if (was) Rho = smallR;
  if (lt(Pr, smallP)) { Pr = smallP; was = true; }
  if (was) {
    const double f = div(Rho, Rho0);
    u[0] = Rho;
    if (P.nf > 1) {
#pragma unroll
      for (int q = 1; q < 4; ++q) u[q] = u[q] * f;
    }
    u[4] = mad(Pr, ihg, mad(ke, f, BxB));
  }
}

// neutral fluid f (from 1)
__device__ __forceinline__ void positivity_neutral(const DevParams& P, int f, double* un) {
  using namespace ieee64;
  const double hg = P.hgamma, ihg = P.invhgamma;
  const double fd = (f == 1) ? P.smallr : (f == 3) ? kNet3Dens : kNet2Dens;
  const double fp = (f == 1) ? P.smallp : (f == 3) ? kNet3Pres : kNet2Pres;
  double Rho = un[0];
  const double ke = half(div(mad(un[3], un[3], mad(un[2], un[2], un[1] * un[1])), Rho));
  double Pr = hg * (un[4] - ke);
  bool was = false;
  if (lt(Rho, fd)) { Rho = fd; was = true; }
  if (lt(Pr, fp)) { Pr = fp; was = true; }
  if (was) {
    const double f = div(Rho, un[0]);
    un[0] = Rho;
#pragma unroll
    for (int q = 1; q < 4; ++q) un[q] = un[q] * f;
    un[4] = mad(Pr, ihg, ke * f);
  }
}

template <int IRHON>
__device__ __forceinline__ void positivity_cell(const DevParams& P, double* u) {
  positivity_plasma(P, u);
#pragma unroll
  for (int f = 1; f < MF_MAX_FLUIDS; ++f)
    if (f < P.nf) positivity_neutral(P, f, u + IRHON + (f - 1) * 5);
}

// MAXWAVESPEED (srcIdeal/PatchIdealMHDF.ChF:5-63) + MAXWAVESPEED_E
// (srcIdeal/PatchEulerF.ChF:5-50) of one cell.  The pressure is recovered
// from the total energy in FP64 (E minus kinetic minus magnetic cancels in
// cold, low-beta flow); the speeds are formed in T (FP64, or FP32 in the
// mixed precision modes, whose time step then carries FP32 rounding).
__device__ __forceinline__ double ws_sqrt(double x) { return ieee64::root(x); }
__device__ __forceinline__ float ws_sqrt(float x) { return sqrtf(x); }
__device__ __forceinline__ double ws_max(double a, double b) { return ieee64::maxnum(a, b); }
__device__ __forceinline__ float ws_max(float a, float b) { return fmaxf(a, b); }
__device__ __forceinline__ double ws_abs(double a) { return ieee64::absval(a); }
__device__ __forceinline__ float ws_abs(float a) { return fabsf(a); }

template <typename T = double>
__device__ __forceinline__ T wave_speed_plasma(const DevParams& P, const double* u) {
  const T i4pi = T(kInv4Pi), gam = to_t<T>(P.gamma);
  const double rinv = ieee64::div(1.0, u[0]);
  const double m1 = u[1], m2 = u[2], m3 = u[3], bx = u[5], by = u[6], bz = u[7];
  const double ke = prod(mad(m3, m3, mad(m2, m2, m1 * m1)), rinv);
  const double bb = prod(kInv4Pi, mad(bz, bz, mad(by, by, bx * bx)));
  const double p = ieee64::maxnum(P.hgamma * mad(-0.5, ke + bb, u[4]), P.smallp);
  const T invrho = to_t<T>(rinv), b = to_t<T>(bb);
  const T uu = to_t<T>(m1) * invrho, vv = to_t<T>(m2) * invrho, ww = to_t<T>(m3) * invrho;
  const T bxt = to_t<T>(bx), byt = to_t<T>(by), bzt = to_t<T>(bz);
  const T a2 = gam * to_t<T>(p) * invrho;
  const T as2 = pow2<-1>(mad(invrho, b, a2));
  const T as4 = as2 * as2;
  const T k4 = i4pi * invrho * a2;
  // as4 - k4 b^2 >= 0 exactly; contracted rounding can push it below 0
  T umax = ws_abs(uu) + ws_sqrt(as2 + ws_sqrt(ws_max(T(0), mad(-(k4 * bxt), bxt, as4))));
  umax = ws_max(ws_abs(vv) + ws_sqrt(as2 + ws_sqrt(ws_max(T(0), mad(-(k4 * byt), byt, as4)))), umax);
  return ws_max(ws_abs(ww) + ws_sqrt(as2 + ws_sqrt(ws_max(T(0), mad(-(k4 * bzt), bzt, as4)))), umax);
}

template <typename T = double>
__device__ __forceinline__ T wave_speed_neutral(const DevParams& P, const double* un) {
  const T gam = to_t<T>(P.gamma);
  const double rinv = ieee64::div(1.0, ieee64::maxnum(un[0], P.smallr));
  const double m1 = un[1], m2 = un[2], m3 = un[3];
  const double ke = prod(mad(m3, m3, mad(m2, m2, m1 * m1)), rinv);
  const double p = ieee64::maxnum(P.hgamma * mad(-0.5, ke, un[4]), P.smallp);
  const T invrho = to_t<T>(rinv);
  const T uu = to_t<T>(m1) * invrho, vv = to_t<T>(m2) * invrho, ww = to_t<T>(m3) * invrho;
  const T a = ws_sqrt(gam * to_t<T>(p) * invrho);
  return ws_max(ws_max(ws_abs(uu), ws_abs(vv)), ws_abs(ww)) + a;
}

template <int IRHON, typename T = double>
__device__ __forceinline__ double max_wave_speed(const DevParams& P, const double* u) {
  T cmax = ws_max(wave_speed_plasma<T>(P, u), T(0));
#pragma unroll
  for (int f = 1; f < MF_MAX_FLUIDS; ++f)
    if (f < P.nf) cmax = ws_max(wave_speed_neutral<T>(P, u + IRHON + (f - 1) * 5), cmax);
  return to_d(cmax);
}

}  // namespace fast
}  // namespace mf
