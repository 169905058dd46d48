// mf_sources_exact.cuh - cell sources and post-processing of the FP64 parity
// path (region classification, charge exchange, inner-sphere reset,
// positivity, CFL wave speed) in the reference's evaluation order.  Compiled
// without multiply-add contraction.
#pragma once

#include "mf_device.cuh"

namespace mf {
namespace exact {

// ---------------------------------------------------------------------------
// DEFINE_REGIONS_TRACER_4F (swlism/SWLISMF.ChF:839-1016), Cartesian: regtr
// is the region tracer of the cell (negative: solar wind).  The thresholds
// are the routine's literals.  Its x > 650 test reads the x of the last
// solar-wind cell the routine visited (x is assigned in that branch only);
// here the cell's own x, the same on every domain within x <= 650.
template <typename WA>
__device__ __forceinline__ int region_tracer_cell(const DevParams& P, double dx, int i, int j,
                                                  int k, const WA& w, double regtr) {
  const double x = (i + 0.5) * dx - P.sun_c[0];
  const double ux = w[1], uy = w[2], uz = w[3];
  int reg;
  if (regtr < 0.0) {
    const double y = (j + 0.5) * dx - P.sun_c[1];
    double z = 0.0, r2, invr, ur;
    if (P.sd == 3) {
      z = (k + 0.5) * dx - P.sun_c[2];
      r2 = x * x + y * y + z * z;
      invr = 1.0 / sqrt(r2);
      ur = ux * (x * invr) + uy * (y * invr) + uz * (z * invr);
    } else {
      r2 = x * x + y * y;
      invr = 1.0 / sqrt(r2);
      ur = ux * (x * invr) + uy * (y * invr);
    }
    if (fabs(ur) >= 0.6 * P.sun_v) {
      const double TEMP = P.t_coeff * w[4] / w[0];
      reg = ((TEMP >= 1.0e6) && (r2 > P.sun_r * P.sun_r)) ? 2 : 3;
    } else {
      reg = 2;
    }
    if (P.sd == 3 && ((z < P.zbot) || (z > P.ztop))) reg = 4;
  } else {
    reg = 1;
    double vel = (P.sd == 3) ? (ux * ux + uy * uy + uz * uz) : (ux * ux + uy * uy);
    vel = sqrt(vel);
    const double ang = (ux * P.lism_u[0] + uy * P.lism_u[1] + uz * P.lism_u[2]) / vel;
    const double TEMP = P.t_coeff * w[4] / w[0];
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
  const double x = cell_centre(i) * dx - P.sun_c[0];
  const double y = cell_centre(j) * dx - P.sun_c[1];
  double z = 0.0;
  r2 = x * x + y * y;
  if (P.sd == 3) {
    z = cell_centre(k) * dx - P.sun_c[2];
    r2 = r2 + z * z;
  }
  if (P.reg_tracer) return region_tracer_cell(P, dx, i, j, k, w, regtr);
  const double invr = div(1.0, root(r2));
  double ur = w[1] * (x * invr) + w[2] * (y * invr);
  if (P.sd == 3) ur = ur + w[3] * (z * invr);
  double TEMP = div(P.t_coeff * w[4], w[0]);
  int reg;
  bool zout = (P.sd == 3) && (lt(z, P.zbot) || lt(P.ztop, z));
  if (le(P.lim_sun, absval(ur))) {
    reg = (le(1.0e6, TEMP) && lt(P.sun_r2, r2)) ? 2 : 3;
    if (zout) reg = 1;
  } else {
    if (le(P.tmlim, TEMP)) {
      reg = 2;
      if (zout) reg = 1;
    } else {
      reg = 1;
    }
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

// Pauls & Zank charge exchange of the plasma with one neutral population
// (HeliosphericProblem::explicitSource, swlism/HeliosphericProblem.cpp:1394-1539;
// CHARGE_EXCHANGE_*, swlism/ChargeExchange2F.ChF:294-1149).
struct CeTerms {
  static constexpr int kShared = 9;
  // what the plasma sums over the populations: the terms of h2..h5, ARR UD
  // (-DENPLU) and the terms of PPLUX, PPLUY, PPLUZ, ENPLU
  double shared[kShared];
  double pmi[3], enmi;  // PMIX, PMIY, PMIZ, ENMI
};

// w: the stage-start primitive state; o: the population's first component.
// Factors that are powers of two scale exactly and move out of the products.
template <typename T = double, typename WA>
__device__ __forceinline__ void charge_exchange_terms(const DevParams& P, const WA& w, int o,
                                                      CeTerms& c) {
  using namespace ieee64;
  const double rho = w[0], ux = w[1], uy = w[2], uz = w[3], pp = w[4];
  const double rhoN = w[o], uxN = w[o + 1], uyN = w[o + 2], uzN = w[o + 3], pN = w[o + 4];
  const double U2 = ux * ux + uy * uy + uz * uz;
  const double VVTP = div(pp, rho);
  const double dx_ = ux - uxN, dy_ = uy - uyN, dz_ = uz - uzN;
  const double UH2 = uxN * uxN + uyN * uyN + uzN * uzN;
  const double DU2 = dx_ * dx_ + dy_ * dy_ + dz_ * dz_, DU24 = scale<2>(DU2);
  const double VPHH = dx_ * uxN + dy_ * uyN + dz_ * uzN;
  const double VPHP = dx_ * ux + dy_ * uy + dz_ * uz;
  const double VVTH = div(scale<1>(pN), rhoN);
  const double UD = root(div(scale<2>(VVTP + VVTH), kPi) + DU2);
  const double UPM = root(div(scale<4>(VVTP), kPi) + 2.25 * kPi * VVTH + DU24);
  const double UHM = root(2.25 * kPi * VVTP + div(scale<4>(VVTH), kPi) + DU24);
  const double UPE = root(div(scale<2>(VVTP) + div(scale<6>(VVTH), 9.0), kPi) + DU2);
  const double UHE = root(div(div(scale<6>(VVTP), 9.0) + scale<2>(VVTH), kPi) + DU2);
  const double UDS = P.ce_scale_vel * UD;
  const double t = P.ce_a - P.ce_b * log(UDS);
  double SIG = t * t;
  if (P.ce_damp_c > 0.0) SIG = SIG * pow(1.0 - exp(-P.ce_damp_c / UDS), P.ce_damp_pow);
  SIG = P.ce_sigma_scale * SIG;
  const double ARR = SIG * rhoN * rho;
  const double VVTHU = div(VVTH, UPM);
  const double hs = UD + VVTHU + div(VVTP, UHM);
  c.shared[0] = ARR * dx_ * hs;
  c.shared[1] = ARR * dy_ * hs;
  c.shared[2] = ARR * dz_ * hs;
  c.shared[3] = half(ARR) * (1.5 * (UHE * VVTP - UPE * VVTH) + UD * (U2 - UH2) +
                             scale<1>(VVTHU * VPHH + div(VVTP * VPHP, UHM)));
  c.shared[4] = ARR * UD;
  // -(uxN - ux) == ux - uxN exactly
  c.shared[5] = ARR * (ux * UD + div(dx_ * VVTP, UHM));
  c.shared[6] = ARR * (uy * UD + div(dy_ * VVTP, UHM));
  c.shared[7] = ARR * (uz * UD + div(dz_ * VVTP, UHM));
  c.shared[8] = ARR * (half(U2) * UD + VVTP * (div(VPHP, UHM) + 0.75 * UHE));
  c.pmi[0] = ARR * (uxN * UD - dx_ * VVTHU);
  c.pmi[1] = ARR * (uyN * UD - dy_ * VVTHU);
  c.pmi[2] = ARR * (uzN * UD - dz_ * VVTHU);
  c.enmi = ARR * (half(UH2) * UD - VPHH * VVTHU + 0.75 * VVTH * UPE);
}

// S = -dt H of the plasma (momentum and energy; the magnetic field's and
// psi's S is zero); h: h2..h5.
__device__ __forceinline__ void charge_exchange_source(double dt, double* u, const double* h) {
#pragma unroll
  for (int q = 0; q < 4; ++q) u[1 + q] = u[1 + q] + (-dt * h[q]);
}

// S = -dt H of a population with terms c; rec: it receives the newly created
// neutrals, density H1 and the plasma's totals plu (PPLUX, PPLUY, PPLUZ, ENPLU).
__device__ __forceinline__ void charge_exchange_source(bool rec, double H1, const double* plu,
                                                       const CeTerms& c, double dt, double* un) {
  un[0] = un[0] + (-dt * (rec ? H1 : c.shared[4]));
#pragma unroll
  for (int q = 0; q < 3; ++q)
    un[1 + q] = un[1 + q] + (-dt * (rec ? plu[q] + c.pmi[q] : c.pmi[q]));
  un[4] = un[4] + (-dt * (rec ? plu[3] + c.enmi : c.enmi));
}

// H1 of the recipient f (from 0) of nN populations; lost(q): ARR UD
// (-DENPLU) of population q.
template <typename L>
__device__ __forceinline__ double new_neutrals(int nN, int f, const L& lost) {
  double sum = 0.0;
  bool first = true;
#pragma unroll
  for (int q = 0; q < MF_MAX_FLUIDS - 1; ++q) {
    if (q < nN && (nN > 3 || q != f)) {
      sum = first ? -lost(q) : sum - lost(q);
      first = false;
    }
  }
  return (nN > 3) ? sum + lost(f) : sum;
}

// The same for a thread per fluid; at(f, q): CeTerms::shared[q] of population f.
template <int NN, typename AT>
__device__ __forceinline__ void charge_exchange_plasma(double dt, double* u, const AT& at) {
  double h[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    h[q] = 0.0;
#pragma unroll
    for (int f = 0; f < NN; ++f) h[q] = h[q] + at(f, q);
  }
  charge_exchange_source(dt, u, h);
}
template <int NN, typename WA, typename AT>
__device__ __forceinline__ void charge_exchange_neutral(bool rec, int f, const WA&,
                                                        const CeTerms& c, double dt, double* un,
                                                        const AT& at) {
  double H1 = 0.0, plu[4] = {0.0, 0.0, 0.0, 0.0};
  if (rec) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
#pragma unroll
      for (int e = 0; e < NN; ++e) plu[q] = plu[q] - at(e, 5 + q);
    }
    H1 = new_neutrals(NN, f, [&](int e) { return at(e, 4); });
  }
  charge_exchange_source(rec, H1, plu, c, dt, un);
}

// All populations of one cell by one thread.  T names the arithmetic type for
// interface symmetry with the fast physics; the parity physics is FP64 only.
// NN > 0: the number of populations fixed at compile time; 0: P.nf - 1.
template <int IRHON, typename T = double, typename WA = const double*, int NN = 0>
__device__ __forceinline__ void charge_exchange_add(const DevParams& P, const WA& w, int reg,
                                                    double dt, double* u) {
  static_assert(sizeof(T) == sizeof(double), "FP64 physics");
  const int nN = NN > 0 ? NN : P.nf - 1;
  CeTerms c[MF_MAX_FLUIDS - 1];
  double h[4] = {0.0, 0.0, 0.0, 0.0}, plu[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
  for (int f = 0; f < MF_MAX_FLUIDS - 1; ++f) {
    if (f < nN) {
      charge_exchange_terms(P, w, IRHON + f * 5, c[f]);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        h[q] = h[q] + c[f].shared[q];
        plu[q] = plu[q] - c[f].shared[5 + q];
      }
    }
  }
  charge_exchange_source(dt, u, h);
  const int rk = ce_recipient(nN, reg);
#pragma unroll
  for (int f = 0; f < MF_MAX_FLUIDS - 1; ++f) {
    if (f < nN) {
      const double H1 = new_neutrals(nN, f, [&](int e) { return c[e].shared[4]; });
      charge_exchange_source(f + 1 == rk, H1, plu, c[f], dt, u + IRHON + f * 5);
    }
  }
}

// SOURCE8WAVES (srcIdeal/PatchIdealMHDF.ChF:681-722) + ADDSOURCES
template <typename WA>
__device__ __forceinline__ void source_8wave(const WA& w, double divB, double dtbydx, double* u) {
  const double dB = -divB * dtbydx;
  const double Ux = w[1], Uy = w[2], Uz = w[3];
  const double Bx = kInv4Pi * w[5], By = kInv4Pi * w[6], Bz = kInv4Pi * w[7];
  u[1] = u[1] + dB * Bx;
  u[2] = u[2] + dB * By;
  u[3] = u[3] + dB * Bz;
  u[4] = u[4] + dB * (Bx * Ux + By * Uy + Bz * Uz);
  u[5] = u[5] + dB * Ux;
  u[6] = u[6] + dB * Uy;
  u[7] = u[7] + dB * Uz;
}

// HELIOREINIT_DEFAULT (swlism/HeliosphericPlasmaBCF.ChF:1435-1566) at time t
// (the stage's start time plus its dt), in the routine's order of
// operations; sunBmonopolar != 1: the bipolar field (sign by theta < thetaS)
// and the current-sheet surface iHCS (:1537-1564).
// The wind state of a cell inside the sphere.  Inlined: a call out of line
// would cost the whole calling kernel local-memory traffic.
static __device__ __host__ __forceinline__ void reinit_state(const ReinitIn P, double x,
                                                          double y, double z, double r2,
                                                          double t, ReinitState& o) {
  o.hcs = 0.0;
  double r = sqrt(r2);
  double rr = r / P.rint;
  double xy = sqrt(x * x + y * y);
  double cosT = z / r;
  double sinT = sqrt(1.0 - cosT * cosT);
  double cosF = x / xy;
  double sinF = y / xy;
  double rho = P.sun_rho / (rr * rr);
  double ux = P.sun_v * sinT * cosF;
  double uy = P.sun_v * sinT * sinF;
  double uz = P.sun_v * cosT;
  double pr = P.sun_p / pow(rr, 2.0 * P.gamma);
  double br = P.dir_br * P.sun_b / (rr * rr);
  double bp = -P.sun_beta * br * r * sinT;
  double bx = br * sinT * cosF - bp * sinF;
  double by = br * sinT * sinF + bp * cosF;
  double bz = br * cosT;
  double b = bx * bx + by * by + bz * bz;
  double e0 = pr / P.hgamma + 0.5 * (rho * P.sun_v * P.sun_v + kInv4Pi * b);
  if (!P.monopolar) {
    double theta = acos(cosT);
    // cos / sin of the spiral phase sunBeta (r - sunV t), through the phase
    // in units of pi (an exact argument reduction: no slow path for large
    // phases); the phase only places the current sheet
    double sinBr, cosBr;
    reinit_sincos(P.sun_beta * (r - P.sun_v * t), sinBr, cosBr);
    double sinB = sinF * cosBr + cosF * sinBr;
    double cosB = cosF * cosBr - sinF * sinBr;
    double thetaS = P.sin_tilt * sinB / sqrt((P.cos_tilt * cosB) * (P.cos_tilt * cosB) + sinB * sinB);
    thetaS = asin(thetaS) + 0.5 * kPi;
    if (!(theta < thetaS)) {
      bx = -bx;
      by = -by;
      bz = -bz;
    }
    o.hcs = (theta < thetaS) ? 1.0 : -1.0;
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

// The reset of one cell: the membership test, then the wind state.
__device__ __host__ __forceinline__ bool reinit_wind(const DevParams& P, double dx, int i, int j,
                                                     int k, double t, ReinitState& o) {
  double x = (i + 0.5) * dx - P.sun_c[0];
  double y = (j + 0.5) * dx - P.sun_c[1];
  double z = 0.0;
  if (P.sd == 3) z = (k + 0.5) * dx - P.sun_c[2];
  double r2 = (P.sd == 3) ? (x * x + y * y + z * z) : (x * x + y * y);
  if (!(r2 <= P.r0 * P.r0)) return false;
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
  const double hg = P.hgamma, smallR = P.smallr, smallP = P.smallp;
  if (P.nf == 1) {
    double Rho = u[0];
    bool was = false;
    if (lt(Rho, smallR)) { Rho = smallR; was = true; }
    double invRho = div(1.0, Rho);
    double Ux = u[1] * invRho, Uy = u[2] * invRho, Uz = u[3] * invRho;
    double BxB = kInv8Pi * (u[5] * u[5] + u[6] * u[6] + u[7] * u[7]);
    double UxU = half(Ux * Ux + Uy * Uy + Uz * Uz);
    double Pr = hg * (u[4] - BxB - Rho * UxU);
    if (lt(Pr, smallP)) { Pr = smallP; was = true; }
    if (was) {
      u[0] = Rho;
      u[4] = Pr / hg + Rho * UxU + BxB;
    }
    return;
  }
  {
    double Rho = u[0];
    double invRho = div(1.0, Rho);
    double Ux = u[1] * invRho, Uy = u[2] * invRho, Uz = u[3] * invRho;
    double BxB = kInv8Pi * (u[5] * u[5] + u[6] * u[6] + u[7] * u[7]);
    double UxU = half(Ux * Ux + Uy * Uy + Uz * Uz);
    double Pr = hg * (u[4] - BxB - Rho * UxU);
    bool was = false;
    if (lt(Rho, smallR)) { Rho = smallR; was = true; }
    if (lt(Pr, smallP)) { Pr = smallP; was = true; }
    if (was) {
      u[0] = Rho;
      u[1] = Rho * Ux;
      u[2] = Rho * Uy;
      u[3] = Rho * Uz;
      u[4] = Pr / hg + Rho * UxU + BxB;
    }
  }
}

// neutral fluid f (from 1)
__device__ __forceinline__ void positivity_neutral(const DevParams& P, int f, double* un) {
  using namespace ieee64;
  const double hg = P.hgamma, smallR = P.smallr, smallP = P.smallp;
  double fd = (f == 1) ? smallR : (f == 3) ? kNet3Dens : kNet2Dens;
  double fp = (f == 1) ? smallP : (f == 3) ? kNet3Pres : kNet2Pres;
  double Rho = un[0];
  double invRho = div(1.0, Rho);
  double Ux = un[1] * invRho, Uy = un[2] * invRho, Uz = un[3] * invRho;
  double UxU = half(Ux * Ux + Uy * Uy + Uz * Uz);
  double Pr = hg * (un[4] - Rho * UxU);
  bool was = false;
  if (lt(Rho, fd)) { Rho = fd; was = true; }
  if (lt(Pr, fp)) { Pr = fp; was = true; }
  if (was) {
    un[0] = Rho;
    un[1] = Rho * Ux;
    un[2] = Rho * Uy;
    un[3] = Rho * Uz;
    un[4] = Pr / hg + Rho * UxU;
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
// (srcIdeal/PatchEulerF.ChF:5-50) of one cell.
template <typename T = double>
__device__ __forceinline__ double wave_speed_plasma(const DevParams& P, const double* u) {
  using namespace ieee64;
  double rho = u[0];
  double invrho = div(1.0, rho);
  double ru = u[1], rv = u[2], rw = u[3];
  double uu = ru * invrho, vv = rv * invrho, ww = rw * invrho;
  double ke = ru * uu + rv * vv + rw * ww;
  double bx = u[5], by = u[6], bz = u[7];
  double b = kInv4Pi * (bx * bx + by * by + bz * bz);
  double p = P.hgamma * (u[4] - half(ke + b));
  p = maxnum(p, P.smallp);
  double a2 = P.gamma * p * invrho;
  double as2 = half(a2 + invrho * b);
  double as4 = as2 * as2;
  double bn2 = kInv4Pi * bx * bx * invrho;
  double umax = absval(uu) + root(as2 + root(as4 - a2 * bn2));
  bn2 = kInv4Pi * by * by * invrho;
  umax = maxnum(absval(vv) + root(as2 + root(as4 - a2 * bn2)), umax);
  bn2 = kInv4Pi * bz * bz * invrho;
  return maxnum(absval(ww) + root(as2 + root(as4 - a2 * bn2)), umax);
}

template <typename T = double>
__device__ __forceinline__ double wave_speed_neutral(const DevParams& P, const double* un) {
  using namespace ieee64;
  double rho = maxnum(un[0], P.smallr);
  double invrho = div(1.0, rho);
  double ru = un[1], rv = un[2], rw = un[3];
  double uu = ru * invrho, vv = rv * invrho, ww = rw * invrho;
  double ke = ru * uu + rv * vv + rw * ww;
  double p = P.hgamma * (un[4] - half(ke));
  p = maxnum(p, P.smallp);
  double a = root(P.gamma * p * invrho);
  return maxnum(maxnum(absval(uu), absval(vv)), absval(ww)) + a;
}

template <int IRHON, typename T = double>
__device__ __forceinline__ double max_wave_speed(const DevParams& P, const double* u) {
  static_assert(sizeof(T) == sizeof(double), "FP64 physics");
  double cmax = ieee64::maxnum(wave_speed_plasma(P, u), 0.0);
#pragma unroll
  for (int f = 1; f < MF_MAX_FLUIDS; ++f)
    if (f < P.nf) cmax = ieee64::maxnum(wave_speed_neutral(P, u + IRHON + (f - 1) * 5), cmax);
  return cmax;
}

}  // namespace exact
}  // namespace mf
