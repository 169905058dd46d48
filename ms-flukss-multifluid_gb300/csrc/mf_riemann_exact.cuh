// mf_riemann_exact.cuh - face fluxes of the FP64 parity path: Roe 8/7-wave
// MHD, Rusanov MHD, Dedner (GLM) 2x2 and van Leer splitting, each written in
// the reference's evaluation order (every division and product as in the
// Fortran; structurally zero eigenmatrix entries skipped, which is exact).
// Compiled without multiply-add contraction, so each operation rounds as in
// the CPU restatement.
#pragma once

#include "mf_device.cuh"

// Each product that a sum takes in is written mad(a, b, c) = a b + c or
// nmad(a, b, c) = c - a b.  The parity path (namespace exact) rounds the
// product and the sum; a unit that names another namespace in MF_RIEMANN_NS
// (the fast FP64 path) gets them fused, in the same places in every kernel.
// There a difference that is >= 0 exactly can round below 0, and its root
// takes 0.
#ifdef MF_RIEMANN_NS
#define MF_RIEMANN_FUSED 1
#else
#define MF_RIEMANN_NS exact
#define MF_RIEMANN_FUSED 0
#endif

namespace mf {
namespace MF_RIEMANN_NS {

__device__ __forceinline__ double mad(double a, double b, double c) {
  return MF_RIEMANN_FUSED ? fma(a, b, c) : a * b + c;
}
__device__ __forceinline__ double nmad(double a, double b, double c) {
  return MF_RIEMANN_FUSED ? fma(-a, b, c) : c - a * b;
}
__device__ __forceinline__ double radicand(double x) {
  return MF_RIEMANN_FUSED ? ieee64::maxnum(0.0, x) : x;
}

// ---------------------------------------------------------------------------
// Roe 8-wave / 7-wave MHD flux: RIEMANNF (src/Roe8WaveF.ChF:5-601) and
// RIEMANN7F (src/Roe7WaveF.ChF:5-558).  wl/wr: rho,u,v,w,p,bx,by,bz in the
// global frame; g: fluxes in the same order.  SEVEN drops the normal-B wave
// (RIEMANN7F), whose normal-B flux is zero.
//
// Bound by the FP64 pipe, so everything else goes to the integer pipes
// (mf_ieee64.cuh): divisions, roots, comparisons, signs and the factors 1/2
// and 1/4.  Those factors and the signs are moved through the products they
// stand in (exact: a power of two scales without rounding), which leaves one
// product where the Fortran's coefficients repeat it with another factor:
// e.g. so53 = -0.5 als as hyy sih / cc and sp35 = -als as hyy sih both come
// from q1 = als as hyy.  The mirrored rows (fast and slow pairs) share their
// partial sums: (-a) + (-b) = -(a + b) exactly.
// ---------------------------------------------------------------------------
template <typename R, int DIR, bool SEVEN>
__device__ __forceinline__ void roe_mhd(const DevParams& P, const R* wl, const R* wr, R* g) {
  static_assert(sizeof(R) == sizeof(double), "FP64 physics");
  using namespace ieee64;
  constexpr int in = 1 + DIR, it1 = 1 + (DIR + 1) % 3, it2 = 1 + (DIR + 2) % 3;
  constexpr int inB = 5 + DIR, it1B = 5 + (DIR + 1) % 3, it2B = 5 + (DIR + 2) % 3;
  const double gamma = P.gamma, hgamma = P.hgamma;
  const double smallp = P.smallp, smallr = P.smallr;
  const double i4pi = kInv4Pi, i8pi = kInv8Pi, sq2 = kSqrtHalf;

  const double PGasL = maxnum(smallp, wl[4]), RhoL = maxnum(smallr, wl[0]);
  const double UL = wl[in], VL = wl[it1], WL = wl[it2];
  const double BXL = wl[inB], BYL = wl[it1B], BZL = wl[it2B];
  const double PGasR = maxnum(smallp, wr[4]), RhoR = maxnum(smallr, wr[0]);
  const double UR = wr[in], VR = wr[it1], WR = wr[it2];
  const double BXR = wr[inB], BYR = wr[it1B], BZR = wr[it2B];

  const double RUL = RhoL * UL, RVL = RhoL * VL, RWL = RhoL * WL;
  const double BxBL = i8pi * mad(BZL, BZL, mad(BYL, BYL, BXL * BXL));
  const double RUxUL = half(mad(RWL, WL, mad(RVL, VL, RUL * UL)));
  const double PL = PGasL + BxBL;
  const double EL = div(PGasL, hgamma) + RUxUL + BxBL;
  const double AL2 = div(gamma * PGasL, RhoL);

  const double RUR = RhoR * UR, RVR = RhoR * VR, RWR = RhoR * WR;
  const double BxBR = i8pi * mad(BZR, BZR, mad(BYR, BYR, BXR * BXR));
  const double RUxUR = half(mad(RWR, WR, mad(RVR, VR, RUR * UR)));
  const double PR = PGasR + BxBR;
  const double ER = div(PGasR, hgamma) + RUxUR + BxBR;
  const double AR2 = div(gamma * PGasR, RhoR);

  const bool wide = lt(AR2, AL2);
  const double ccmi = wide ? AR2 : AL2, ccma = wide ? AL2 : AR2;

  double Rho, U, V, W, BX, BY, BZ, BX2, BYZ2, BxBH, kk, cc;
  if (P.aver == 1) {
    const double HL = div(EL + PL, RhoL), HR = div(ER + PR, RhoR);
    const double coefRL = div(1.0, 1.0 + root(div(RhoR, RhoL)));
    const double coefRR = 1.0 - coefRL;
    Rho = mad(RhoL, coefRR, RhoR * coefRL);
    U = mad(UR, coefRR, UL * coefRL);
    V = mad(VR, coefRR, VL * coefRL);
    W = mad(WR, coefRR, WL * coefRL);
    const double HAV = mad(HR, coefRR, HL * coefRL);
    BX = mad(BXL, coefRR, BXR * coefRL);
    BY = mad(BYL, coefRR, BYR * coefRL);
    BZ = mad(BZL, coefRR, BZR * coefRL);
    const double BXAV = half(BXL + BXR);
    BX2 = BXAV * BXAV;
    BYZ2 = mad(BZ, BZ, BY * BY);
    BxBH = i8pi * (BX2 + BYZ2);
    kk = half(mad(W, W, mad(V, V, U * U)));
    const double DBX = BXR - BXL, DBY = BYR - BYL, DBZ = BZR - BZL;
    const double X =
        div(i8pi * mad(DBZ, DBZ, mad(DBY, DBY, DBX * DBX)) * coefRL * coefRL, RhoL);
    cc = mad(2.0 - gamma, X, hgamma * (HAV - kk - div(i4pi * mad(BX, BXAV, BYZ2), Rho)));
  } else {
    Rho = half(RhoL + RhoR);
    U = half(UL + UR);
    V = half(VL + VR);
    W = half(WL + WR);
    BX = half(BXL + BXR);
    BY = half(BYL + BYR);
    BZ = half(BZL + BZR);
    const double Pav = half(PL + PR);
    BX2 = BX * BX;
    BYZ2 = mad(BZ, BZ, BY * BY);
    BxBH = i8pi * (BX2 + BYZ2);
    kk = half(mad(W, W, mad(V, V, U * U)));
    const double PGas = Pav - BxBH;
    cc = div(gamma * PGas, Rho);
  }

  const double bb = div(i4pi * BX2, Rho);
  const double b = root(bb);
  if (lt(cc, ccmi)) cc = ccmi;
  if (lt(ccma, cc)) cc = ccma;
  const double c = root(cc);

  double hyy, hzz, aaf, aas, af, as;
  if (lt(BYZ2, P.smallB2)) {
    hyy = sq2;
    hzz = sq2;
    const bool alfven = lt(cc, bb);
    aaf = alfven ? bb : cc;
    aas = alfven ? cc : bb;
    af = alfven ? b : c;
    as = alfven ? c : b;
  } else {
    const double hyz = root(BYZ2);
    hyy = div(BY, hyz);
    hzz = div(BZ, hyz);
    const double szb = cc + div(scale<1>(BxBH), Rho);
    const double h = root(radicand(nmad(scale<2>(cc), bb, szb * szb)));
    aas = half(szb - h);
    const bool gone = le(aas, 0.0), capped = le(cc, aas);
    as = root(gone | capped ? 0.0 : aas);
    if (capped) { aas = cc; as = c; }
    if (gone) { aas = 0.0; as = 0.0; }
    aaf = half(szb + h);
    const bool low = le(aaf, cc);
    af = root(low ? 0.0 : aaf);
    if (low) { aaf = cc; af = c; }
  }

  // entropy-fixed speeds (Roe8 numbering: 1 entropy, 2 div-B, 3/4 Alfven,
  // 5/6 fast, 7/8 slow)
  const double eigmax = absval(U) + absval(V) + absval(W) + af;
  const double del = P.del2 * eigmax;
  const double dell2 = del * del;
  auto fix = [&](double e) -> double {
    const double z = absval(e);
    if (le(del, z)) return z;
    return div(half(mad(z, z, dell2)), del);
  };
  const double A1 = fix(U);
  const double A2 = A1;
  const double A3 = fix(U + b), A4 = fix(U - b);
  const double A5 = fix(U + af), A6 = fix(U - af);
  const double A7 = fix(U + as), A8 = fix(U - as);

  double alf, als;
  const double dfs = aaf - aas;
  const double dcs = cc - aas, dfc = aaf - cc;
  if (lt(dfs, 1.0e-8)) { alf = 1.0; als = 0.0; }
  else if (le(dcs, 0.0)) { alf = 0.0; als = 1.0; }
  else if (le(dfc, 0.0)) { alf = 1.0; als = 0.0; }
  else { alf = root(div(dcs, dfs)); als = root(div(dfc, dfs)); }

  // the sign bit of sih: clear where BX >= 0
  const uint32_t sih = le(0.0, BX) ? 0u : 0x80000000u;

  const double fl1 = RUL;
  const double fl2 = nmad(BXL * BXL, i4pi, UL * RUL) + PL;
  const double fl3 = nmad(BXL * BYL, i4pi, UL * RVL);
  const double fl4 = nmad(BXL * BZL, i4pi, UL * RWL);
  const double fl5 =
      nmad(BXL * mad(WL, BZL, mad(VL, BYL, UL * BXL)), i4pi, UL * (EL + PL));
  const double fl7 = nmad(BXL, VL, UL * BYL);
  const double fl8 = nmad(BXL, WL, UL * BZL);
  const double fr1 = RUR;
  const double fr2 = nmad(BXR * BXR, i4pi, UR * RUR) + PR;
  const double fr3 = nmad(BXR * BYR, i4pi, UR * RVR);
  const double fr4 = nmad(BXR * BZR, i4pi, UR * RWR);
  const double fr5 =
      nmad(BXR * mad(WR, BZR, mad(VR, BYR, UR * BXR)), i4pi, UR * (ER + PR));
  const double fr7 = nmad(BXR, VR, UR * BYR);
  const double fr8 = nmad(BXR, WR, UR * BZR);

  const double du1 = RhoL - RhoR;
  double du2 = RUL - RUR;
  double du3 = RVL - RVR;
  double du4 = RWL - RWR;
  double du5 = EL - ER;
  const double du6 = BXL - BXR;
  const double du7 = BYL - BYR;
  const double du8 = BZL - BZR;
  const double bdb = mad(BZ, du8, SEVEN ? BY * du7 : mad(BY, du7, BX * du6));
  du5 = -hgamma *
        mad(bdb, i4pi, mad(W, du4, mad(V, du3, mad(U, du2, -kk * du1))) - du5);
  du2 = div(nmad(U, du1, du2), Rho);
  du3 = div(nmad(V, du1, du3), Rho);
  du4 = div(nmad(W, du1, du4), Rho);

  const double sqPiRho = root(kPi * Rho);
  const double sq2PiRho = root(k2Pi * Rho);

  // products that the eigenvectors share
  const double p1 = alf * af, p2 = als * as;
  const double q1 = p2 * hyy, q2 = p2 * hzz, q3 = p1 * hyy, q4 = p1 * hzz;
  const double ccr = cc * Rho, csq = c * sqPiRho;
  const double h7 = half(du7), h8 = half(du8);

  const double lu1 = A1 * nmad(div(1.0, cc), du5, du1);
  const double lu2 = A2 * du6;
  const double s33 = hzz * sq2, s34 = hyy * sq2;
  const double e34 = nmad(s33, du3, s34 * du4);
  const double d37 = flip(div(hzz, sq2PiRho), sih), d38 = flip(div(hyy, sq2PiRho), sih);
  const double lu3 = A3 * nmad(d38, h8, mad(d37, h7, e34));
  const double lu4 = A4 * mad(d38, h8, nmad(d37, h7, e34));
  // twice the amplitudes of the fast and slow waves' common parts
  const double f234 = nmad(flip(div(q2, cc), sih), du4,
                           nmad(flip(div(q1, cc), sih), du3, div(p1, cc) * du2));
  const double x5 = div(alf, ccr), x7 = div(als * hyy, csq), x8 = div(als * hzz, csq);
  const double lu5 = half(A5 * mad(x8, h8, mad(x7, h7, mad(x5, du5, f234))));
  const double lu6 = half(A6 * mad(x8, h8, mad(x7, h7, mad(x5, du5, -f234))));
  const double g234 = mad(flip(div(q4, cc), sih), du4,
                          mad(flip(div(q3, cc), sih), du3, div(p2, cc) * du2));
  const double y5 = div(als, ccr), y7 = div(alf * hyy, csq), y8 = div(alf * hzz, csq);
  const double lu7 = half(A7 * nmad(y8, h8, nmad(y7, h7, mad(y5, du5, g234))));
  const double lu8 = half(A8 * nmad(y8, h8, nmad(y7, h7, mad(y5, du5, -g234))));

  // right eigenvectors (non-zero entries only)
  const double sp15 = Rho * alf, sp17 = Rho * als;
  double ra1 = mad(sp17, lu8, mad(sp17, lu7, mad(sp15, lu6, mad(sp15, lu5, lu1))));
  double ra2 = nmad(p2, lu8, mad(p2, lu7, nmad(p1, lu6, p1 * lu5)));
  const double r1 = flip(q1, sih), r2 = flip(q2, sih), r3 = flip(q3, sih), r4 = flip(q4, sih);
  double ra3 = nmad(r3, lu8, mad(r3, lu7, mad(r1, lu6, nmad(r1, lu5, nmad(s33, lu4, -(s33 * lu3))))));
  double ra4 = nmad(r4, lu8, mad(r4, lu7, mad(r2, lu6, nmad(r2, lu5, mad(s34, lu4, s34 * lu3)))));
  const double sp55 = sp15 * cc, sp57 = sp17 * cc;
  double ra5 = mad(sp57, lu8, mad(sp57, lu7, mad(sp55, lu6, sp55 * lu5)));
  const double ra6 = lu2;
  const double sp73 = flip(hzz * sq2PiRho, sih), sp84 = flip(hyy * sq2PiRho, sih);
  const double t5 = scale<1>(als * sqPiRho * c), t7 = scale<1>(alf * sqPiRho * c);
  const double sp75 = t5 * hyy, sp77 = t7 * hyy, sp85 = t5 * hzz, sp87 = t7 * hzz;
  const double ra7 =
      nmad(sp77, lu8, nmad(sp77, lu7, mad(sp75, lu6, mad(sp75, lu5, nmad(sp73, lu4, sp73 * lu3)))));
  const double ra8 =
      nmad(sp87, lu8, nmad(sp87, lu7, mad(sp85, lu6, mad(sp85, lu5, nmad(sp84, lu3, sp84 * lu4)))));

  const double bra = mad(BZ, ra8, SEVEN ? BY * ra7 : mad(BY, ra7, BX * ra6));
  ra5 = mad(i4pi, bra, mad(Rho, mad(W, ra4, mad(V, ra3, U * ra2)), ra1 * kk) + div(ra5, hgamma));
  ra2 = mad(Rho, ra2, U * ra1);
  ra3 = mad(Rho, ra3, V * ra1);
  ra4 = mad(Rho, ra4, W * ra1);

  g[0] = half(fl1 + fr1 + ra1);
  g[in] = half(fl2 + fr2 + ra2);
  g[it1] = half(fl3 + fr3 + ra3);
  g[it2] = half(fl4 + fr4 + ra4);
  g[4] = half(fl5 + fr5 + ra5);
  g[inB] = SEVEN ? 0.0 : half(ra6);
  g[it1B] = half(fl7 + fr7 + ra7);
  g[it2B] = half(fl8 + fr8 + ra8);
}

// RUSANOVF (src/RusanovF.ChF:4-197)
template <typename R, int DIR>
__device__ __forceinline__ void rusanov_mhd(const DevParams& P, const R* wl, const R* wr, R* g) {
  constexpr int in = 1 + DIR, it1 = 1 + (DIR + 1) % 3, it2 = 1 + (DIR + 2) % 3;
  constexpr int inB = 5 + DIR, it1B = 5 + (DIR + 1) % 3, it2B = 5 + (DIR + 2) % 3;
  const R gamma = R(P.gamma), hgamma = R(P.hgamma);
  const R i4pi = R(kInv4Pi), i8pi = R(kInv8Pi);
  R PGasL = rmax<R>(R(P.smallp), wl[4]), RhoL = rmax<R>(R(P.smallr), wl[0]);
  R UL = wl[in], VL = wl[it1], WL = wl[it2], BXL = wl[inB], BYL = wl[it1B], BZL = wl[it2B];
  R PGasR = rmax<R>(R(P.smallp), wr[4]), RhoR = rmax<R>(R(P.smallr), wr[0]);
  R UR = wr[in], VR = wr[it1], WR = wr[it2], BXR = wr[inB], BYR = wr[it1B], BZR = wr[it2B];
  R RUL = RhoL * UL, RVL = RhoL * VL, RWL = RhoL * WL;
  R BxBL = i8pi * (BXL * BXL + BYL * BYL + BZL * BZL);
  R RUxUL = R(0.5) * (RUL * UL + RVL * VL + RWL * WL);
  R PL = PGasL + BxBL;
  R EL = PGasL / hgamma + RUxUL + BxBL;
  R BXL_4PI = BXL * i4pi;
  R RUR = RhoR * UR, RVR = RhoR * VR, RWR = RhoR * WR;
  R BxBR = i8pi * (BXR * BXR + BYR * BYR + BZR * BZR);
  R RUxUR = R(0.5) * (RUR * UR + RVR * VR + RWR * WR);
  R PR = PGasR + BxBR;
  R ER = PGasR / hgamma + RUxUR + BxBR;
  R BXR_4PI = BXR * i4pi;
  R Rho, U, BX2, BxBH, A2;
  if (P.aver == 1) {
    R HL = (EL + PL) / RhoL, HR = (ER + PR) / RhoR;
    R coefRL = R(1) / (R(1) + sqrt_r<R>(RhoR / RhoL));
    R coefRR = R(1) - coefRL;
    Rho = RhoR * coefRL + RhoL * coefRR;
    U = UL * coefRL + UR * coefRR;
    R V = VL * coefRL + VR * coefRR;
    R W = WL * coefRL + WR * coefRR;
    R HAV = HL * coefRL + HR * coefRR;
    R BX = BXR * coefRL + BXL * coefRR;
    R BY = BYR * coefRL + BYL * coefRR;
    R BZ = BZR * coefRL + BZL * coefRR;
    R BXAV = R(0.5) * (BXL + BXR);
    BX2 = BXAV * BXAV;
    R BY2 = BY * BY, BZ2 = BZ * BZ;
    R BYZ2 = BY2 + BZ2;
    BxBH = i8pi * (BX2 + BYZ2);
    R kk = R(0.5) * (U * U + V * V + W * W);
    R DBX = BXR - BXL, DBY = BYR - BYL, DBZ = BZR - BZL;
    R X = i8pi * (DBX * DBX + DBY * DBY + DBZ * DBZ) * coefRL * coefRL / RhoL;
    A2 = hgamma * (HAV - kk - i4pi * (BX * BXAV + BYZ2) / Rho) + (R(2) - gamma) * X;
  } else {
    Rho = R(0.5) * (RhoL + RhoR);
    U = R(0.5) * (UL + UR);
    R BX = R(0.5) * (BXL + BXR), BY = R(0.5) * (BYL + BYR), BZ = R(0.5) * (BZL + BZR);
    R PGas = R(0.5) * (PGasL + PGasR);
    BX2 = BX * BX;
    R BY2 = BY * BY, BZ2 = BZ * BZ;
    BxBH = i8pi * (BX2 + BY2 + BZ2);
    A2 = gamma * PGas / Rho;
  }
  R bb = i4pi * BX2 / Rho;
  R szb = A2 + (BxBH + BxBH) / Rho;
  R h = sqrt_r<R>(radicand(szb * szb - R(4) * A2 * bb));
  R aaf = R(0.5) * (szb + h);
  R af = sqrt_r<R>(aaf);
  R em = rabs<R>(U) + af;
  g[0] = R(0.5) * (RUL + RUR + em * (RhoL - RhoR));
  g[in] = R(0.5) * ((UL * RUL - BXL_4PI * BXL + PL) + (UR * RUR - BXR_4PI * BXR + PR) + em * (RUL - RUR));
  g[it1] = R(0.5) * ((UL * RVL - BXL_4PI * BYL) + (UR * RVR - BXR_4PI * BYR) + em * (RVL - RVR));
  g[it2] = R(0.5) * ((UL * RWL - BXL_4PI * BZL) + (UR * RWR - BXR_4PI * BZR) + em * (RWL - RWR));
  g[4] = R(0.5) * ((UL * (EL + PL) - BXL_4PI * (UL * BXL + VL * BYL + WL * BZL)) +
                   (UR * (ER + PR) - BXR_4PI * (UR * BXR + VR * BYR + WR * BZR)) + em * (EL - ER));
  g[inB] = R(0.5) * (R(0) + R(0) + em * (BXL - BXR));
  g[it1B] = R(0.5) * ((UL * BYL - BXL * VL) + (UR * BYR - BXR * VR) + em * (BYL - BYR));
  g[it2B] = R(0.5) * ((UL * BZL - BXL * WL) + (UR * BZR - BXR * WR) + em * (BZL - BZR));
}

// DEDNER2X2F (src/DednerF.ChF:89-170): returns the Bn and psi fluxes.
template <typename R>
__device__ __forceinline__ void dedner_2x2(R ch, R bxl, R psil, R bxr, R psir, R& fbn, R& fpsi) {
  using namespace ieee64;
  const R ch2 = ch * ch;
  const R hc = div(0.5, ch);
  const R du1 = half(bxl - bxr), du2 = psil - psir;
  const R lu1 = ch * nmad(hc, du2, du1);
  const R lu2 = ch * mad(hc, du2, du1);
  const R ra1 = lu1 + lu2;
  const R ra2 = nmad(ch, lu1, ch * lu2);
  fbn = half(psil + psir + ra1);
  fpsi = half(mad(ch2, bxr, ch2 * bxl) + ra2);
}

// VANLEERF (src/VanLeerRSF.ChF:4-130): wl/wr = rho,u,v,w,p of one Euler fluid.
// Divisions, roots, comparisons and powers of two as in roe_mhd, and here the
// products that no sum takes in: with the warps that fit, the integer pipes
// have room for them (fluxes of three populations, 128^3: 6.04 -> 5.67 ms a
// step; in roe_mhd, whose chain is longer and warps are fewer, they cost as
// much as they save: 12.2 -> 12.1 ms).
template <typename R, int DIR>
__device__ __forceinline__ void vanleer_euler(const DevParams& P, const R* wl, const R* wr, R* g) {
  using namespace ieee64;
  constexpr int in = 1 + DIR, it1 = 1 + (DIR + 1) % 3, it2 = 1 + (DIR + 2) % 3;
  const R gamma = R(P.gamma), hgamma = R(P.hgamma);
  R fl1, fl2, fl3, fl4, fl5, fr1, fr2, fr3, fr4, fr5;
  const R PGasL = maxnum(P.smallp, wl[4]), RhoL = maxnum(P.smallr, wl[0]);
  const R UL = wl[in], VL = wl[it1], WL = wl[it2];
  const R RUL = mul(RhoL, UL), RVL = mul(RhoL, VL), RWL = mul(RhoL, WL);
  const R RUxUL = half(mad(RWL, WL, mad(RVL, VL, RUL * UL)));
  const R EL = div(PGasL, hgamma) + RUxUL;
  const R AL = root(div(gamma * PGasL, RhoL));
  if (le(UL, -AL)) {
    fr1 = fr2 = fr3 = fr4 = fr5 = R(0);
  } else if (le(AL, UL)) {
    fr1 = RhoL * UL;
    fr2 = mad(fr1, UL, PGasL);
    fr3 = mul(fr1, VL);
    fr4 = mul(fr1, WL);
    fr5 = UL * (EL + PGasL);
  } else {
    const R UA = div(scale<1>(AL) - UL, gamma);
    const R H = div(EL + PGasL, RhoL);
    const R HU = UL + AL;
    fr1 = scale<-2>(div(mul(mul(RhoL, HU), HU), AL));
    fr2 = fr1 * (UL + UA);
    fr3 = mul(fr1, VL);
    fr4 = mul(fr1, WL);
    fr5 = mul(fr1, H);
  }
  const R PGasR = maxnum(P.smallp, wr[4]), RhoR = maxnum(P.smallr, wr[0]);
  const R UR = wr[in], VR = wr[it1], WR = wr[it2];
  const R RUR = mul(RhoR, UR), RVR = mul(RhoR, VR), RWR = mul(RhoR, WR);
  const R RUxUR = half(mad(RWR, WR, mad(RVR, VR, RUR * UR)));
  const R ER = div(PGasR, hgamma) + RUxUR;
  const R AR = root(div(gamma * PGasR, RhoR));
  if (le(AR, UR)) {
    fl1 = fl2 = fl3 = fl4 = fl5 = R(0);
  } else if (le(UR, -AR)) {
    fl1 = RhoR * UR;
    fl2 = mad(fl1, UR, PGasR);
    fl3 = mul(fl1, VR);
    fl4 = mul(fl1, WR);
    fl5 = UR * (ER + PGasR);
  } else {
    const R UA = div(-UR - scale<1>(AR), gamma);
    const R H = div(ER + PGasR, RhoR);
    const R HU = UR - AR;
    fl1 = -scale<-2>(div(mul(mul(RhoR, HU), HU), AR));
    fl2 = fl1 * (UR + UA);
    fl3 = mul(fl1, VR);
    fl4 = mul(fl1, WR);
    fl5 = mul(fl1, H);
  }
  g[0] = fl1 + fr1;
  g[in] = fl2 + fr2;
  g[it1] = fl3 + fr3;
  g[it2] = fl4 + fr4;
  g[4] = fl5 + fr5;
}


}  // namespace MF_RIEMANN_NS
}  // namespace mf
