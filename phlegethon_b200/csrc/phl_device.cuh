// phl_device.cuh -- device building blocks of the explicit FV step: ghost-index mapping,
// LIM2ND reconstruction, Riemann solvers (LHLLC/HLLC/HLLD/LHLLD) and the Helmholtz EoS.
//
// Every function mirrors the operation order of the corresponding reference routine in
// source/source.F90 (line ranges in each comment) so that the FP64 path, compiled without FMA
// contraction, reproduces the reference's rounding.  The same templates run in FP32 for the
// split-precision path (R = float), where the flux arithmetic is done on well-balanced
// deviations and only the state/EoS stay in FP64.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace phl {

constexpr double CONST_RGAS = 8.31446261815324e7;
constexpr double CONST_RAD = 7.565767381646406e-15;
constexpr double CONST_C = 2.99792458e10;
constexpr double CONST_C2 = 8.987551787368177e20;
constexpr double HELM_TOL = 1.0e-11;  // helm_tol (source.F90:754)
constexpr double EM15 = 1.0e-15;

enum { R_LHLLC = 0, R_HLLC = 1, R_HLLD = 2, R_LHLLD = 3 };
enum { BC_PERIODIC = 0, BC_REFLECTIVE = 1 };

// Unsigned division by a divisor fixed on the host: q = n m >> (31 + L) with L = ceil(log2 d) and
// m = floor(2^(31+L) / d) + 1, exact for n < 2^31 (m d exceeds 2^(31+L) by e <= d <= 2^L, and
// n e < 2^(31+L)).  A division by a run-time divisor is a ~20-instruction sequence, and every
// index decomposition has two: they were half of the instructions of the corner and face-B kernels.
struct FastDiv {
  unsigned d, m, s;
  static FastDiv by(unsigned div) {
    FastDiv f;
    unsigned L = 0;
    while ((1ull << L) < div) ++L;
    f.d = div;
    f.s = 31 + L;
    f.m = (unsigned)((1ull << f.s) / div + 1);
    return f;
  }
  __host__ __device__ __forceinline__ unsigned quot(unsigned n) const {
    return (unsigned)(((unsigned long long)n * m) >> s);
  }
};

// ------------------------------------------------------------------ grid description
struct Geo {
  int sdims, nx[3];
  long long N;        // interior cells
  int bc[3][2];
  double inv_dx[3];
  double gm, mu, cfl, mach_cutoff, mach_ct;
  // divisors of the index decompositions: nx[0], nx[0] + 1 and nx[1], nx[1] + 1
  FastDiv div0[2], div1[2];
  int bg_profile;     // 1: background fields stored as profiles along x2
  int all_mach;       // FLUX_IS_ALL_MACH: LHLLC / LHLLD take the upwind state outside the wave fan
  int use_acc;        // USE_CONSTANT_ACCELERATION with the vector acc
  double acc[3];
};

// USE_CONSTANT_ACCELERATION (source.F90:12806-12836): body force rho a on the momenta and its
// work on the energy, from the current RK state u (before the stage's combine), subtracted from
// the residual in the reference's order
template <int DIM, int IP>
__device__ __forceinline__ void constant_acceleration(const Geo &g, const double *u, double *res) {
  const double rho = u[0];
#pragma unroll
  for (int d = 0; d < DIM; ++d) res[1 + d] = res[1 + d] - rho * g.acc[d];
  double r = res[IP];
  if (DIM == 3) r = r - u[3] * g.acc[2];
  r = r - u[1] * g.acc[0];
  r = r - u[2] * g.acc[1];
  res[IP] = r;
}

// Map a (possibly ghost) 0-based index along dimension d to its interior image.
// Periodic: wrap; reflective: mirror (ghost -1 <- 0, -2 <- 1), flip set.  The composition over
// dimensions equals communicate_ndarray (with corners) followed by the reflective BC loops
// (source.F90:2293-2306, 7532-7958).
__device__ __forceinline__ int map_index(int i, int n, int bcl, int bcu, bool &flip) {
  if (i < 0) {
    if (bcl == BC_PERIODIC) return i + n;
    flip = true;  // velocity / B component along this dimension changes sign
    return -1 - i;
  }
  if (i >= n) {
    if (bcu == BC_PERIODIC) return i - n;
    flip = true;
    return 2 * n - 1 - i;
  }
  return i;
}

// (i, j, k) of a linear index t = i + n0 * (j + n1 * k) with 32-bit unsigned division (index
// spaces stay below 2^32, checked at phl_init; 64-bit division is a long software sequence)
__device__ __forceinline__ void unflatten3(long long t, int n0, int n1, int &i, int &j, int &k) {
  const unsigned u = (unsigned)t, q = u / (unsigned)n0, r = q / (unsigned)n1;
  i = (int)(u - q * (unsigned)n0);
  j = (int)(q - r * (unsigned)n1);
  k = (int)r;
}

// the same with host-prepared divisors; index spaces of 2^31 and more do not fit device memory
__device__ __forceinline__ void unflatten3(long long t, const FastDiv &d0, const FastDiv &d1, int &i, int &j, int &k) {
  const unsigned u = (unsigned)t, q = d0.quot(u), r = d1.quot(q);
  i = (int)(u - q * d0.d);
  j = (int)(q - r * d1.d);
  k = (int)r;
}

// index spaces stay below 2^32 (checked at phl_init), so linear indices are formed in 32 bits and
// widened once
__device__ __forceinline__ long long lin3(int n0, int n1, int i, int j, int k) {
  return (long long)((unsigned)i + (unsigned)n0 * ((unsigned)j + (unsigned)n1 * (unsigned)k));
}
__device__ __forceinline__ long long lin(const Geo &g, int i, int j, int k) { return lin3(g.nx[0], g.nx[1], i, j, k); }

// ------------------------------------------------------------------ reconstructions
enum { REC_LIM2ND = 0, REC_PPH = 1, REC_LIM5TH = 2 };
// Edge values of the centre cell qc (lo = left edge, hi = right edge) from its neighbours:
// PPH_REC (source.F90:8183-8259; third order, limited only when `limited`, i.e. for the
// advected scalars) and LIM5TH_REC (source.F90:8261-8323; fifth order, always limited), with
// the reference's limiter and operation order.  LIM2ND_REC is plm below.
template <typename R, int REC>
__device__ __forceinline__ void rec_edges(bool limited, R qmm, R qm, R qc, R qp, R qpp, R &lo, R &hi) {
  R am, ap;
  if (REC == REC_PPH) {
    R tmp = R(5.0 / 6.0) * qc;
    am = R(1.0 / 3.0) * qm + tmp - R(1.0 / 6.0) * qp;
    ap = -R(1.0 / 6.0) * qm + tmp + R(1.0 / 3.0) * qp;
    if (!limited) {
      lo = am;
      hi = ap;
      return;
    }
  } else {
    R tmp = R(329) * qc;
    am = (-R(21) * qmm + R(189) * qm + tmp - R(91) * qp + R(14) * qpp) * R(1.0 / 420.0);
    ap = (R(14) * qmm - R(91) * qm + tmp + R(189) * qp - R(21) * qpp) * R(1.0 / 420.0);
  }
  R mn = fmin(qm, qc), mx = fmax(qm, qc);
  if (am < mn) am = mn;
  if (am > mx) am = mx;
  mn = fmin(qc, qp);
  mx = fmax(qc, qp);
  if (ap < mn) ap = mn;
  if (ap > mx) ap = mx;
  am = am - qc;
  ap = ap - qc;
  if (ap * am >= R(0)) {
    ap = R(0);
    am = R(0);
  } else {
    if (fabs(ap) >= R(2) * fabs(am)) ap = -R(2) * am;
    if (fabs(am) >= R(2) * fabs(ap)) am = -R(2) * ap;
  }
  lo = am + qc;
  hi = ap + qc;
}

// ------------------------------------------------------------------ LIM2ND reconstruction
// source.F90:8141-8181: slope = df*db/(df+db) if df*db > 0 else 0; faces at qc -/+ slope/2.
template <typename R>
__device__ __forceinline__ void plm(R qm, R qc, R qp, R &lo, R &hi) {
  R slopef = qp - qc, slopeb = qc - qm;
  R prod = slopef * slopeb;
  R slope = R(0);
  if (prod > R(0)) slope = prod / (slopef + slopeb);
  R tmp = R(0.5) * slope;
  lo = qc - tmp;
  hi = qc + tmp;
}

template <typename R>
__device__ __forceinline__ R sgn1(R x) { return copysign(R(1), x); }

// ------------------------------------------------------------------ hydro Riemann
// qL/qR: [rho, v1, v2, (v3), p, scalars...] in the normal frame.  Side thermodynamics by EOSM:
// EOS_IDEAL gamma-law; EOS_FAST gL/gR = (gammae, gammac) (USE_FASTEOS); EOS_GIVEN gL/gR =
// (rho*e, sound speed) already evaluated by helm_rhoP_given (Helmholtz without USE_FASTEOS,
// source.F90:15777-15781).  LHLLC source.F90:15681-16122 (Minoshima & Miyoshi low-dissipation
// pressure), HLLC source.F90:16124-16252.
enum { EOS_IDEAL = 0, EOS_FAST = 1, EOS_GIVEN = 2 };
template <typename R, int DIM, int NV, int EOSM, int RIEM>
__device__ __forceinline__ void riemann_hydro(const R *qL, const R *qR, const R *gL, const R *gR,
                                              R gm, R mach_cutoff, R *flux, bool flat = false,
                                              bool all_mach = false) {
  constexpr int IP = 1 + DIM, IAS = 2 + DIM;
  const R gmm1 = gm - R(1), igmm1 = R(1) / gmm1;
  R rhoL = qL[0], inv_rhoL = R(1) / rhoL, vx1L = qL[1], vx2L = qL[2], vx3L = DIM == 3 ? qL[3] : R(0);
  R v2L = vx1L * vx1L + vx2L * vx2L + vx3L * vx3L;
  R pL = qL[IP], eint, cL, cR;
  if (EOSM == EOS_FAST) { eint = pL / (gL[0] - R(1)); cL = sqrt(gL[1] * pL * inv_rhoL); }
  else if (EOSM == EOS_GIVEN) { eint = gL[0]; cL = gL[1]; }
  else { eint = igmm1 * pL; cL = sqrt(gm * pL * inv_rhoL); }
  R rhoeL = eint + R(0.5) * rhoL * v2L;
  R rhoR = qR[0], inv_rhoR = R(1) / rhoR, vx1R = qR[1], vx2R = qR[2], vx3R = DIM == 3 ? qR[3] : R(0);
  R v2R = vx1R * vx1R + vx2R * vx2R + vx3R * vx3R;
  R pR = qR[IP];
  if (EOSM == EOS_FAST) { eint = pR / (gR[0] - R(1)); cR = sqrt(gR[1] * pR * inv_rhoR); }
  else if (EOSM == EOS_GIVEN) { eint = gR[0]; cR = gR[1]; }
  else { eint = igmm1 * pR; cR = sqrt(gm * pR * inv_rhoR); }
  R rhoeR = eint + R(0.5) * rhoR * v2R;
  R max_c = fmax(cL, cR);
  R sL = fmin(vx1L, vx1R) - max_c;
  R sR = fmax(vx1L, vx1R) + max_c;
  R dsuL = sL - vx1L, dsuR = sR - vx1R;
  R ustar = (pR - pL + rhoL * vx1L * dsuL - rhoR * vx1R * dsuR) / (rhoL * dsuL - rhoR * dsuR);
  R rhostarL = rhoL * (dsuL / (sL - ustar));
  R rhoestarL = rhostarL * (rhoeL * inv_rhoL + (ustar - vx1L) * (ustar + pL * inv_rhoL / dsuL));
  R rhostarR = rhoR * (dsuR / (sR - ustar));
  R rhoestarR = rhostarR * (rhoeR * inv_rhoR + (ustar - vx1R) * (ustar + pR * inv_rhoR / dsuR));
  if (flat) {
    // two-wave HLL flux on a face next to a detected shock (USE_SHOCK_FLATTENING,
    // source.F90:15929-16010)
    sL = fmin(R(0), sL);
    sR = fmax(R(0), sR);
    R UL[NV], UR[NV], fL[NV], fR[NV];
    UL[0] = rhoL; UL[1] = rhoL * vx1L; UL[2] = rhoL * vx2L; if (DIM == 3) UL[3] = rhoL * vx3L; UL[IP] = rhoeL;
    UR[0] = rhoR; UR[1] = rhoR * vx1R; UR[2] = rhoR * vx2R; if (DIM == 3) UR[3] = rhoR * vx3R; UR[IP] = rhoeR;
    fL[0] = rhoL * vx1L; fL[1] = rhoL * vx1L * vx1L + pL; fL[2] = rhoL * vx1L * vx2L;
    if (DIM == 3) fL[3] = rhoL * vx1L * vx3L;
    fL[IP] = (rhoeL + pL) * vx1L;
    fR[0] = rhoR * vx1R; fR[1] = rhoR * vx1R * vx1R + pR; fR[2] = rhoR * vx1R * vx2R;
    if (DIM == 3) fR[3] = rhoR * vx1R * vx3R;
    fR[IP] = (rhoeR + pR) * vx1R;
#pragma unroll
    for (int iv = IAS; iv < NV; ++iv) {
      UL[iv] = rhoL * qL[iv];
      UR[iv] = rhoR * qR[iv];
      fL[iv] = UL[iv] * vx1L;
      fR[iv] = UR[iv] * vx1R;
    }
    const R dummy = R(1) / (sR - sL), phi = sL * sR;
#pragma unroll
    for (int iv = 0; iv < NV; ++iv) flux[iv] = dummy * (sR * fL[iv] - sL * fR[iv] + phi * (UR[iv] - UL[iv]));
    return;
  }
  if (RIEM == R_LHLLC) {
    R machL = sqrt(v2L) / cL, machR = sqrt(v2R) / cR;
    R chi = fmin(R(1), fmax(machL, machR));
    chi = fmax(mach_cutoff, chi);
    R phi = chi * (R(2) - chi);
    R rhobar = R(0.5) * (rhoL + rhoR), cbar = R(0.5) * (cL + cR);
    R pstar = R(0.5) * (pL + pR) - R(0.5) * phi * rhobar * cbar * (vx1R - vx1L);
    if (all_mach && (sL > R(0) || sR < R(0))) {
      // FLUX_IS_ALL_MACH: the upwind state's flux outside the wave fan (source.F90:16032-16077)
      const bool left = sL > R(0);
      const R *q = left ? qL : qR;
      R rho = left ? rhoL : rhoR, vx1 = left ? vx1L : vx1R, vx2 = left ? vx2L : vx2R, vx3 = left ? vx3L : vx3R;
      R p = left ? pL : pR, rhoe = left ? rhoeL : rhoeR;
      flux[0] = rho * vx1;
      flux[1] = rho * vx1 * vx1 + p;
      flux[2] = rho * vx1 * vx2;
      if (DIM == 3) flux[3] = rho * vx1 * vx3;
      flux[IP] = (rhoe + p) * vx1;
#pragma unroll
      for (int iv = IAS; iv < NV; ++iv) flux[iv] = rho * q[iv] * vx1;
      return;
    }
    R sgn = sgn1(ustar);
    R hp = R(0.5) * (R(1) + sgn), hm = R(0.5) * (R(1) - sgn);
    R rhostar = hp * rhostarL + hm * rhostarR;
    flux[0] = rhostar * ustar;
    flux[1] = rhostar * ustar * ustar + pstar;
    flux[2] = rhostar * ustar * (hp * vx2L + hm * vx2R);
    if (DIM == 3) flux[3] = rhostar * ustar * (hp * vx3L + hm * vx3R);
    flux[IP] = (hp * rhoestarL + hm * rhoestarR + pstar) * ustar;
#pragma unroll
    for (int iv = IAS; iv < NV; ++iv) flux[iv] = rhostar * ustar * (hp * qL[iv] + hm * qR[iv]);
  } else {
    const bool left = ustar > R(0);
    const R *q = left ? qL : qR;
    R rho = left ? rhoL : rhoR, vx1 = left ? vx1L : vx1R, vx2 = left ? vx2L : vx2R, vx3 = left ? vx3L : vx3R;
    R p = left ? pL : pR, rhoe = left ? rhoeL : rhoeR, rhostar = left ? rhostarL : rhostarR;
    R rhoestar = left ? rhoestarL : rhoestarR, s = left ? sL : sR;
    const bool sup = left ? (sL >= R(0)) : (sR < R(0));
    R U[NV], f[NV];
    U[0] = rho; U[1] = rho * vx1; U[2] = rho * vx2; if (DIM == 3) U[3] = rho * vx3; U[IP] = rhoe;
    f[0] = rho * vx1; f[1] = rho * vx1 * vx1 + p; f[2] = rho * vx1 * vx2;
    if (DIM == 3) f[3] = rho * vx1 * vx3;
    f[IP] = (rhoe + p) * vx1;
#pragma unroll
    for (int iv = IAS; iv < NV; ++iv) { U[iv] = rho * q[iv]; f[iv] = rho * vx1 * q[iv]; }
    if (sup) {
#pragma unroll
      for (int iv = 0; iv < NV; ++iv) flux[iv] = f[iv];
    } else {
      R Us[NV];
      Us[0] = rhostar; Us[1] = rhostar * ustar; Us[2] = rhostar * vx2; if (DIM == 3) Us[3] = rhostar * vx3;
      Us[IP] = rhoestar;
#pragma unroll
      for (int iv = IAS; iv < NV; ++iv) Us[iv] = rhostar * q[iv];
#pragma unroll
      for (int iv = 0; iv < NV; ++iv) flux[iv] = f[iv] + s * (Us[iv] - U[iv]);
    }
  }
}

// ------------------------------------------------------------------ MHD Riemann
// HLLD (Miyoshi & Kusano) source.F90:13969-15016, LHLLD source.F90:14364-14384, 14663-14732.
// b*: [Bn, Bt1, Bt2]; fluxb receives [0, Ft1, Ft2].
template <typename R, int DIM, int NV, int EOSM, int RIEM>
__device__ __forceinline__ void riemann_mhd(const R *qL, const R *qR, const R *bL, const R *bR,
                                            const R *gL, const R *gR, R gm, R mach_cutoff,
                                            R *flux, R *fluxb, bool flat = false, bool all_mach = false) {
  constexpr int IP = 1 + DIM, IAS = 2 + DIM;
  const R gmm1 = gm - R(1), igmm1 = R(1) / gmm1;
  R rhoL = qL[0], inv_rhoL = R(1) / rhoL, vx1L = qL[1], vx2L = qL[2], vx3L = DIM == 3 ? qL[3] : R(0);
  R v2L = vx1L * vx1L + vx2L * vx2L + vx3L * vx3L;
  R pL = qL[IP], eint, c2L, c2R;
  if (EOSM == EOS_FAST) { eint = pL / (gL[0] - R(1)); c2L = gL[1] * pL * inv_rhoL; }
  else if (EOSM == EOS_GIVEN) { eint = gL[0]; c2L = gL[1] * gL[1]; }
  else { eint = pL * igmm1; c2L = gm * pL * inv_rhoL; }
  R rhoeL = eint + R(0.5) * rhoL * v2L;
  R bx1L = bL[0], bx2L = bL[1], bx3L = DIM == 3 ? bL[2] : R(0);
  R rhoR = qR[0], inv_rhoR = R(1) / rhoR, vx1R = qR[1], vx2R = qR[2], vx3R = DIM == 3 ? qR[3] : R(0);
  R v2R = vx1R * vx1R + vx2R * vx2R + vx3R * vx3R;
  R pR = qR[IP];
  if (EOSM == EOS_FAST) { eint = pR / (gR[0] - R(1)); c2R = gR[1] * pR * inv_rhoR; }
  else if (EOSM == EOS_GIVEN) { eint = gR[0]; c2R = gR[1] * gR[1]; }
  else { eint = pR * igmm1; c2R = gm * pR * inv_rhoR; }
  R rhoeR = eint + R(0.5) * rhoR * v2R;
  R bx1R = bR[0], bx2R = bR[1], bx3R = DIM == 3 ? bR[2] : R(0);

  R bx1 = R(0.5) * (bx1L + bx1R), bx1_2 = bx1 * bx1;
  R pbL = R(0.5) * (bx1_2 + bx2L * bx2L + bx3L * bx3L);
  R pbR = R(0.5) * (bx1_2 + bx2R * bx2R + bx3R * bx3R);
  rhoeL = rhoeL + pbL;
  rhoeR = rhoeR + pbR;
  R ptL = pL + pbL, ptR = pR + pbR;
  R a2L = R(2) * pbL * inv_rhoL, a2R = R(2) * pbR * inv_rhoR;
  R an2L = bx1_2 * inv_rhoL, an2R = bx1_2 * inv_rhoR;
  R dummy = c2L + a2L;
  R cL = sqrt(R(0.5) * (c2L + a2L + sqrt(dummy * dummy - R(4) * c2L * an2L)));
  dummy = c2R + a2R;
  R cR = sqrt(R(0.5) * (c2R + a2R + sqrt(dummy * dummy - R(4) * c2R * an2R)));
  R max_c = fmax(cL, cR);
  R sL = fmin(vx1L, vx1R) - max_c;
  R sR = fmax(vx1L, vx1R) + max_c;
  R dsuL = sL - vx1L, dsuR = sR - vx1R;
  R inv_temp1 = R(1) / (dsuR * rhoR - dsuL * rhoL);
  R ustar = (dsuR * rhoR * vx1R - dsuL * rhoL * vx1L - ptR + ptL) * inv_temp1;
  R dsumL = sL - ustar, dsumR = sR - ustar;
  R phi = R(1);
  if (RIEM == R_LHLLD) {
    dummy = v2L + a2L;
    R cu2L = R(0.5) * (v2L + a2L + sqrt(dummy * dummy - R(4) * v2L * an2L));
    dummy = v2R + a2R;
    R cu2R = R(0.5) * (v2R + a2R + sqrt(dummy * dummy - R(4) * v2R * an2R));
    R machL = sqrt(cu2L) / cL, machR = sqrt(cu2R) / cR;
    R mm = fmax(machL, machR);
    if (mm < R(0.6)) {
      R chi = fmin(R(1), fmax(machL, machR));
      chi = fmax(mach_cutoff, chi);
      phi = chi * (R(2) - chi);
    } else {
      phi = R(1);
    }
  }
  if (flat) {
    // HLL flux on a flattened face (USE_SHOCK_FLATTENING, source.F90:14386-14495)
    sL = fmin(R(0), sL);
    sR = fmax(R(0), sR);
    R UL[NV], UR[NV], fL[NV], fR[NV];
    UL[0] = rhoL; UL[1] = rhoL * vx1L; UL[2] = rhoL * vx2L; if (DIM == 3) UL[3] = rhoL * vx3L; UL[IP] = rhoeL;
    UR[0] = rhoR; UR[1] = rhoR * vx1R; UR[2] = rhoR * vx2R; if (DIM == 3) UR[3] = rhoR * vx3R; UR[IP] = rhoeR;
    fL[0] = rhoL * vx1L; fL[1] = rhoL * vx1L * vx1L + ptL - bx1_2; fL[2] = rhoL * vx1L * vx2L - bx1 * bx2L;
    if (DIM == 3) fL[3] = rhoL * vx1L * vx3L - bx1 * bx3L;
    fL[IP] = (rhoeL + ptL) * vx1L - bx1 * (bx1 * vx1L + bx2L * vx2L + bx3L * vx3L);
    fR[0] = rhoR * vx1R; fR[1] = rhoR * vx1R * vx1R + ptR - bx1_2; fR[2] = rhoR * vx1R * vx2R - bx1 * bx2R;
    if (DIM == 3) fR[3] = rhoR * vx1R * vx3R - bx1 * bx3R;
    fR[IP] = (rhoeR + ptR) * vx1R - bx1 * (bx1 * vx1R + bx2R * vx2R + bx3R * vx3R);
#pragma unroll
    for (int iv = IAS; iv < NV; ++iv) {
      UL[iv] = rhoL * qL[iv];
      UR[iv] = rhoR * qR[iv];
      fL[iv] = UL[iv] * vx1L;
      fR[iv] = UR[iv] * vx1R;
    }
    const R UbL[3] = {bx1, bx2L, bx3L}, UbR[3] = {bx1, bx2R, bx3R};
    const R fbL[3] = {R(0), vx1L * bx2L - vx2L * bx1, vx1L * bx3L - vx3L * bx1};
    const R fbR[3] = {R(0), vx1R * bx2R - vx2R * bx1, vx1R * bx3R - vx3R * bx1};
    const R dh = R(1) / (sR - sL), ph = sL * sR;
#pragma unroll
    for (int iv = 0; iv < NV; ++iv) flux[iv] = dh * (sR * fL[iv] - sL * fR[iv] + ph * (UR[iv] - UL[iv]));
#pragma unroll
    for (int iv = 0; iv < DIM; ++iv) fluxb[iv] = dh * (sR * fbL[iv] - sL * fbR[iv] + ph * (UbR[iv] - UbL[iv]));
    return;
  }
  R pstar = (dsuR * rhoR * ptL - dsuL * rhoL * ptR - phi * rhoL * rhoR * dsuR * dsuL * (vx1L - vx1R)) * inv_temp1;
  R rhostarL = rhoL * dsuL / dsumL, rhostarR = rhoR * dsuR / dsumR;
  R a1_inv = R(1) / (rhoL * dsuL * dsumL - bx1_2);
  R vx2starL = vx2L - bx1 * bx2L * (ustar - vx1L) * a1_inv;
  R bx2starL = bx2L * (rhoL * dsuL * dsuL - bx1_2) * a1_inv;
  R vx3starL = vx3L - bx1 * bx3L * (ustar - vx1L) * a1_inv;
  R bx3starL = bx3L * (rhoL * dsuL * dsuL - bx1_2) * a1_inv;
  R a2_inv = R(1) / (rhoR * dsuR * dsumR - bx1_2);
  R vx2starR = vx2R - bx1 * bx2R * (ustar - vx1R) * a2_inv;
  R bx2starR = bx2R * (rhoR * dsuR * dsuR - bx1_2) * a2_inv;
  R vx3starR = vx3R - bx1 * bx3R * (ustar - vx1R) * a2_inv;
  R bx3starR = bx3R * (rhoR * dsuR * dsuR - bx1_2) * a2_inv;
  R vdotbL = vx1L * bx1 + vx2L * bx2L + vx3L * bx3L;
  R vdotbR = vx1R * bx1 + vx2R * bx2R + vx3R * bx3R;
  R vdotbstarL = ustar * bx1 + vx2starL * bx2starL + vx3starL * bx3starL;
  R vdotbstarR = ustar * bx1 + vx2starR * bx2starR + vx3starR * bx3starR;
  R rhoestarL = (dsuL * rhoeL - ptL * vx1L + pstar * ustar + bx1 * (vdotbL - vdotbstarL)) / dsumL;
  R rhoestarR = (dsuR * rhoeR - ptR * vx1R + pstar * ustar + bx1 * (vdotbR - vdotbstarR)) / dsumR;
  R sqrt_rhostarL = sqrt(rhostarL), sqrt_rhostarR = sqrt(rhostarR);
  R abs_bx1 = fabs(bx1);
  R sstarL = ustar - abs_bx1 / sqrt_rhostarL;
  R sstarR = ustar + abs_bx1 / sqrt_rhostarR;
  R inv_sqr_bar = R(1) / (sqrt_rhostarL + sqrt_rhostarR);
  R sgn = sgn1(bx1);
  R vx22star = (sqrt_rhostarL * vx2starL + sqrt_rhostarR * vx2starR + (bx2starR - bx2starL) * sgn) * inv_sqr_bar;
  R bx22star = (sqrt_rhostarL * bx2starR + sqrt_rhostarR * bx2starL +
                sqrt_rhostarL * sqrt_rhostarR * (vx2starR - vx2starL) * sgn) * inv_sqr_bar;
  R vx32star = (sqrt_rhostarL * vx3starL + sqrt_rhostarR * vx3starR + (bx3starR - bx3starL) * sgn) * inv_sqr_bar;
  R bx32star = (sqrt_rhostarL * bx3starR + sqrt_rhostarR * bx3starL +
                sqrt_rhostarL * sqrt_rhostarR * (vx3starR - vx3starL) * sgn) * inv_sqr_bar;
  R vdotb2star = ustar * bx1 + vx22star * bx22star + vx32star * bx32star;
  R rhoe2starL = rhoestarL - sqrt_rhostarL * (vdotbstarL - vdotb2star) * sgn;
  R rhoe2starR = rhoestarR + sqrt_rhostarR * (vdotbstarR - vdotb2star) * sgn;

  fluxb[0] = R(0);
  if (RIEM == R_LHLLD) {
    R rho, vx1, vx2, vx3, rhoe, bx2, bx3, pres = pstar;
    if (all_mach && sL > R(0)) {
      // FLUX_IS_ALL_MACH: the outer states as well (source.F90:14576-14632)
      rho = rhoL; vx1 = vx1L; vx2 = vx2L; vx3 = vx3L; rhoe = rhoeL; bx2 = bx2L; bx3 = bx3L; pres = ptL;
    } else if (sstarL > R(0)) {
      rho = rhostarL; vx1 = ustar; vx2 = vx2starL; vx3 = vx3starL; rhoe = rhoestarL; bx2 = bx2starL; bx3 = bx3starL;
    } else if (ustar > R(0)) {
      rho = rhostarL; vx1 = ustar; vx2 = vx22star; vx3 = vx32star; rhoe = rhoe2starL; bx2 = bx22star; bx3 = bx32star;
    } else if (sstarR > R(0)) {
      rho = rhostarR; vx1 = ustar; vx2 = vx22star; vx3 = vx32star; rhoe = rhoe2starR; bx2 = bx22star; bx3 = bx32star;
    } else if (!all_mach || sR > R(0)) {
      rho = rhostarR; vx1 = ustar; vx2 = vx2starR; vx3 = vx3starR; rhoe = rhoestarR; bx2 = bx2starR; bx3 = bx3starR;
    } else {
      rho = rhoR; vx1 = vx1R; vx2 = vx2R; vx3 = vx3R; rhoe = rhoeR; bx2 = bx2R; bx3 = bx3R; pres = ptR;
    }
    flux[0] = rho * vx1;
    flux[1] = rho * vx1 * vx1 + pres - bx1_2;
    flux[2] = rho * vx1 * vx2 - bx1 * bx2;
    if (DIM == 3) flux[3] = rho * vx1 * vx3 - bx1 * bx3;
    flux[IP] = (rhoe + pres) * vx1 - bx1 * (bx1 * vx1 + vx2 * bx2 + vx3 * bx3);
    R sg = sgn1(vx1), hp = R(0.5) * (R(1) + sg), hm = R(0.5) * (R(1) - sg);
#pragma unroll
    for (int iv = IAS; iv < NV; ++iv) flux[iv] = rho * vx1 * (hp * qL[iv] + hm * qR[iv]);
    fluxb[1] = vx1 * bx2 - bx1 * vx2;
    if (DIM == 3) fluxb[2] = vx1 * bx3 - bx1 * vx3;
    return;
  }
  const bool left = ustar > R(0);
  const R *q = left ? qL : qR;
  R rho = left ? rhoL : rhoR, vx1 = left ? vx1L : vx1R, vx2 = left ? vx2L : vx2R, vx3 = left ? vx3L : vx3R;
  R rhoe = left ? rhoeL : rhoeR, pt = left ? ptL : ptR, bx2 = left ? bx2L : bx2R, bx3 = left ? bx3L : bx3R;
  R vdotb = left ? vdotbL : vdotbR, rhostar = left ? rhostarL : rhostarR;
  R vx2s = left ? vx2starL : vx2starR, vx3s = left ? vx3starL : vx3starR;
  R bx2s = left ? bx2starL : bx2starR, bx3s = left ? bx3starL : bx3starR;
  R rhoes = left ? rhoestarL : rhoestarR, rhoe2s = left ? rhoe2starL : rhoe2starR;
  R s = left ? sL : sR, sst = left ? sstarL : sstarR;
  const bool outer = left ? (sL > R(0)) : (sR < R(0));
  const bool single = left ? (sstarL > R(0)) : (sstarR < R(0));
  constexpr int NB = DIM == 3 ? 3 : 2;
  R U[NV], f[NV], Ub[3], fb[3];
  U[0] = rho; U[1] = rho * vx1; U[2] = rho * vx2; if (DIM == 3) U[3] = rho * vx3; U[IP] = rhoe;
  f[0] = rho * vx1; f[1] = rho * vx1 * vx1 + pt - bx1_2; f[2] = rho * vx1 * vx2 - bx1 * bx2;
  if (DIM == 3) f[3] = rho * vx1 * vx3 - bx1 * bx3;
  f[IP] = (rhoe + pt) * vx1 - bx1 * vdotb;
#pragma unroll
  for (int iv = IAS; iv < NV; ++iv) { U[iv] = rho * q[iv]; f[iv] = rho * vx1 * q[iv]; }
  Ub[0] = bx1; Ub[1] = bx2; Ub[2] = bx3;
  fb[0] = R(0); fb[1] = vx1 * bx2 - bx1 * vx2; fb[2] = vx1 * bx3 - bx1 * vx3;
  if (outer) {
#pragma unroll
    for (int iv = 0; iv < NV; ++iv) flux[iv] = f[iv];
#pragma unroll
    for (int iv = 0; iv < NB; ++iv) fluxb[iv] = fb[iv];
    return;
  }
  R Us[NV], Ubs[3];
  Us[0] = rhostar; Us[1] = rhostar * ustar; Us[2] = rhostar * vx2s; if (DIM == 3) Us[3] = rhostar * vx3s;
  Us[IP] = rhoes;
#pragma unroll
  for (int iv = IAS; iv < NV; ++iv) Us[iv] = rhostar * q[iv];
  Ubs[0] = bx1; Ubs[1] = bx2s; Ubs[2] = bx3s;
  if (single) {
#pragma unroll
    for (int iv = 0; iv < NV; ++iv) flux[iv] = f[iv] + s * (Us[iv] - U[iv]);
#pragma unroll
    for (int iv = 0; iv < NB; ++iv) fluxb[iv] = fb[iv] + s * (Ubs[iv] - Ub[iv]);
    return;
  }
  R Uss[NV], Ubss[3];
  Uss[0] = rhostar; Uss[1] = rhostar * ustar; Uss[2] = rhostar * vx22star; if (DIM == 3) Uss[3] = rhostar * vx32star;
  Uss[IP] = rhoe2s;
#pragma unroll
  for (int iv = IAS; iv < NV; ++iv) Uss[iv] = rhostar * q[iv];
  Ubss[0] = bx1; Ubss[1] = bx22star; Ubss[2] = bx32star;
#pragma unroll
  for (int iv = 0; iv < NV; ++iv) {
    R d0 = Us[iv];
    flux[iv] = f[iv] + s * (d0 - U[iv]) + sst * (Uss[iv] - d0);
  }
#pragma unroll
  for (int iv = 0; iv < NB; ++iv) {
    R d0 = Ubs[iv];
    fluxb[iv] = fb[iv] + s * (d0 - Ub[iv]) + sst * (Ubss[iv] - d0);
  }
}

// ------------------------------------------------------------------ Helmholtz EoS
struct HelmTable {
  const double *tab;    // helm_table_var(1:9, 1:nrho, 1:nT)
  const double *dpdr;   // dpdrho_table_var(1:4, 1:nrho, 1:nT)
  const double *rho;    // helm_rho(1:nrho)
  const double *T;      // helm_T(1:nT)
  // reciprocal node spacings 1 / (helm_rho(i+1) - helm_rho(i)), 1 / (helm_T(j+1) - helm_T(j)),
  // index i-1 / j-1 (the same IEEE quotients a division at the point of use gives)
  const double *inv_drho, *inv_dT;
  int nrho, nT;
  double drho, dT, log10_rho1, log10_T1;  // log10(helm_rho(1)), log10(helm_T(1)) from the host
  double Tl, Th;
};

// ---- The FP64 evaluations below follow the reference operation by operation, so their results are
// its results to the last bit; what they leave out are operations whose result is already known.  Of
// a Newton iteration's twelve divisions and two double-precision logarithms one division remains:
// the density part (cell, bases, reciprocals) is formed once per solve, a table cell is found
// without a logarithm away from the nodes, and a quotient by a value with a known reciprocal takes
// five multiply-adds (div_by).  The FP64 pipe was busy 61% of the time in cons->prim (3,000 FP64
// instructions a cell), which ran 241 us on 96^3 cells.

// a / b correctly rounded from rb = RN(1 / b): two Newton steps on the quotient with exact residuals
// (Markstein, IBM J. Res. Dev. 34, 1990: with RN(1/b) and a faithful quotient the last step rounds
// correctly, and the first step makes the quotient faithful).  For finite a, b well inside the
// exponent range (HELM_LO .. HELM_HI below); callers divide plainly otherwise.
__device__ __forceinline__ double div_by(double a, double b, double rb) {
  double q = __dmul_rn(a, rb);
  q = __fma_rn(__fma_rn(-b, q, a), rb, q);
  return __fma_rn(__fma_rn(-b, q, a), rb, q);
}
constexpr double HELM_LO = 1.0e-30, HELM_HI = 1.0e60;
__device__ __forceinline__ bool helm_in_range(double x) { return x > HELM_LO && x < HELM_HI; }

// table node index (1-based like the reference) of x in the log-spaced nodes: an estimate in
// single precision (within one node of the cell for any x in the table's range), then exact
// comparisons against the node values
__device__ __forceinline__ int helm_node_estimate(int n, double log10_first, double dlog, double x) {
  const float lx = __log2f((float)x) * 0.30102999566398120f;
  const int i = (int)(__fdividef(lx - (float)log10_first, (float)dlog)) + 1;
  return max(1, min(i, n - 1));
}
__device__ __forceinline__ int helm_node_index(const double *nodes, int n, double log10_first, double dlog,
                                               double x) {
  int i = helm_node_estimate(n, log10_first, dlog, x);
  if (i < n - 1 && __ldg(nodes + i) <= x) ++i;
  if (i > 1 && __ldg(nodes + i - 1) > x) --i;
  return i;
}
// the reference's index (source.F90:23702-23709); the reference does not check the table's ends
static __device__ __noinline__ int helm_log_index(int n, double log10_first, double dlog, double x) {
  const int i = (int)((log10(x) - log10_first) / dlog) + 1;
  return max(1, min(i, n - 1));
}
// The same index without the logarithm: x more than HELM_EDGE (relative) inside the cell of its node
// index has the reference's index there (the logarithm, the nodes and the quotient are off by less
// than 1e-13 of a cell together); next to a node, outside the table or for NaN the logarithm decides.
// lo and up are the cell's nodes: two loads, a third where the estimate is one cell off (with the nodes
// read again by every user 2^22 energies took 351 us, now 287; reading the estimated cell's
// coefficients ahead of the comparison 383).
constexpr double HELM_EDGE = 1.0e-12;
__device__ __forceinline__ int helm_index(const double *nodes, int n, double log10_first, double dlog, double x,
                                          double &lo, double &up) {
  int i = helm_node_estimate(n, log10_first, dlog, x);
  lo = __ldg(nodes + i - 1);
  up = __ldg(nodes + i);
  if (up <= x && i < n - 1) {
    ++i;
    lo = up;
    up = __ldg(nodes + i);
  } else if (lo > x && i > 1) {
    --i;
    up = lo;
    lo = __ldg(nodes + i - 1);
  }
  if (x >= lo * (1.0 + HELM_EDGE) && x <= up * (1.0 - HELM_EDGE)) return i;
  i = helm_log_index(n, log10_first, dlog, x);
  lo = __ldg(nodes + i - 1);
  up = __ldg(nodes + i);
  return i;
}

// density part of an evaluation: table row, position in it, and the reciprocals the others divide by
struct HelmRho {
  int ih;
  bool ok;  // rho within the range of div_by
  double rho, irho, iabar, Ye, rhos, x, omx, drho, drho2;
};
__device__ __forceinline__ HelmRho helm_rho_part(const HelmTable &h, double rho, double abar, double zbar) {
  HelmRho r;
  r.rho = rho;
  r.irho = 1.0 / rho;
  r.ok = helm_in_range(rho);
  r.iabar = 1.0 / abar;
  r.Ye = zbar / abar;
  r.rhos = rho * r.Ye;
  double lo, up;
  r.ih = helm_index(h.rho, h.nrho, h.log10_rho1, h.drho, r.rhos, lo, up);
  r.drho = up - lo;
  r.x = (r.rhos - lo) / r.drho;
  r.omx = 1.0 - r.x;
  r.drho2 = r.drho * r.drho;
  return r;
}
// temperature part: the cell, kept while T stays inside it (lo <= T <= hi: HELM_EDGE off its nodes)
struct HelmTemp {
  int jh = 0;
  double T0, dT, idT, lo = 1.0, hi = 0.0, y, omy;
};
__device__ __forceinline__ void helm_temp_part(const HelmTable &h, double T, HelmTemp &t) {
  if (!(T >= t.lo && T <= t.hi)) {
    double up;
    t.jh = helm_index(h.T, h.nT, h.log10_T1, h.dT, T, t.T0, up);
    t.dT = up - t.T0;
    t.idT = __ldg(h.inv_dT + t.jh - 1);
    t.lo = t.T0 * (1.0 + HELM_EDGE);
    t.hi = up * (1.0 - HELM_EDGE);
  }
  const double a = T - t.T0;
  t.y = helm_in_range(T) ? div_by(a, t.dT, t.idT) : a / t.dT;
  t.omy = 1.0 - t.y;
}

// quintic Hermite bases (source.F90:24708-24738) and their derivatives
__device__ __forceinline__ void hb0(double x, double d, double d2, double b[3]) {
  double x2 = x * x, x3 = x2 * x, x4 = x3 * x, x5 = x4 * x;
  b[0] = -6.0 * x5 + 15.0 * x4 - 10.0 * x3 + 1.0;
  b[1] = (-3.0 * x5 + 8.0 * x4 - 6.0 * x3 + x) * d;
  b[2] = (0.5 * (-x5 + 3.0 * x4 - 3.0 * x3 + x2)) * d2;
}
__device__ __forceinline__ void hb0m(double om, double d, double d2, double b[3]) {
  double o2 = om * om, o3 = o2 * om, o4 = o3 * om, o5 = o4 * om;
  b[0] = -6.0 * o5 + 15.0 * o4 - 10.0 * o3 + 1.0;
  b[1] = (3.0 * o5 - 8.0 * o4 + 6.0 * o3 - om) * d;
  b[2] = (0.5 * (-o5 + 3.0 * o4 - 3.0 * o3 + o2)) * d2;
}
__device__ __forceinline__ void hb1(double x, double id, double d, double b[3]) {
  double x2 = x * x, x3 = x2 * x, x4 = x3 * x;
  b[0] = (-30.0 * x4 + 60.0 * x3 - 30.0 * x2) * id;
  b[1] = (-15.0 * x4 + 32.0 * x3 - 18.0 * x2 + 1.0);
  b[2] = (0.5 * (-5.0 * x4 + 12.0 * x3 - 9.0 * x2 + 2.0 * x)) * d;
}
__device__ __forceinline__ void hb1m(double om, double id, double d, double b[3]) {
  double o2 = om * om, o3 = o2 * om, o4 = o3 * om;
  b[0] = -(-30.0 * o4 + 60.0 * o3 - 30.0 * o2) * id;
  b[1] = (-15.0 * o4 + 32.0 * o3 - 18.0 * o2 + 1.0);
  b[2] = -(0.5 * (-5.0 * o4 + 12.0 * o3 - 9.0 * o2 + 2.0 * om)) * d;
}
__device__ __forceinline__ void hb2(double y, double id2, double id, double b[3]) {
  double y2 = y * y, y3 = y2 * y;
  b[0] = (-120.0 * y3 + 180.0 * y2 - 60.0 * y) * id2;
  b[1] = (-60.0 * y3 + 96.0 * y2 - 36.0 * y) * id;
  b[2] = (0.5 * (-20.0 * y3 + 36.0 * y2 - 18.0 * y + 2.0));
}
__device__ __forceinline__ void hb2m(double om, double id2, double id, double b[3]) {
  double o2 = om * om, o3 = o2 * om;
  b[0] = (-120.0 * o3 + 180.0 * o2 - 60.0 * om) * id2;
  b[1] = -(-60.0 * o3 + 96.0 * o2 - 36.0 * om) * id;
  b[2] = (0.5 * (-20.0 * o3 + 36.0 * o2 - 18.0 * om + 2.0));
}

// Sum over the 36 coefficients in loc_eos1..36 order, left to right.  The rho-order and T-order
// of the 9 table variables (id_f .. id_d4fdrho2dT2, source.F90:520-528) are
// rho: 0,0,0,1,2,1,2,1,2 and T: 0,1,2,0,0,1,1,2,2.
__device__ __forceinline__ double helm_sum36(const double c[36], const double r0[3], const double r1[3],
                                             const double t0[3], const double t1[3]) {
  double s = 0.0;
#pragma unroll
  for (int v = 0; v < 9; ++v) {
    const int orr = v < 3 ? 0 : ((v & 1) ? 1 : 2);   // matches HELM_ORD_R
    const int ort = v == 0 ? 0 : (v == 1 ? 1 : (v == 2 ? 2 : (v <= 4 ? 0 : (v <= 6 ? 1 : 2))));
    double a = (c[4 * v + 0] * r0[orr]) * t0[ort];
    double b = (c[4 * v + 1] * r1[orr]) * t0[ort];
    double cc = (c[4 * v + 2] * r0[orr]) * t1[ort];
    double d = (c[4 * v + 3] * r1[orr]) * t1[ort];
    if (v == 0) s = a; else s = s + a;
    s = s + b;
    s = s + cc;
    s = s + d;
  }
  return s;
}

__device__ __forceinline__ void helm_load36(const HelmTable &h, int ih, int jh, double c[36]) {
  const double *p00 = h.tab + 9 * ((long long)(ih - 1) + (long long)h.nrho * (jh - 1));
  const double *p10 = p00 + 9;
  const double *p01 = p00 + 9 * (long long)h.nrho;
  const double *p11 = p01 + 9;
#pragma unroll
  for (int v = 0; v < 9; ++v) {
    c[4 * v + 0] = __ldg(p00 + v);
    c[4 * v + 1] = __ldg(p10 + v);
    c[4 * v + 2] = __ldg(p01 + v);
    c[4 * v + 3] = __ldg(p11 + v);
  }
}

// helm_rhoT_given2 (source.F90:24571-24941): E and dE/dT; r0, r1 the density bases of the row
__device__ __forceinline__ void helm_rho_bases(const HelmRho &r, double r0[3], double r1[3]) {
  hb0(r.x, r.drho, r.drho2, r0);
  hb0m(r.omx, r.drho, r.drho2, r1);
}
template <bool DERIV>
__device__ __forceinline__ void helm_energy(const HelmTable &h, const HelmRho &r, const double r0[3],
                                            const double r1[3], HelmTemp &t, double T, double &E, double &dEdT) {
  helm_temp_part(h, T, t);
  double c[36];
  helm_load36(h, r.ih, t.jh, c);
  const double dT2 = t.dT * t.dT;
  double t0[3], t1[3];
  hb0(t.y, t.dT, dT2, t0);
  hb0m(t.omy, t.dT, dT2, t1);
  double f = helm_sum36(c, r0, r1, t0, t1);
  double d0[3], d1[3];
  hb1(t.y, t.idT, t.dT, d0);
  hb1m(t.omy, t.idT, t.dT, d1);
  double df_dT = helm_sum36(c, r0, r1, d0, d1);
  double df_dT2 = 0.0;
  if (DERIV) {
    const double idT2 = t.idT * t.idT;
    double e0[3], e1[3];
    hb2(t.y, idT2, t.idT, e0);
    hb2m(t.omy, idT2, t.idT, e1);
    df_dT2 = helm_sum36(c, r0, r1, e0, e1);
  }
  const bool safe = r.ok && helm_in_range(T);
  double s = -r.Ye * df_dT;
  double e = r.Ye * f + T * s;
  double T2 = T * T, T3 = T2 * T, T4 = T3 * T;
  const double aT4 = CONST_RAD * T4;
  e = e + 1.5 * CONST_RGAS * T * r.iabar + (safe ? div_by(aT4, r.rho, r.irho) : aT4 / r.rho);
  E = e;
  if (DERIV) {
    double ds_dT = -r.Ye * df_dT2;
    double de = T * ds_dT;
    const double aT3 = 4.0 * CONST_RAD * T3;
    dEdT = de + 1.5 * CONST_RGAS * r.iabar + (safe ? div_by(aT3, r.rho, r.irho) : aT3 / r.rho);
  }
}
// E at table temperature node j (1-based).  There the position in the cell is exactly 0 (or 1 in the
// cell below), the T bases are exactly 1 and 0, and of the 36 terms of f and df/dT only the node's
// own 6 are left, in the reference's order: 12 coefficients instead of 36 and no T basis.
__device__ __forceinline__ double helm_energy_at_node(const HelmTable &h, const HelmRho &r, const double r0[3],
                                                      const double r1[3], int j) {
  const double *lo = h.tab + 9 * ((long long)(r.ih - 1) + (long long)h.nrho * (j - 1)), *hi = lo + 9;
  const double T = __ldg(h.T + j - 1);
  double f = __ldg(lo) * r0[0];
  f = f + __ldg(hi) * r1[0];
  f = f + __ldg(lo + 3) * r0[1];
  f = f + __ldg(hi + 3) * r1[1];
  f = f + __ldg(lo + 4) * r0[2];
  f = f + __ldg(hi + 4) * r1[2];
  double df_dT = __ldg(lo + 1) * r0[0];
  df_dT = df_dT + __ldg(hi + 1) * r1[0];
  df_dT = df_dT + __ldg(lo + 5) * r0[1];
  df_dT = df_dT + __ldg(hi + 5) * r1[1];
  df_dT = df_dT + __ldg(lo + 6) * r0[2];
  df_dT = df_dT + __ldg(hi + 6) * r1[2];
  double s = -r.Ye * df_dT;
  double e = r.Ye * f + T * s;
  double T2 = T * T, T3 = T2 * T, T4 = T3 * T;
  const double aT4 = CONST_RAD * T4;
  return e + 1.5 * CONST_RGAS * T * r.iabar + (r.ok && helm_in_range(T) ? div_by(aT4, r.rho, r.irho) : aT4 / r.rho);
}
__device__ __forceinline__ double helm_given2_energy(const HelmTable &h, double rho, double T, double abar, double zbar) {
  const HelmRho r = helm_rho_part(h, rho, abar, zbar);
  double r0[3], r1[3], E, dE;
  helm_rho_bases(r, r0, r1);
  HelmTemp t;
  helm_energy<false>(h, r, r0, r1, t, T, E, dE);
  return E;
}

// helm_rhoT_given1 (source.F90:24234-24569): P and dP/dT; dr0, dr1 the derivative density bases
__device__ __forceinline__ void helm_rho_dbases(const HelmTable &h, const HelmRho &r, double dr0[3], double dr1[3]) {
  const double idrho = __ldg(h.inv_drho + r.ih - 1);
  hb1(r.x, idrho, r.drho, dr0);
  hb1m(r.omx, idrho, r.drho, dr1);
}
__device__ __forceinline__ void helm_pressure(const HelmTable &h, const HelmRho &r, const double dr0[3],
                                              const double dr1[3], HelmTemp &t, double T, double &P, double &dPdT) {
  helm_temp_part(h, T, t);
  double c[36];
  helm_load36(h, r.ih, t.jh, c);
  const double dT2 = t.dT * t.dT;
  double t0[3], t1[3];
  hb0(t.y, t.dT, dT2, t0);
  hb0m(t.omy, t.dT, dT2, t1);
  double df_drho = helm_sum36(c, dr0, dr1, t0, t1);
  double d0[3], d1[3];
  hb1(t.y, t.idT, t.dT, d0);
  hb1m(t.omy, t.idT, t.dT, d1);
  double df_drhodT = helm_sum36(c, dr0, dr1, d0, d1);
  double tmp = r.rhos * r.rhos;
  double pp = tmp * df_drho;
  double dp = tmp * df_drhodT;
  double T2 = T * T, T3 = T2 * T, T4 = T3 * T;
  double pion = CONST_RGAS * r.rho * T * r.iabar;
  double dpiondt = CONST_RGAS * r.rho * r.iabar;
  P = pp + pion + CONST_RAD * T4 * (1.0 / 3.0);
  dPdT = dp + dpiondt + (4.0 / 3.0) * CONST_RAD * T3;
}

// helm_rhoT_given_full (source.F90:23686-24232): P, E, relativistic sound speed, cv
__device__ __forceinline__ void helm_full(const HelmTable &h, const HelmRho &r, HelmTemp &t, double T, double &P,
                                          double &E, double &sound, double &cv) {
  helm_temp_part(h, T, t);
  double c[36];
  helm_load36(h, r.ih, t.jh, c);
  const double dT2 = t.dT * t.dT, idT2 = t.idT * t.idT;
  double r0[3], r1[3], t0[3], t1[3], dr0[3], dr1[3], dt0[3], dt1[3], et0[3], et1[3];
  helm_rho_bases(r, r0, r1);
  hb0(t.y, t.dT, dT2, t0);
  hb0m(t.omy, t.dT, dT2, t1);
  double f = helm_sum36(c, r0, r1, t0, t1);
  helm_rho_dbases(h, r, dr0, dr1);
  double df_drho = helm_sum36(c, dr0, dr1, t0, t1);
  hb1(t.y, t.idT, t.dT, dt0);
  hb1m(t.omy, t.idT, t.dT, dt1);
  double df_dT = helm_sum36(c, r0, r1, dt0, dt1);
  double df_drhodT = helm_sum36(c, dr0, dr1, dt0, dt1);
  hb2(t.y, idT2, t.idT, et0);
  hb2m(t.omy, idT2, t.idT, et1);
  double df_dT2 = helm_sum36(c, r0, r1, et0, et1);
  // bicubic Hermite of dP/d(rho Ye) (source.F90:24082-24118)
  double x = r.x, x2 = x * x, x3 = x2 * x, omx = r.omx, omx2 = omx * omx, omx3 = omx2 * omx;
  double y = t.y, y2 = y * y, y3 = y2 * y, omy = t.omy, omy2 = omy * omy, omy3 = omy2 * omy;
  double p0r = 2.0 * x3 - 3.0 * x2 + 1.0;
  double p1r = (x3 - 2.0 * x2 + x) * r.drho;
  double p0mr = 2.0 * omx3 - 3.0 * omx2 + 1.0;
  double p1mr = -(omx3 - 2.0 * omx2 + omx) * r.drho;
  double p0t = 2.0 * y3 - 3.0 * y2 + 1.0;
  double p1t = (y3 - 2.0 * y2 + y) * t.dT;
  double p0mt = 2.0 * omy3 - 3.0 * omy2 + 1.0;
  double p1mt = -(omy3 - 2.0 * omy2 + omy) * t.dT;
  const double *q00 = h.dpdr + 4 * ((long long)(r.ih - 1) + (long long)h.nrho * (t.jh - 1));
  const double *q10 = q00 + 4, *q01 = q00 + 4 * (long long)h.nrho, *q11 = q01 + 4;
  double l[16];
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    l[4 * v + 0] = __ldg(q00 + v);
    l[4 * v + 1] = __ldg(q10 + v);
    l[4 * v + 2] = __ldg(q01 + v);
    l[4 * v + 3] = __ldg(q11 + v);
  }
  double dP_drho = l[0] * p0r * p0t + l[1] * p0mr * p0t + l[2] * p0r * p0mt + l[3] * p0mr * p0mt +
                   l[4] * p0r * p1t + l[5] * p0mr * p1t + l[6] * p0r * p1mt + l[7] * p0mr * p1mt +
                   l[8] * p1r * p0t + l[9] * p1mr * p0t + l[10] * p1r * p0mt + l[11] * p1mr * p0mt +
                   l[12] * p1r * p1t + l[13] * p1mr * p1t + l[14] * p1r * p1mt + l[15] * p1mr * p1mt;
  dP_drho = r.Ye * dP_drho;
  const double rho = r.rho, tmp2 = r.iabar;
  double tmp = r.rhos * r.rhos;
  double pp = tmp * df_drho;
  double dP_dT = tmp * df_drhodT;
  double s = -r.Ye * df_dT;
  double ds_dT = -r.Ye * df_dT2;
  double e = r.Ye * f + T * s;
  double dE_dT = T * ds_dT;
  double T2 = T * T, T3 = T2 * T, T4 = T3 * T;
  double pion = CONST_RGAS * rho * T * tmp2;
  double dpiondt = CONST_RGAS * rho * tmp2;
  double dpiondd = CONST_RGAS * T * tmp2;
  pp = pp + pion + CONST_RAD * T4 * (1.0 / 3.0);
  dP_dT = dP_dT + dpiondt + (4.0 / 3.0) * CONST_RAD * T3;
  dP_drho = dP_drho + dpiondd;
  const bool safe = r.ok && helm_in_range(T);
  const double aT4 = CONST_RAD * T4, aT3 = 4.0 * CONST_RAD * T3;
  e = e + 1.5 * CONST_RGAS * T * tmp2 + (safe ? div_by(aT4, rho, r.irho) : aT4 / rho);
  dE_dT = dE_dT + 1.5 * CONST_RGAS * tmp2 + (safe ? div_by(aT3, rho, r.irho) : aT3 / rho);
  double zz = pp / rho;
  double c_v = dE_dT;
  double chiT = T / pp * dP_dT;
  double chirho = dP_drho / zz;
  double xx = zz * chiT / (T * c_v);
  double gam1 = chiT * xx + chirho;
  double z = 1.0 + (e + CONST_C2) / zz;
  P = pp;
  E = e;
  cv = c_v;
  sound = CONST_C * sqrt(gam1 / z);
}
__device__ __forceinline__ void helm_given_full(const HelmTable &h, double rho, double T, double abar,
                                                double zbar, double &P, double &E, double &sound,
                                                double &cv) {
  HelmTemp t;
  helm_full(h, helm_rho_part(h, rho, abar, zbar), t, T, P, E, sound, cv);
}

// helm_rhoe_given Newton (source.F90:24982-25019).  Returns the iterations used; `clamped`
// counts resets to the starting guess after leaving [Tl_eos, Th_eos].
__device__ __forceinline__ int helm_rhoe_newton(const HelmTable &h, const HelmRho &r, HelmTemp &t, double E0, double &T,
                                                int max_iter, int &clamped, bool *converged = nullptr) {
  double Told = T;
  int used = 0;
  bool conv = false;
  double r0[3], r1[3];
  helm_rho_bases(r, r0, r1);
  for (int iter = 1; iter <= max_iter; ++iter) {
    used = iter;
    double E, dE;
    helm_energy<true>(h, r, r0, r1, t, T, E, dE);
    double res = E - E0;
    T = T - res / dE;
    double error = fabs(res / E0);
    if ((T < h.Tl) || (T > h.Th)) {
      T = Told;
      error = EM15;
      ++clamped;
    }
    if (error < HELM_TOL) { conv = true; break; }
  }
  if (converged) *converged = conv;
  return used;
}

// helm_rhoP_given Newton (source.F90:24943-24980)
__device__ __forceinline__ int helm_rhoP_newton(const HelmTable &h, const HelmRho &r, HelmTemp &t, double P0, double &T,
                                                int &clamped) {
  double Told = T;
  int used = 0;
  double dr0[3], dr1[3];
  helm_rho_dbases(h, r, dr0, dr1);
  for (int iter = 1; iter <= 100; ++iter) {
    used = iter;
    double P, dP;
    helm_pressure(h, r, dr0, dr1, t, T, P, dP);
    double res = P - P0;
    T = T - res / dP;
    double error = fabs(res / P0);
    if ((T < h.Tl) || (T > h.Th)) {
      T = Told;
      error = EM15;
      ++clamped;
    }
    if (error < HELM_TOL) break;
  }
  return used;
}

// helm_rhoP_given with return_sound (source.F90:24943-24980) for one Riemann side: returns
// rho * e and the sound speed
__device__ __forceinline__ void helm_side_eos_inl(const HelmTable &h, double rho, double p, double abar,
                                                  double zbar, double T, double &rhoe, double &sound) {
  int clamped = 0;
  const HelmRho r = helm_rho_part(h, rho, abar, zbar);
  HelmTemp t;
  helm_rhoP_newton(h, r, t, p, T, clamped);
  double Pd, E, cv;
  helm_full(h, r, t, T, Pd, E, sound, cv);
  rhoe = E * rho;
}

}  // namespace phl
