// phl_split.cu -- FP32 split-precision form of the explicit FV step (hydro and MHD
// configurations).
//
// Storage per cell: conserved state U (FP64, carried across stages and steps), primitive
// deviations W' = (rho - rho_eq, v, p - p_eq, scalars) and (gammae - gammae_eq, gammac) in FP32,
// temperature and internal energy in FP64; MHD adds the face B (FP64), the scaled cell B and
// cell EMFs (FP32).  Reconstruction (LIM2ND, PPH, LIM5TH), the Riemann solvers, face and corner
// EMFs and the flux divergence run in FP32 on the well-balanced deviations: the pressure enters
// every flux as a deviation, so pR - pL, p* - p_eq,face and the momentum flux after the WB fix
// (source/source.F90:8953-8959) are formed without cancelling large numbers, and Mach 1e-3
// perturbations keep their FP32 precision.  The RK combine, the face-B update, cons->prim, the
// Helmholtz Newton inversion and the CFL maximum stay in FP64.  All FP32 quantities are in scaled
// units (rho / rho_ref, p / p_ref, v / v_ref with v_ref^2 = p_ref / rho_ref, phi / v_ref^2,
// B / sqrt(p_ref)), fixed per run, so products of deviations never leave FP32 range whatever the
// problem's cgs magnitudes.
//
// Stage: k_face_split_row along x1 and k_face_split_walk along x2 and x3 (PLM), or k_face_split per
// direction (PPH, LIM5TH); for MHD k_corner_split and k_bface_split; then k_c2p_split.  With the
// learned temperature guess k_c2p_split_features, k_mlp_guess, k_c2p_split_guessed.  Hydro on small
// grids: k_stage_split, one kernel.
#include <cuda_runtime.h>
#include <cstdlib>
#include <algorithm>
#include <cstring>
#include "phl_eos_fast.cuh"
#include "phl_mlp.cuh"
#include "phl_umma.cuh"
// kernel namespace of this unit (FP32 flux arithmetic with contraction); see phl_kernels.cuh
#define PHL_KERNEL_UNIT split_unit
#include "phl_runner.h"

namespace phl {

// LIM2ND slope df db / (df + db) in FP32 for differences of the same sign, else 0, without forming
// df db (which can overflow or underflow) and without a branch: |db| / (|df| + |db|) lies in (0, 1).
// The test of the sum keeps 0 / 0 out, and a NaN difference: it gives slope 0, as the reference's
// df db > 0 does, so that a cell beside a NaN keeps finite edges.
__device__ __forceinline__ float plm_slope_f32(float sf, float sb) {
  const float sum = fabsf(sf) + fabsf(sb);
  const float s = sf * (fabsf(sb) * (1.0f / sum));
  return (__float_as_int(sf) ^ __float_as_int(sb)) >= 0 && sum > 0.0f ? s : 0.0f;
}
__device__ __forceinline__ void plm_f32(float qm, float qc, float qp, float &lo, float &hi) {
  const float slope = plm_slope_f32(qp - qc, qc - qm);
  lo = fmaf(-0.5f, slope, qc);
  hi = fmaf(0.5f, slope, qc);
}

// --------------------------------------------------------------------- packed FP32 pairs
// Two FP32 lanes in one 64-bit register pair: add, sub, mul and fma take one issue slot for both
// (the sm_100 f32x2 instructions).  The MHD solver holds the left state in .x and the right one in
// .y; its arithmetic is the same on both sides, and the face kernels are bound by issue slots (66% of
// the cycles issued while the FMA pipe was 29% busy).  With the branch-free limiter, a x2 or x3 face
// took 550 instructions instead of 945 and the faces of a direction at 128^3 57 us instead of 92.
#define PHL_F2OP(name, op)                                                                              \
  __device__ __forceinline__ float2 name(float2 a, float2 b) {                                          \
    float2 r;                                                                                           \
    asm("{.reg .b64 a, b, r; mov.b64 a, {%2, %3}; mov.b64 b, {%4, %5}; " op ".rn.ftz.f32x2 r, a, b; "   \
        "mov.b64 {%0, %1}, r;}"                                                                         \
        : "=f"(r.x), "=f"(r.y)                                                                          \
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));                                                      \
    return r;                                                                                           \
  }
PHL_F2OP(f2add, "add")
PHL_F2OP(f2sub, "sub")
PHL_F2OP(f2mul, "mul")
#undef PHL_F2OP
__device__ __forceinline__ float2 f2fma(float2 a, float2 b, float2 c) {
  float2 r;
  asm("{.reg .b64 a, b, c, r; mov.b64 a, {%2, %3}; mov.b64 b, {%4, %5}; mov.b64 c, {%6, %7}; "
      "fma.rn.ftz.f32x2 r, a, b, c; mov.b64 {%0, %1}, r;}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return r;
}
__device__ __forceinline__ float2 f2dup(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 f2rcp(float2 a) { return make_float2(1.0f / a.x, 1.0f / a.y); }
__device__ __forceinline__ float2 f2sqrt0(float2 a) {
  return make_float2(sqrtf(fmaxf(a.x, 0.0f)), sqrtf(fmaxf(a.y, 0.0f)));
}

// --------------------------------------------------------------------- FP32 Riemann (hydro)
// qL/qR: [rho (full), v1, v2, (v3), p' (deviation), scalars...] in the normal frame, pe the face
// equilibrium pressure.  Returns the flux with the momentum flux already reduced by pe (the
// reference's WB fix).  Same solver as riemann_hydro (source.F90:15681-16252).
template <int DIM, int NV, int EOSM, int RIEM>
__device__ __forceinline__ void riemann_hydro_split(const float *qL, const float *qR, const float *gL,
                                                    const float *gR, float pe, float gm, float mach_cutoff,
                                                    float *flux, bool flat = false, bool all_mach = false) {
  constexpr int IP = 1 + DIM, IAS = 2 + DIM;
  constexpr bool D3 = DIM == 3;
  // pairs: .x left, .y right
  const float2 rho2 = make_float2(qL[0], qR[0]), u2 = make_float2(qL[1], qR[1]), v2v = make_float2(qL[2], qR[2]);
  const float2 w2 = D3 ? make_float2(qL[3], qR[3]) : f2dup(0.0f);
  const float2 pd2 = make_float2(qL[IP], qR[IP]), p2 = f2add(f2dup(pe), pd2);
  const float2 irho = f2rcp(rho2), pr2 = f2mul(p2, irho);
  float2 vsq = f2fma(v2v, v2v, f2mul(u2, u2));
  if (D3) vsq = f2fma(w2, w2, vsq);
  float2 eint, csq, cs;
  if (EOSM == EOS_FAST) {
    eint = f2mul(p2, f2rcp(make_float2(gL[0] - 1.0f, gR[0] - 1.0f)));
    csq = f2mul(make_float2(gL[1], gR[1]), pr2);
    cs = make_float2(sqrtf(csq.x), sqrtf(csq.y));
  } else if (EOSM == EOS_GIVEN) {
    eint = make_float2(gL[0], gR[0]);
    cs = make_float2(gL[1], gR[1]);
    csq = f2mul(cs, cs);
  } else {
    eint = f2mul(p2, f2dup(1.0f / (gm - 1.0f)));
    csq = f2mul(f2dup(gm), pr2);
    cs = make_float2(sqrtf(csq.x), sqrtf(csq.y));
  }
  const float2 rhoe2 = f2fma(f2mul(f2dup(0.5f), rho2), vsq, eint);
  const float max_c = fmaxf(cs.x, cs.y);
  float sL = fminf(u2.x, u2.y) - max_c;
  float sR = fmaxf(u2.x, u2.y) + max_c;
  const float2 s2 = make_float2(sL, sR), dsu2 = f2sub(s2, u2), rd2 = f2mul(rho2, dsu2), rdu2 = f2mul(rd2, u2);
  const float ustar = ((pd2.y - pd2.x) + rdu2.x - rdu2.y) / (rd2.x - rd2.y);
  const float2 us2 = f2dup(ustar), du2 = f2sub(us2, u2);
  const float2 rs2 = f2mul(rd2, f2rcp(f2sub(s2, us2)));  // rho*
  const float2 rhoes2 = f2mul(rs2, f2fma(du2, f2fma(pr2, f2rcp(dsu2), us2), f2mul(rhoe2, irho)));
  if (flat) {
    // HLL on a flattened face (USE_SHOCK_FLATTENING, source.F90:15929-16010); the momentum
    // flux takes the pressure deviations, sR pe - sL pe over sR - sL being exactly pe
    sL = fminf(0.0f, sL);
    sR = fmaxf(0.0f, sR);
    const float rhoL = rho2.x, rhoR = rho2.y, vx1L = u2.x, vx1R = u2.y, vx2L = v2v.x, vx2R = v2v.y, vx3L = w2.x;
    const float vx3R = w2.y, rhoeL = rhoe2.x, rhoeR = rhoe2.y, pLd = pd2.x, pRd = pd2.y, pL = p2.x, pR = p2.y;
    float UL[NV], UR[NV], fL[NV], fR[NV];
    UL[0] = rhoL; UL[1] = rhoL * vx1L; UL[2] = rhoL * vx2L; if (DIM == 3) UL[3] = rhoL * vx3L; UL[IP] = rhoeL;
    UR[0] = rhoR; UR[1] = rhoR * vx1R; UR[2] = rhoR * vx2R; if (DIM == 3) UR[3] = rhoR * vx3R; UR[IP] = rhoeR;
    fL[0] = rhoL * vx1L; fL[1] = rhoL * vx1L * vx1L + pLd; fL[2] = rhoL * vx1L * vx2L;
    if (DIM == 3) fL[3] = rhoL * vx1L * vx3L;
    fL[IP] = (rhoeL + pL) * vx1L;
    fR[0] = rhoR * vx1R; fR[1] = rhoR * vx1R * vx1R + pRd; fR[2] = rhoR * vx1R * vx2R;
    if (DIM == 3) fR[3] = rhoR * vx1R * vx3R;
    fR[IP] = (rhoeR + pR) * vx1R;
#pragma unroll
    for (int iv = IAS; iv < NV; ++iv) {
      UL[iv] = rhoL * qL[iv];
      UR[iv] = rhoR * qR[iv];
      fL[iv] = UL[iv] * vx1L;
      fR[iv] = UR[iv] * vx1R;
    }
    const float dh = 1.0f / (sR - sL), ph = sL * sR;
#pragma unroll
    for (int iv = 0; iv < NV; ++iv) flux[iv] = dh * (sR * fL[iv] - sL * fR[iv] + ph * (UR[iv] - UL[iv]));
    return;
  }
  if (RIEM == R_LHLLC) {
    // the Mach numbers compared as squares: one square root, for the larger
    const float2 m2 = f2mul(vsq, f2rcp(csq));
    const float chi = fmaxf(mach_cutoff, fminf(1.0f, sqrtf(fmaxf(m2.x, m2.y))));
    const float phi = chi * (2.0f - chi);
    const float pstar_d = 0.5f * (pd2.x + pd2.y) -
                          0.125f * phi * (rho2.x + rho2.y) * (cs.x + cs.y) * (u2.y - u2.x);
    if (all_mach && (sL > 0.0f || sR < 0.0f)) {
      // FLUX_IS_ALL_MACH: the upwind state outside the wave fan, pe removed from the momentum flux
      const bool left = sL > 0.0f;
      const float m = left ? rho2.x * u2.x : rho2.y * u2.y, vx1 = left ? u2.x : u2.y;
      flux[0] = m;
      flux[1] = m * vx1 + (left ? pd2.x : pd2.y);
      flux[2] = m * (left ? v2v.x : v2v.y);
      if (D3) flux[3] = m * (left ? w2.x : w2.y);
      flux[IP] = (left ? rhoe2.x + p2.x : rhoe2.y + p2.y) * vx1;
#pragma unroll
      for (int iv = IAS; iv < NV; ++iv) flux[iv] = m * (left ? qL[iv] : qR[iv]);
      return;
    }
    const bool left = !signbit(ustar);
    const float m = (left ? rs2.x : rs2.y) * ustar;
    flux[0] = m;
    flux[1] = m * ustar + pstar_d;
    flux[2] = m * (left ? v2v.x : v2v.y);
    if (D3) flux[3] = m * (left ? w2.x : w2.y);
    flux[IP] = ((left ? rhoes2.x : rhoes2.y) + (pe + pstar_d)) * ustar;
#pragma unroll
    for (int iv = IAS; iv < NV; ++iv) flux[iv] = m * (left ? qL[iv] : qR[iv]);
  } else {
    const bool left = ustar > 0.0f;
    const float *q = left ? qL : qR;
    const float rho = left ? rho2.x : rho2.y, vx1 = left ? u2.x : u2.y, vx2 = left ? v2v.x : v2v.y;
    const float vx3 = left ? w2.x : w2.y, p = left ? p2.x : p2.y, pd = left ? pd2.x : pd2.y;
    const float rhoe = left ? rhoe2.x : rhoe2.y, rhostar = left ? rs2.x : rs2.y;
    const float rhoestar = left ? rhoes2.x : rhoes2.y, s = left ? sL : sR;
    const bool sup = left ? (sL >= 0.0f) : (sR < 0.0f);
    float U[NV], f[NV];
    U[0] = rho; U[1] = rho * vx1; U[2] = rho * vx2; if (DIM == 3) U[3] = rho * vx3; U[IP] = rhoe;
    f[0] = rho * vx1; f[1] = rho * vx1 * vx1 + pd; f[2] = rho * vx1 * vx2;
    if (DIM == 3) f[3] = rho * vx1 * vx3;
    f[IP] = (rhoe + p) * vx1;
#pragma unroll
    for (int iv = IAS; iv < NV; ++iv) { U[iv] = rho * q[iv]; f[iv] = rho * vx1 * q[iv]; }
    if (sup) {
#pragma unroll
      for (int iv = 0; iv < NV; ++iv) flux[iv] = f[iv];
    } else {
      float Us[NV];
      Us[0] = rhostar; Us[1] = rhostar * ustar; Us[2] = rhostar * vx2; if (DIM == 3) Us[3] = rhostar * vx3;
      Us[IP] = rhoestar;
#pragma unroll
      for (int iv = IAS; iv < NV; ++iv) Us[iv] = rhostar * q[iv];
#pragma unroll
      for (int iv = 0; iv < NV; ++iv) flux[iv] = f[iv] + s * (Us[iv] - U[iv]);
    }
  }
}

// --------------------------------------------------------------------- FP32 Riemann (MHD)
// HLLD / LHLLD (source.F90:13969-15024) on the split variables: qL/qR as for
// riemann_hydro_split, bL/bR the face B in the normal frame (units sqrt(p_ref)), pe the face
// equilibrium pressure.  Every difference of total pressures is formed from the deviations
// (pT' = p' + B^2/2), the star pressure as pe + pT*' with the weights of the reference, and the
// normal momentum flux is returned with pe removed (the reference's WB fix).  fluxb is the
// induction flux (0, v1 B2 - B1 v2, v1 B3 - B1 v3).
template <int DIM, int NV, int EOSM, int RIEM>
__device__ __forceinline__ void riemann_mhd_split(const float *qL, const float *qR, const float *bL,
                                                  const float *bR, const float *gL, const float *gR, float pe,
                                                  float gm, float mach_cutoff, float *flux, float *fluxb,
                                                  bool flat = false, bool all_mach = false) {
  constexpr int IP = 1 + DIM, IAS = 2 + DIM;
  constexpr bool D3 = DIM == 3;
  // pairs: .x left, .y right
  const float2 rho2 = make_float2(qL[0], qR[0]), u2 = make_float2(qL[1], qR[1]), v2v = make_float2(qL[2], qR[2]);
  const float2 w2 = D3 ? make_float2(qL[3], qR[3]) : f2dup(0.0f);
  const float2 pd2 = make_float2(qL[IP], qR[IP]), p2 = f2add(f2dup(pe), pd2);
  const float2 irho = f2rcp(rho2);
  float2 vsq = f2fma(v2v, v2v, f2mul(u2, u2));
  if (D3) vsq = f2fma(w2, w2, vsq);
  float2 eint, c2;
  if (EOSM == EOS_FAST) {
    eint = f2mul(p2, f2rcp(make_float2(gL[0] - 1.0f, gR[0] - 1.0f)));
    c2 = f2mul(make_float2(gL[1], gR[1]), f2mul(p2, irho));
  } else if (EOSM == EOS_GIVEN) {
    eint = make_float2(gL[0], gR[0]);
    c2 = f2mul(make_float2(gL[1], gR[1]), make_float2(gL[1], gR[1]));
  } else {
    eint = f2mul(p2, f2dup(1.0f / (gm - 1.0f)));
    c2 = f2mul(f2dup(gm), f2mul(p2, irho));
  }
  // both sides of a face carry the same normal field
  const float bx1 = bL[0], bx1_2 = bx1 * bx1;
  const float2 by2 = make_float2(bL[1], bR[1]), bz2 = D3 ? make_float2(bL[2], bR[2]) : f2dup(0.0f);
  float2 bsq = f2fma(by2, by2, f2dup(bx1_2));
  if (D3) bsq = f2fma(bz2, bz2, bsq);
  const float2 pb2 = f2mul(f2dup(0.5f), bsq);
  const float2 rhoe2 = f2add(f2fma(f2mul(f2dup(0.5f), rho2), vsq, eint), pb2);
  const float2 ptd2 = f2add(pd2, pb2);  // total pressure deviations
  const float2 a2 = f2mul(bsq, irho), an2 = f2mul(f2dup(bx1_2), irho);
  const float2 c2a2 = f2add(c2, a2);
  const float2 cf2 = f2mul(f2dup(0.5f), f2add(c2a2, f2sqrt0(f2fma(f2dup(-4.0f), f2mul(c2, an2), f2mul(c2a2, c2a2)))));
  const float max_c = sqrtf(fmaxf(cf2.x, cf2.y));
  float sL = fminf(u2.x, u2.y) - max_c;
  float sR = fmaxf(u2.x, u2.y) + max_c;
  const float2 s2 = make_float2(sL, sR);
  const float2 dsu2 = f2sub(s2, u2), rd2 = f2mul(rho2, dsu2);
  const float inv_temp1 = 1.0f / (rd2.y - rd2.x);
  const float2 rdu2 = f2mul(rd2, u2);
  const float ustar = ((rdu2.y - rdu2.x) - (ptd2.y - ptd2.x)) * inv_temp1;
  float phi = 1.0f;
  if (RIEM == R_LHLLD) {
    const float2 va2 = f2add(vsq, a2);
    const float2 cu2 = f2add(va2, f2sqrt0(f2fma(f2dup(-4.0f), f2mul(vsq, an2), f2mul(va2, va2))));
    // the fast Mach numbers compared as squares (cu^2 / cf^2): one square root, for the larger
    const float2 m2 = f2mul(f2mul(f2dup(0.5f), cu2), f2rcp(cf2));
    const float mm2 = fmaxf(m2.x, m2.y);
    const float chi = fmaxf(mach_cutoff, fminf(1.0f, sqrtf(mm2)));
    if (mm2 < 0.36f) phi = chi * (2.0f - chi);
  }
  if (flat) {
    // HLL on a flattened face (source.F90:14386-14495), total-pressure deviations in the
    // momentum flux as in the HLL of riemann_hydro_split
    sL = fminf(0.0f, sL);
    sR = fmaxf(0.0f, sR);
    const float rhoL = rho2.x, rhoR = rho2.y, vx1L = u2.x, vx1R = u2.y, vx2L = v2v.x, vx2R = v2v.y, vx3L = w2.x;
    const float vx3R = w2.y, bx2L = by2.x, bx2R = by2.y, bx3L = bz2.x, bx3R = bz2.y, rhoeL = rhoe2.x;
    const float rhoeR = rhoe2.y, ptLd = ptd2.x, ptRd = ptd2.y, ptL = pe + ptLd, ptR = pe + ptRd;
    float UL[NV], UR[NV], fL[NV], fR[NV];
    UL[0] = rhoL; UL[1] = rhoL * vx1L; UL[2] = rhoL * vx2L; if (DIM == 3) UL[3] = rhoL * vx3L; UL[IP] = rhoeL;
    UR[0] = rhoR; UR[1] = rhoR * vx1R; UR[2] = rhoR * vx2R; if (DIM == 3) UR[3] = rhoR * vx3R; UR[IP] = rhoeR;
    fL[0] = rhoL * vx1L; fL[1] = rhoL * vx1L * vx1L + ptLd - bx1_2; fL[2] = rhoL * vx1L * vx2L - bx1 * bx2L;
    if (DIM == 3) fL[3] = rhoL * vx1L * vx3L - bx1 * bx3L;
    fL[IP] = (rhoeL + ptL) * vx1L - bx1 * (bx1 * vx1L + bx2L * vx2L + bx3L * vx3L);
    fR[0] = rhoR * vx1R; fR[1] = rhoR * vx1R * vx1R + ptRd - bx1_2; fR[2] = rhoR * vx1R * vx2R - bx1 * bx2R;
    if (DIM == 3) fR[3] = rhoR * vx1R * vx3R - bx1 * bx3R;
    fR[IP] = (rhoeR + ptR) * vx1R - bx1 * (bx1 * vx1R + bx2R * vx2R + bx3R * vx3R);
#pragma unroll
    for (int iv = IAS; iv < NV; ++iv) {
      UL[iv] = rhoL * qL[iv];
      UR[iv] = rhoR * qR[iv];
      fL[iv] = UL[iv] * vx1L;
      fR[iv] = UR[iv] * vx1R;
    }
    const float UbL[3] = {bx1, bx2L, bx3L}, UbR[3] = {bx1, bx2R, bx3R};
    const float fbL[3] = {0.0f, vx1L * bx2L - vx2L * bx1, vx1L * bx3L - vx3L * bx1};
    const float fbR[3] = {0.0f, vx1R * bx2R - vx2R * bx1, vx1R * bx3R - vx3R * bx1};
    const float dh = 1.0f / (sR - sL), ph = sL * sR;
#pragma unroll
    for (int iv = 0; iv < NV; ++iv) flux[iv] = dh * (sR * fL[iv] - sL * fR[iv] + ph * (UR[iv] - UL[iv]));
#pragma unroll
    for (int iv = 0; iv < DIM; ++iv) fluxb[iv] = dh * (sR * fbL[iv] - sL * fbR[iv] + ph * (UbR[iv] - UbL[iv]));
    return;
  }
  // star total pressure: the weights sum to one, so pe factors out
  const float pstar_d = (rd2.y * ptd2.x - rd2.x * ptd2.y - phi * rd2.x * rd2.y * (u2.x - u2.y)) * inv_temp1;
  const float2 us2 = f2dup(ustar), dsum2 = f2sub(s2, us2), idsum2 = f2rcp(dsum2);
  const float2 rs2 = f2mul(rd2, idsum2);  // rho*
  const float2 ainv2 = f2rcp(f2fma(rd2, dsum2, f2dup(-bx1_2)));
  const float2 du2 = f2sub(us2, u2);
  const float2 nk2 = f2mul(f2mul(f2dup(-bx1), du2), ainv2);
  const float2 bk2 = f2mul(f2fma(rd2, dsu2, f2dup(-bx1_2)), ainv2);
  const float2 vs2 = f2fma(by2, nk2, v2v), bs2 = f2mul(by2, bk2);
  const float2 ws2 = D3 ? f2fma(bz2, nk2, w2) : f2dup(0.0f), bt2 = D3 ? f2mul(bz2, bk2) : f2dup(0.0f);
  float2 vdotb2 = f2fma(v2v, by2, f2mul(u2, f2dup(bx1))), vdotbs2 = f2fma(vs2, bs2, f2dup(ustar * bx1));
  if (D3) {
    vdotb2 = f2fma(w2, bz2, vdotb2);
    vdotbs2 = f2fma(ws2, bt2, vdotbs2);
  }
  // -pT u + pT* u* with pe factored: pe (u* - u) + (pT*' u* - pT' u)
  const float2 work2 = f2sub(f2dup(pstar_d * ustar), f2mul(ptd2, u2));
  const float2 rhoes2 = f2mul(f2fma(f2dup(bx1), f2sub(vdotb2, vdotbs2),
                                    f2add(f2fma(f2dup(pe), du2, f2mul(dsu2, rhoe2)), work2)), idsum2);
  // sqrt(rho*) and 1 / sqrt(rho*) from one reciprocal square root per side
  const float2 rsq2 = make_float2(rsqrtf(rs2.x), rsqrtf(rs2.y)), sq2 = f2mul(rs2, rsq2);
  const float abs_bx1 = fabsf(bx1);
  const float sstarL = ustar - abs_bx1 * rsq2.x;
  const float sstarR = ustar + abs_bx1 * rsq2.y;
  const float inv_sqr_bar = 1.0f / (sq2.x + sq2.y);
  const float sgn = copysignf(1.0f, bx1), sqsg = sq2.x * sq2.y * sgn;
  const float vx22star = (sq2.x * vs2.x + sq2.y * vs2.y + (bs2.y - bs2.x) * sgn) * inv_sqr_bar;
  const float bx22star = (sq2.x * bs2.y + sq2.y * bs2.x + sqsg * (vs2.y - vs2.x)) * inv_sqr_bar;
  float vx32star = 0.0f, bx32star = 0.0f;
  if (D3) {
    vx32star = (sq2.x * ws2.x + sq2.y * ws2.y + (bt2.y - bt2.x) * sgn) * inv_sqr_bar;
    bx32star = (sq2.x * bt2.y + sq2.y * bt2.x + sqsg * (ws2.y - ws2.x)) * inv_sqr_bar;
  }
  const float vdotb2star = ustar * bx1 + vx22star * bx22star + vx32star * bx32star;
  // rho e** = rho e* -/+ sqrt(rho*) (v*.B* - v**.B**) sgn
  const float2 rhoe2s2 = f2fma(f2mul(sq2, f2sub(vdotbs2, f2dup(vdotb2star))), make_float2(-sgn, sgn), rhoes2);

  fluxb[0] = 0.0f;
  // sstarL <= ustar <= sstarR: the side follows from ustar, and single says that the face lies
  // between that side's outer and Alfven waves
  const bool left = ustar > 0.0f;
  const float rhostar = left ? rs2.x : rs2.y, vx2s = left ? vs2.x : vs2.y, vx3s = left ? ws2.x : ws2.y;
  const float bx2s = left ? bs2.x : bs2.y, bx3s = left ? bt2.x : bt2.y;
  const float rhoes = left ? rhoes2.x : rhoes2.y, rhoe2s = left ? rhoe2s2.x : rhoe2s2.y;
  if (RIEM == R_LHLLD) {
    const bool single = left ? sstarL > 0.0f : !(sstarR > 0.0f);
    float rho = rhostar, vx1 = ustar, pres_d = pstar_d;
    float vx2 = single ? vx2s : vx22star, vx3 = single ? vx3s : vx32star;
    float bx2 = single ? bx2s : bx22star, bx3 = single ? bx3s : bx32star, rhoe = single ? rhoes : rhoe2s;
    if (all_mach && (sL > 0.0f || !(sR > 0.0f))) {
      // FLUX_IS_ALL_MACH: the outer states as well (source.F90:14576-14632)
      const bool ol = sL > 0.0f;
      rho = ol ? rho2.x : rho2.y; vx1 = ol ? u2.x : u2.y; vx2 = ol ? v2v.x : v2v.y; vx3 = ol ? w2.x : w2.y;
      rhoe = ol ? rhoe2.x : rhoe2.y; bx2 = ol ? by2.x : by2.y; bx3 = ol ? bz2.x : bz2.y;
      pres_d = ol ? ptd2.x : ptd2.y;
    }
    const float m = rho * vx1;
    flux[0] = m;
    flux[1] = m * vx1 + pres_d - bx1_2;
    flux[2] = m * vx2 - bx1 * bx2;
    if (D3) flux[3] = m * vx3 - bx1 * bx3;
    flux[IP] = (rhoe + (pe + pres_d)) * vx1 - bx1 * (bx1 * vx1 + vx2 * bx2 + vx3 * bx3);
    const bool up = !signbit(vx1);
#pragma unroll
    for (int iv = IAS; iv < NV; ++iv) flux[iv] = m * (up ? qL[iv] : qR[iv]);
    fluxb[1] = vx1 * bx2 - bx1 * vx2;
    if (D3) fluxb[2] = vx1 * bx3 - bx1 * vx3;
    return;
  }
  const float *q = left ? qL : qR;
  const float rho = left ? rho2.x : rho2.y, vx1 = left ? u2.x : u2.y, vx2 = left ? v2v.x : v2v.y;
  const float vx3 = left ? w2.x : w2.y, rhoe = left ? rhoe2.x : rhoe2.y, ptd = left ? ptd2.x : ptd2.y, pt = pe + ptd;
  const float bx2 = left ? by2.x : by2.y, bx3 = left ? bz2.x : bz2.y, vdotb = left ? vdotb2.x : vdotb2.y;
  float s = left ? sL : sR, sst = left ? sstarL : sstarR;
  const bool outer = left ? (sL > 0.0f) : (sR < 0.0f);
  const bool single = left ? (sstarL > 0.0f) : (sstarR < 0.0f);
  constexpr int NB = DIM == 3 ? 3 : 2;
  float U[NV], f[NV], Ub[3], fb[3];
  U[0] = rho; U[1] = rho * vx1; U[2] = rho * vx2; if (DIM == 3) U[3] = rho * vx3; U[IP] = rhoe;
  f[0] = rho * vx1; f[1] = rho * vx1 * vx1 + ptd - bx1_2; f[2] = rho * vx1 * vx2 - bx1 * bx2;
  if (DIM == 3) f[3] = rho * vx1 * vx3 - bx1 * bx3;
  f[IP] = (rhoe + pt) * vx1 - bx1 * vdotb;
#pragma unroll
  for (int iv = IAS; iv < NV; ++iv) { U[iv] = rho * q[iv]; f[iv] = rho * vx1 * q[iv]; }
  Ub[0] = bx1; Ub[1] = bx2; Ub[2] = bx3;
  fb[0] = 0.0f; fb[1] = vx1 * bx2 - bx1 * vx2; fb[2] = vx1 * bx3 - bx1 * vx3;
  if (outer) {
#pragma unroll
    for (int iv = 0; iv < NV; ++iv) flux[iv] = f[iv];
#pragma unroll
    for (int iv = 0; iv < NB; ++iv) fluxb[iv] = fb[iv];
    return;
  }
  float Us[NV], Ubs[3];
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
  float Uss[NV], Ubss[3];
  Uss[0] = rhostar; Uss[1] = rhostar * ustar; Uss[2] = rhostar * vx22star; if (DIM == 3) Uss[3] = rhostar * vx32star;
  Uss[IP] = rhoe2s;
#pragma unroll
  for (int iv = IAS; iv < NV; ++iv) Uss[iv] = rhostar * q[iv];
  Ubss[0] = bx1; Ubss[1] = bx22star; Ubss[2] = bx32star;
#pragma unroll
  for (int iv = 0; iv < NV; ++iv) {
    float d0 = Us[iv];
    flux[iv] = f[iv] + s * (d0 - U[iv]) + sst * (Uss[iv] - d0);
  }
#pragma unroll
  for (int iv = 0; iv < NB; ++iv) {
    float d0 = Ubs[iv];
    fluxb[iv] = fb[iv] + s * (d0 - Ub[iv]) + sst * (Ubss[iv] - d0);
  }
}

// --------------------------------------------------------------------- face flux storage
// The NV flux components of a face in P.fflux[d] lie in planes of vectors over the faces: one
// plane of float4 per four components, then a float2 and a float plane for the rest (7 components:
// 16 + 8 + 4 B).  A face is stored and read with 3 accesses instead of 7 and without padding.
template <int NV>
struct FluxPlanes {
  static constexpr int N4 = NV / 4, N2 = (NV % 4) / 2, N1 = NV % 2;
  static __device__ __forceinline__ void store(float *p, long long nf, long long f, const float *F) {
#pragma unroll
    for (int q = 0; q < N4; ++q)
      reinterpret_cast<float4 *>(p + 4ll * q * nf)[f] = make_float4(F[4 * q], F[4 * q + 1], F[4 * q + 2], F[4 * q + 3]);
    if (N2) reinterpret_cast<float2 *>(p + 4ll * N4 * nf)[f] = make_float2(F[4 * N4], F[4 * N4 + 1]);
    if (N1) p[(4ll * N4 + 2 * N2) * nf + f] = F[NV - 1];
  }
  static __device__ __forceinline__ void load(const float *p, long long nf, long long f, float *F) {
#pragma unroll
    for (int q = 0; q < N4; ++q) {
      const float4 v = __ldg(reinterpret_cast<const float4 *>(p + 4ll * q * nf) + f);
      F[4 * q] = v.x; F[4 * q + 1] = v.y; F[4 * q + 2] = v.z; F[4 * q + 3] = v.w;
    }
    if (N2) {
      const float2 v = __ldg(reinterpret_cast<const float2 *>(p + 4ll * N4 * nf) + f);
      F[4 * N4] = v.x; F[4 * N4 + 1] = v.y;
    }
    if (N1) F[NV - 1] = __ldg(p + (4ll * N4 + 2 * N2) * nf + f);
  }
};

// --------------------------------------------------------------------- FP32 loads
template <class C>
__device__ __forceinline__ void load_wf(const Prm &P, int i, int j, int k, float w[C::NV], float g2[2]) {
  const Geo &g = P.g;
  bool f0 = false, f1 = false, f2 = false;
  int si = map_index(i, g.nx[0], g.bc[0][0], g.bc[0][1], f0);
  int sj = map_index(j, g.nx[1], g.bc[1][0], g.bc[1][1], f1);
  int sk = C::DIM == 3 ? map_index(k, g.nx[2], g.bc[2][0], g.bc[2][1], f2) : 0;
  long long c = lin(g, si, sj, sk);
#pragma unroll
  for (int iv = 0; iv < C::NV; ++iv) w[iv] = __ldg(P.Wf_in + (long long)iv * g.N + c);
  if (f0) w[1] = -w[1];
  if (f1) w[2] = -w[2];
  if (C::DIM == 3 && f2) w[3] = -w[3];
  if (C::HELM) {
    g2[0] = __ldg(P.gf_in + c);
    g2[1] = __ldg(P.gf_in + g.N + c);
  }
}

// the same for an interior cell given by its linear index (no mapping, no mirror)
template <class C>
__device__ __forceinline__ void load_wf_at(const Prm &P, long long c, float w[C::NV], float g2[2]) {
  const long long N = P.g.N;
#pragma unroll
  for (int iv = 0; iv < C::NV; ++iv) w[iv] = __ldg(P.Wf_in + iv * N + c);
  if (C::HELM) {
    g2[0] = __ldg(P.gf_in + c);
    g2[1] = __ldg(P.gf_in + N + c);
  }
}

// linear-index step between neighbours along d
__device__ __forceinline__ long long dir_stride(const Geo &g, int d) {
  return d == 0 ? 1 : (d == 1 ? (long long)g.nx[0] : (long long)g.nx[0] * g.nx[1]);
}

// the per-side helm_rhoP_given of the split form, out of line: the split stage kernels call it
// twice per face, and an inlined Helmholtz evaluation at each site costs them their registers.
// It runs the contracted-coefficient evaluation of phl_eos_fast.cuh (the FP64 form keeps the
// reference's evaluation order, helm_side_eos_inl); results agree to rounding.
static __device__ __noinline__ void helm_side_eos(const HelmTable &h, double rho, double p, double abar,
                                                  double zbar, double T, double &rhoe, double &sound) {
  helm_side_eos_fast_inl(h, rho, p, abar, zbar, T, rhoe, sound);
}

// Helmholtz without USE_FASTEOS, split form: helm_rhoP_given (FP64) for one side of a face from
// the scaled FP32 face state and temperature guess; returns rho*e and the sound speed, scaled
template <class C>
__device__ __forceinline__ void split_side_eos(const Prm &P, const float *q, float pe, float tguess, float &rhoe_s,
                                               float &c_s) {
  const double rho = (double)q[0] * P.rho_ref, p = ((double)pe + (double)q[C::IP]) * P.p_ref;
  const double ye = q[C::IAS], abar = 1.0 / (double)q[C::IAS + 1], zbar = ye * abar;
  double rhoe, snd;
  helm_side_eos(P.helm, rho, p, abar, zbar, (double)tguess, rhoe, snd);
  rhoe_s = (float)(rhoe * P.inv_p_ref);
  c_s = (float)(snd * P.inv_v_ref);
}

// FP32 face values of one variable from the values of cells m-3 .. m+2 (v[0] .. v[5]; LIM2ND and
// PPH read v[1] .. v[4])
template <class C>
__device__ __forceinline__ void rec_face_f32(const float v[6], bool limited, float &qL, float &qR) {
  float lo, hi;
  if (C::REC == REC_LIM2ND) {
    plm_f32(v[1], v[2], v[3], lo, hi);
    qL = hi;
    plm_f32(v[2], v[3], v[4], lo, hi);
    qR = lo;
  } else {
    rec_edges<float, C::REC>(limited, v[0], v[1], v[2], v[3], v[4], lo, hi);
    qL = hi;
    rec_edges<float, C::REC>(limited, v[1], v[2], v[3], v[4], v[5], lo, hi);
    qR = lo;
  }
}

// USE_SHOCK_FLATTENING on the FP32 edge values: v holds cells m-3..m+2 of the face; a flagged
// cell m-1 (fa) or m (fb) gives its edge by LIM2ND PLM (source.F90:8743-8827, 9635-9700)
__device__ __forceinline__ void flatten_face_f32(const float v[6], bool fa, bool fb, float &qL, float &qR) {
  float lo, hi;
  if (fa) {
    plm_f32(v[1], v[2], v[3], lo, hi);
    qL = hi;
  }
  if (fb) {
    plm_f32(v[2], v[3], v[4], lo, hi);
    qR = lo;
  }
}
// the x1 sweep's gamma handling on flagged faces with WB (source.F90:8829-8872), reproduced as
// written: PLM gammas without the equilibrium gamma_e replace the flagged side, and the face's
// eq_gammae_x1 is added once more to the other side; cell m-1 before cell m
__device__ __forceinline__ void flatten_gamma_x1(const float gv[2][6], bool fa, bool fb, float ge, float gL[2],
                                                 float gR[2]) {
  float lo, hi;
  if (fa) {
#pragma unroll
    for (int iv = 0; iv < 2; ++iv) {
      plm_f32(gv[iv][1], gv[iv][2], gv[iv][3], lo, hi);
      gL[iv] = hi;
    }
    gR[0] = gR[0] + ge;
  }
  if (fb) {
#pragma unroll
    for (int iv = 0; iv < 2; ++iv) {
      plm_f32(gv[iv][2], gv[iv][3], gv[iv][4], lo, hi);
      gR[iv] = lo;
    }
    gL[0] = gL[0] + ge;
  }
}

// --------------------------------------------------------------------- split stage kernels
// Per-cell statistics of a stage, reduced once per block.
// per-thread counters (32-bit: a thread's cells times 100 iterations stay far below 2^32; the
// block sums go to the 64-bit counters of the context)
struct SplitStat {
  double smax = 0.0;
  unsigned calls = 0, iters = 0, nonconv = 0, clamp = 0, bad = 0;
  unsigned mlp_acc = 0, mlp_rej = 0, gevals = 0;  // learned guess in the step
};

template <class C>
__device__ __forceinline__ void split_stat_flush(const Prm &P, const SplitStat &st) {
  if (P.last_stage) block_max_atomic(st.smax, P.smax_bits);
  if (C::HELM && P.mlp_w) {
    const unsigned v[8] = {st.bad, st.calls, st.iters, st.nonconv, st.clamp, st.mlp_acc, st.mlp_rej, st.gevals};
    const int slot[8] = {STAT_NONFINITE, STAT_NEWTON_CALLS, STAT_NEWTON_ITERS, STAT_NEWTON_NONCONV, STAT_NEWTON_CLAMP,
                         STAT_MLP_ACC, STAT_MLP_REJ, STAT_GUESS_EVALS};
    block_counters(v, slot, P.stat);
  } else if (C::HELM) {
    const unsigned v[5] = {st.bad, st.calls, st.iters, st.nonconv, st.clamp};
    const int slot[5] = {STAT_NONFINITE, STAT_NEWTON_CALLS, STAT_NEWTON_ITERS, STAT_NEWTON_NONCONV, STAT_NEWTON_CLAMP};
    block_counters(v, slot, P.stat);
  } else {
    const unsigned v[1] = {st.bad};
    const int slot[1] = {STAT_NONFINITE};
    block_counters(v, slot, P.stat);
  }
}

// 8-byte asynchronous global -> shared copy (cp.async, completes at the next wait)
__device__ __forceinline__ void cp_async8(double *smem_dst, const double *gmem_src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// --------------------------------------------------------------------- shock detector (split)
// USE_SHOCK_FLATTENING on the split state (source.F90:8073-8136): the full pressure of a
// (possibly ghost) cell is its FP32 deviation in physical units plus the equilibrium stored
// for that ghost cell; marks go to P.sf_mark, and k_sf_flag forms is_flattened as in FP64
template <class C>
__device__ __forceinline__ double sf_pressure_split(const Prm &P, int i, int j, int k) {
  const Geo &g = P.g;
  bool f = false;
  int si = map_index(i, g.nx[0], g.bc[0][0], g.bc[0][1], f);
  int sj = map_index(j, g.nx[1], g.bc[1][0], g.bc[1][1], f);
  int sk = C::DIM == 3 ? map_index(k, g.nx[2], g.bc[2][0], g.bc[2][1], f) : 0;
  double p = (double)__ldg(P.Wf_in + (long long)C::IP * g.N + lin(g, si, sj, sk)) * P.p_ref;
  if (C::WB) {
    const int G = P.sf_G, G3 = C::DIM == 3 ? P.sf_G : 0;
    long long e = P.sf_eq_profile ? (long long)(j + G)
                                  : (long long)(i + G) + (long long)(g.nx[0] + 2 * G) *
                                        ((long long)(j + G) + (long long)(g.nx[1] + 2 * G) * (k + G3));
    p = p + __ldg(P.sf_eq_p + e);
  }
  return p;
}

template <class C>
__global__ void __launch_bounds__(256) k_sf_mark_split(Prm P) {
  if (!*P.active) return;
  const Geo &g = P.g;
  const long long n = sf_mark_cells<C>(g);
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const int m0 = g.nx[0] + 4, m1 = g.nx[1] + 4;
  int i, j, k;
  unflatten3(t, m0, m1, i, j, k);
  i -= 2;
  j -= 2;
  k = C::DIM == 3 ? k - 2 : 0;
  double tmp;
  if (C::DIM == 3)
    tmp = (fabs(sf_pressure_split<C>(P, i, j, k + 1) - sf_pressure_split<C>(P, i, j, k - 1)) +
           fabs(sf_pressure_split<C>(P, i, j + 1, k) - sf_pressure_split<C>(P, i, j - 1, k)) +
           fabs(sf_pressure_split<C>(P, i + 1, j, k) - sf_pressure_split<C>(P, i - 1, j, k))) /
          sf_pressure_split<C>(P, i, j, k);
  else
    tmp = (fabs(sf_pressure_split<C>(P, i, j + 1, k) - sf_pressure_split<C>(P, i, j - 1, k)) +
           fabs(sf_pressure_split<C>(P, i + 1, j, k) - sf_pressure_split<C>(P, i - 1, j, k))) /
          sf_pressure_split<C>(P, i, j, k);
  P.sf_mark[t] = tmp > P.eps_sf ? 1 : 0;
}

// --------------------------------------------------------------------- split MHD
// Cell-centred B of a (possibly ghost) cell in units of b_ref, component d negated for each
// mirrored dimension d.
template <class C>
__device__ __forceinline__ void load_bccf(const Prm &P, int i, int j, int k, float b[3]) {
  const Geo &g = P.g;
  b[0] = b[1] = b[2] = 0.0f;
  if (!C::MHD) return;
  bool f0 = false, f1 = false, f2 = false;
  int si = map_index(i, g.nx[0], g.bc[0][0], g.bc[0][1], f0);
  int sj = map_index(j, g.nx[1], g.bc[1][0], g.bc[1][1], f1);
  int sk = C::DIM == 3 ? map_index(k, g.nx[2], g.bc[2][0], g.bc[2][1], f2) : 0;
  long long c = lin(g, si, sj, sk);
  b[0] = __ldg(P.bccf + c);
  b[1] = __ldg(P.bccf + g.N + c);
  b[2] = C::DIM == 3 ? __ldg(P.bccf + 2 * g.N + c) : 0.0f;
  if (f0) b[0] = -b[0];
  if (f1) b[1] = -b[1];
  if (C::DIM == 3 && f2) b[2] = -b[2];
}

template <class C>
__device__ __forceinline__ void load_bccf_at(const Prm &P, long long c, float b[3]) {
  b[0] = b[1] = b[2] = 0.0f;
  if (!C::MHD) return;
  b[0] = __ldg(P.bccf + c);
  b[1] = __ldg(P.bccf + P.g.N + c);
  b[2] = C::DIM == 3 ? __ldg(P.bccf + 2 * P.g.N + c) : 0.0f;
}

// Riemann part of a face along d (face index fidx, face background bg): the edge states
// in the cell frame (qL/qR in the order of the FP32 state, transverse B in bL/bR; FASTEOS gammas
// gL/gR with the equilibrium gamma_e already added, or the face temperature guess tface of the
// Helmholtz configurations without FASTEOS) are rotated to the normal frame, the WB background
// and the face-normal B are added, and the flux and the induction flux Fb come back in the cell
// frame with rho_L + rho_R for the CT upwinding sign (source.F90:8138-9105 with the MHD parts
// 8327-8469, 8926-8959)
template <class C>
__device__ __forceinline__ void face_solve_split(const Prm &P, int d, long long fidx, const float4 &bg, float qL[C::NV],
                                                     float qR[C::NV], float bL[3], float bR[3], const float gLin[2],
                                                     const float gRin[2], float tface, bool flat, float F[C::NV],
                                                     float Fb[3], float &rho_sum) {
  constexpr int NV = C::NV, IP = C::IP;
  const Geo &g = P.g;
  if (C::MHD) {
    const float bn = (float)(P.bf[d][fidx] * P.inv_b_ref);
    bL[d] = bn;
    bR[d] = bn;
  }
  if (d == 1) {
    float a = qL[1], c = qL[2]; qL[1] = c; qL[2] = -a;
    a = qR[1]; c = qR[2]; qR[1] = c; qR[2] = -a;
    if (C::MHD) {
      a = bL[0]; c = bL[1]; bL[0] = c; bL[1] = -a;
      a = bR[0]; c = bR[1]; bR[0] = c; bR[1] = -a;
    }
  } else if (C::DIM == 3 && d == 2) {
    float a = qL[1], c = qL[2], e = qL[3]; qL[1] = e; qL[2] = a; qL[3] = c;
    a = qR[1]; c = qR[2]; e = qR[3]; qR[1] = e; qR[2] = a; qR[3] = c;
    if (C::MHD) {
      a = bL[0]; c = bL[1]; e = bL[2]; bL[0] = e; bL[1] = a; bL[2] = c;
      a = bR[0]; c = bR[1]; e = bR[2]; bR[0] = e; bR[1] = a; bR[2] = c;
    }
  }
  const float pe = bg.y;
  if (C::WB) {
    qL[0] = bg.x + qL[0];
    qR[0] = bg.x + qR[0];
  }
  float gL[2] = {gLin[0], gLin[1]}, gR[2] = {gRin[0], gRin[1]};
  if (!C::FAST && C::HELM) {
    split_side_eos<C>(P, qL, pe, tface, gL[0], gL[1]);
    split_side_eos<C>(P, qR, pe, tface, gR[0], gR[1]);
  }
  if constexpr (C::MHD)
    riemann_mhd_split<C::DIM, NV, C::EOSM, C::RIEM>(qL, qR, bL, bR, gL, gR, pe, (float)g.gm, (float)g.mach_cutoff, F,
                                                    Fb, flat, g.all_mach != 0);
  else
    riemann_hydro_split<C::DIM, NV, C::EOSM, C::RIEM>(qL, qR, gL, gR, pe, (float)g.gm, (float)g.mach_cutoff, F, flat,
                                                      g.all_mach != 0);
  if (d == 1) {
    float a = F[1], c = F[2]; F[1] = -c; F[2] = a;
    if (C::MHD) { a = Fb[0]; c = Fb[1]; Fb[0] = -c; Fb[1] = a; }
  } else if (C::DIM == 3 && d == 2) {
    float a = F[1], c = F[2], e = F[3]; F[1] = c; F[2] = e; F[3] = a;
    if (C::MHD) { a = Fb[0]; c = Fb[1]; e = Fb[2]; Fb[0] = c; Fb[1] = e; Fb[2] = a; }
  }
  rho_sum = qL[0] + qR[0];
  if (C::ETOT) F[IP] = F[IP] + F[0] * bg.w;
}

// flux through the low face of cell m along d from cells m-SW..m+SW-1 (w, gm, b: cells
// m-3..m+2); reconstruction, then face_solve_split
template <class C>
__device__ __forceinline__ void face_flux_split_rec(const Prm &P, int d, int fi, int fj, int fk, const float *const w[6],
                                                    const float *const gm[6], const float *const b[6], float F[C::NV],
                                                    float Fb[3], float &rho_sum) {
  constexpr int NV = C::NV;
  const Geo &g = P.g;
  bool fa = false, fb = false;  // USE_SHOCK_FLATTENING: is_flattened of cells m-1 and m
  if (C::SF) {
    fa = P.sf_flag[sf_flag_index<C>(g, fi - (d == 0), fj - (d == 1), fk - (d == 2))] != 0;
    fb = P.sf_flag[sf_flag_index<C>(g, fi, fj, fk)] != 0;
  }
  float qL[NV], qR[NV];
#pragma unroll
  for (int iv = 0; iv < NV; ++iv) {
    const float v[6] = {w[0][iv], w[1][iv], w[2][iv], w[3][iv], w[4][iv], w[5][iv]};
    rec_face_f32<C>(v, C::REC == REC_LIM5TH || iv >= C::IAS, qL[iv], qR[iv]);
    if (C::SF && C::REC != REC_LIM2ND) flatten_face_f32(v, fa, fb, qL[iv], qR[iv]);
  }
  float bL[3] = {0, 0, 0}, bR[3] = {0, 0, 0};
#pragma unroll
  for (int iv = 0; iv < C::DIM; ++iv) {
    if (!C::MHD || iv == d) continue;
    const float v[6] = {b[0][iv], b[1][iv], b[2][iv], b[3][iv], b[4][iv], b[5][iv]};
    rec_face_f32<C>(v, C::REC == REC_LIM5TH, bL[iv], bR[iv]);
    if (C::SF && C::REC != REC_LIM2ND) flatten_face_f32(v, fa, fb, bL[iv], bR[iv]);
  }
  float4 bg = make_float4(0.f, 0.f, 0.f, 0.f);
  if (C::WB) bg = __ldg(P.sf_bg[d] + bg_face(g, d, fi, fj, fk));
  float gL[2] = {0.f, 0.f}, gR[2] = {0.f, 0.f}, tface = 0.0f;
  if (C::FAST) {
    const bool late = C::SF && C::WB && d == 0;
    float gv[2][6];
#pragma unroll
    for (int iv = 0; iv < 2; ++iv) {
#pragma unroll
      for (int q = 0; q < 6; ++q) gv[iv][q] = gm[q][iv];
      rec_face_f32<C>(gv[iv], C::REC == REC_LIM5TH, gL[iv], gR[iv]);
      if (C::SF && C::REC != REC_LIM2ND && !late) flatten_face_f32(gv[iv], fa, fb, gL[iv], gR[iv]);
    }
    if (C::WB) {
      gL[0] = gL[0] + bg.z;
      gR[0] = gR[0] + bg.z;
      if (late) flatten_gamma_x1(gv, fa, fb, bg.z, gL, gR);
    }
  } else if (C::HELM) {
    tface = 0.5f * (gm[2][0] + gm[3][0]);
  }
  face_solve_split<C>(P, d, face_lin(g, d, fi, fj, fk), bg, qL, qR, bL, bR, gL, gR, tface, C::SF && (fa || fb), F,
                          Fb, rho_sum);
}

// FP32 face EMF components (units v_ref b_ref) and the CT mass-flux sign (source.F90:8926-8951)
template <class C>
__device__ __forceinline__ void store_face_emf_split(const Prm &P, int d, long long fidx, int q, const float Fb[3],
                                                     float frho, float rho_sum, float smax_s) {
  const Geo &g = P.g;
  long long nf = nfaces(g, d);
  float *e = P.femf[d];
  if (d == 0) { if (C::DIM == 3) e[1 * nf + fidx] = Fb[2]; e[2 * nf + fidx] = -Fb[1]; }
  if (d == 1) { if (C::DIM == 3) e[0 * nf + fidx] = -Fb[2]; e[2 * nf + fidx] = Fb[0]; }
  if (d == 2) { e[0 * nf + fidx] = Fb[1]; e[1 * nf + fidx] = -Fb[0]; }
  // the reference's dead band |f_rho| / (rho_bar smax) <= mach_ct in physical units: with f_rho and
  // rho in scaled units the ratio carries one factor v_ref, folded into smax_s = smax / v_ref
  const float band = (float)g.mach_ct * (0.5f * rho_sum * smax_s);
  float sgn = 0.0f;
  if (frho > band) sgn = 1.0f;
  if (frho < -band) sgn = -1.0f;
  // a reflective wall face has mirror-image states and no mass flux: the reference (no FMA) gets
  // exactly zero there, while FP32 with contracted products leaves a rounding residue whose sign
  // would select an upwind side; the wall's dead-band value is restored explicitly (q is the
  // face's index along d)
  if ((q == 0 && g.bc[d][0] != BC_PERIODIC) || (q == g.nx[d] && g.bc[d][1] != BC_PERIODIC)) sgn = 0.0f;
  P.fsgn[d][fidx] = sgn;
}

// Stage, part 1: one thread per face of direction d solves it once: the FP32 flux goes to
// P.fflux[d] ([NV][faces]), the face EMF and the CT sign to their arrays
// (one instantiation per direction D: index strides and rotations fold into constants)
template <class C, int D>
__device__ __forceinline__ void face_split_at(const Prm &P, long long f) {
  constexpr int d = D;
  constexpr int NV = C::NV;
  const Geo &g = P.g;
  const long long nf = nfaces(g, d);
  int fi, fj, fk;
  unflatten3(f, g.div0[d == 0], g.div1[d == 1], fi, fj, fk);
  // cells m-3 .. m+2 (the reconstruction reads m-SW .. m+SW-1); a stencil inside the domain
  // is read by linear index, one at a boundary maps each ghost index
  float w[6][NV], gm4[6][2], b4[6][3];
  const int fd = d == 0 ? fi : (d == 1 ? fj : fk);
  const bool inside = fd >= C::SW && fd + C::SW <= g.nx[d];
  const long long base = lin(g, fi, fj, fk), stride = dir_stride(g, d);
#pragma unroll
  for (int s = 0; s < 6; ++s) {
    gm4[s][0] = gm4[s][1] = 0.0f;
    b4[s][0] = b4[s][1] = b4[s][2] = 0.0f;
    if (s < 3 - C::SW || s >= 3 + C::SW) {
#pragma unroll
      for (int iv = 0; iv < NV; ++iv) w[s][iv] = 0.0f;
      continue;
    }
    if (inside) {
      const long long c = base + (s - 3) * stride;
      load_wf_at<C>(P, c, w[s], gm4[s]);
      load_bccf_at<C>(P, c, b4[s]);
    } else {
      const int ii = fi + (d == 0 ? s - 3 : 0), jj = fj + (d == 1 ? s - 3 : 0), kk = fk + (d == 2 ? s - 3 : 0);
      load_wf<C>(P, ii, jj, kk, w[s], gm4[s]);
      load_bccf<C>(P, ii, jj, kk, b4[s]);
    }
  }
  const float *const wv[6] = {w[0], w[1], w[2], w[3], w[4], w[5]};
  const float *const gv[6] = {gm4[0], gm4[1], gm4[2], gm4[3], gm4[4], gm4[5]};
  const float *const bv[6] = {b4[0], b4[1], b4[2], b4[3], b4[4], b4[5]};
  float F[NV], Fb[3], rs;
  face_flux_split_rec<C>(P, d, fi, fj, fk, wv, gv, bv, F, Fb, rs);
  FluxPlanes<NV>::store(P.fflux[d], nf, f, F);
  if (C::MHD) store_face_emf_split<C>(P, d, f, d == 0 ? fi : (d == 1 ? fj : fk), Fb, F[0], rs, (float)(P.scal[2] * P.inv_v_ref));
}

template <class C, int D>
__global__ void __launch_bounds__(128, C::MINB_FACE32) k_face_split(Prm P) {
  if (!*P.active) return;
  const long long f = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= nfaces(P.g, D)) return;
  face_split_at<C, D>(P, f);
}

// faces per thread of the walking face kernels: along x (threads of a warp step K0 cells apart,
// so their loads stay within a few cache lines) and along y, z (threads of a warp are
// neighbours in x and walk side by side)
constexpr int WALK_K0 = 4, WALK_K = 8;
// grid of the rescue-queue kernels: 4 blocks of 128 threads per SM of a B200 (148 SMs)
constexpr int RESCUE_BLOCKS = 4 * 148;
// resident blocks of 128 threads per SM the face kernels are compiled for.  The packed solver keeps
// its values in register pairs: walks at 5 (96 registers, almost no spills) ran the x2 faces of a
// 128^3 MHD stage in 57 us against 78 at 6 (80 registers) and more at 7; the row kernel carries
// nothing between faces and needs 72 registers.  Without USE_FASTEOS, where each face runs two FP64
// (rho, P) -> T solves, 4 (128 registers): a 256^3 MHD step took 36.9 ms against 43.4 with the
// registers unbounded (253 registers, 2 blocks per SM), 37.5 at 3
constexpr int WALK_MINB = 5, WALK_MINB_GIVEN = 4, ROW_MINB = 6;

// Raw values of one cell for the walking face kernel along D: the FP32 state (0 .. NV-1), the
// cell B components transverse to D (NBT of them from NV on; the component along D is not
// reconstructed, the face carries it) and the two FASTEOS gammas or the temperature (IG, IG+1).
template <class C, int D>
struct WalkCell {
  static constexpr int NBT = C::MHD ? C::DIM - 1 : 0, IG = C::NV + NBT, NR = IG + 2;
  // cell B component held in transverse slot t
  static __device__ __forceinline__ constexpr int comp(int t) { return t < D ? t : t + 1; }
};

// q is the cell's index along D and c[] its other two coordinates; a cell inside the domain
// along D is read by linear index lc, a ghost maps its index.
template <class C, int D>
__device__ __forceinline__ void load_walk_cell(const Prm &P, const int c[3], int q, long long lc,
                                               float r[WalkCell<C, D>::NR]) {
  using L = WalkCell<C, D>;
  float *gm = r + L::IG;
  gm[0] = gm[1] = 0.0f;
  if (q >= 0 && q < P.g.nx[D]) {
    load_wf_at<C>(P, lc, r, gm);
#pragma unroll
    for (int t = 0; t < L::NBT; ++t) r[C::NV + t] = __ldg(P.bccf + L::comp(t) * P.g.N + lc);
  } else {
    const int i = D == 0 ? q : c[0], j = D == 1 ? q : c[1], k = D == 2 ? q : c[2];
    float b[3];
    load_wf<C>(P, i, j, k, r, gm);
    load_bccf<C>(P, i, j, k, b);
#pragma unroll
    for (int t = 0; t < L::NBT; ++t) r[C::NV + t] = b[L::comp(t)];
  }
}

// One face along D from the edge values of its two sides (WalkCell order; hip: high side of the cell
// below, lo: low side of the cell above): background, solve, stores.  q is the face's index along D,
// j its x2 index, fidx its linear index.
template <class C, int D>
__device__ __forceinline__ void face_from_edges(const Prm &P, long long fidx, int q, int j, const float *hip,
                                                const float *lo, float tface, bool fa, bool fb, float smax_s) {
  using L = WalkCell<C, D>;
  constexpr int NV = C::NV, IG = L::IG;
  const Geo &g = P.g;
  float qL[NV], qR[NV], bL[3] = {0.f, 0.f, 0.f}, bR[3] = {0.f, 0.f, 0.f}, gL[2] = {0.f, 0.f}, gR[2] = {0.f, 0.f};
#pragma unroll
  for (int iv = 0; iv < NV; ++iv) {
    qL[iv] = hip[iv];
    qR[iv] = lo[iv];
  }
#pragma unroll
  for (int t = 0; t < L::NBT; ++t) {
    bL[L::comp(t)] = hip[NV + t];
    bR[L::comp(t)] = lo[NV + t];
  }
  float4 bg = make_float4(0.f, 0.f, 0.f, 0.f);
  if (C::WB) bg = __ldg(P.sf_bg[D] + (g.bg_profile ? (long long)j : fidx));
  if (C::FAST) {
    gL[0] = hip[IG]; gL[1] = hip[IG + 1];
    gR[0] = lo[IG]; gR[1] = lo[IG + 1];
    if (C::WB) {
      gL[0] = gL[0] + bg.z;
      gR[0] = gR[0] + bg.z;
      // the x1 sweep's gamma handling on flagged faces (flatten_gamma_x1 with the LIM2ND
      // edges already at hand)
      if (C::SF && D == 0) {
        if (fa) { gL[0] = hip[IG]; gL[1] = hip[IG + 1]; gR[0] = gR[0] + bg.z; }
        if (fb) { gR[0] = lo[IG]; gR[1] = lo[IG + 1]; gL[0] = gL[0] + bg.z; }
      }
    }
  }
  float F[NV], Fb[3], rs;
  face_solve_split<C>(P, D, fidx, bg, qL, qR, bL, bR, gL, gR, tface, C::SF && (fa || fb), F, Fb, rs);
  FluxPlanes<NV>::store(P.fflux[D], nfaces(g, D), fidx, F);
  if (C::MHD) store_face_emf_split<C>(P, D, fidx, q, Fb, F[0], rs, smax_s);
}

// Stage, part 1 for LIM2ND reconstruction: one thread walks K consecutive faces along D.  A
// cell borders two faces of the walk, so its values are loaded and its PLM slope formed once
// (the per-face kernel does both twice) and its edge values are carried to the next face.  The
// faces, their arithmetic and the stored results are those of k_face_split.
template <class C, int D, int K>
__global__ void __launch_bounds__(128, C::EOSM == EOS_GIVEN ? WALK_MINB_GIVEN : WALK_MINB) k_face_split_walk(Prm P) {
  static_assert(C::REC == REC_LIM2ND, "the walk carries LIM2ND edge values");
  if (!*P.active) return;
  using L = WalkCell<C, D>;
  constexpr int NV = C::NV, NR = L::NR, IG = L::IG;
  const Geo &g = P.g;
  const int nd = g.nx[D] + 1, nch = (nd + K - 1) / K;
  const int e0 = D == 0 ? nch : g.nx[0], e1 = D == 1 ? nch : g.nx[1];
  const int e2 = D == 2 ? nch : (C::DIM == 3 ? g.nx[2] : 1);
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)e0 * e1 * e2) return;
  int c[3];
  unflatten3(t, e0, e1, c[0], c[1], c[2]);
  const int q0 = c[D] * K, qend = min(q0 + K, nd);
  c[D] = 0;
  const long long nf = nfaces(g, D), cstride = dir_stride(g, D);
  const long long fstride = D == 0 ? 1 : (D == 1 ? (long long)g.nx[0] : (long long)g.nx[0] * g.nx[1]);
  const long long crow = lin(g, c[0], c[1], c[2]), frow = face_lin(g, D, c[0], c[1], c[2]);
  const long long sfrow = C::SF ? sf_flag_index<C>(g, c[0], c[1], c[2]) : 0;
  const long long sfstride = D == 0 ? 1 : (D == 1 ? (long long)(g.nx[0] + 2) : (long long)(g.nx[0] + 2) * (g.nx[1] + 2));
  const float smax_s = (float)(P.scal[2] * P.inv_v_ref);
  // window: rc = cell q, sb = its difference to cell q-1, hip = edge values at the high side of
  // cell q-1
  float rc[NR], sb[NR], rp[NR], lo[NR], hip[NR];
  float tm = 0.0f;  // without USE_FASTEOS: the temperature of cell q-1
  {
    float rm[NR];
    load_walk_cell<C, D>(P, c, q0 - 2, crow + (long long)(q0 - 2) * cstride, rm);
    load_walk_cell<C, D>(P, c, q0 - 1, crow + (long long)(q0 - 1) * cstride, rc);
    load_walk_cell<C, D>(P, c, q0, crow + (long long)q0 * cstride, rp);
#pragma unroll
    for (int v = 0; v < NR; ++v) {
      const float sf = rp[v] - rc[v];
      hip[v] = fmaf(0.5f, plm_slope_f32(sf, rc[v] - rm[v]), rc[v]);
      sb[v] = sf;
    }
    if (!C::FAST && C::HELM) tm = rc[IG];
#pragma unroll
    for (int v = 0; v < NR; ++v) rc[v] = rp[v];
  }
  bool fprev = C::SF && P.sf_flag[sfrow + (long long)(q0 - 1) * sfstride] != 0;
#pragma unroll 1
  for (int q = q0; q < qend; ++q) {
    load_walk_cell<C, D>(P, c, q + 1, crow + (long long)(q + 1) * cstride, rp);
    float hi[NR];
#pragma unroll
    for (int v = 0; v < NR; ++v) {
      const float sf = rp[v] - rc[v], slope = plm_slope_f32(sf, sb[v]);
      lo[v] = fmaf(-0.5f, slope, rc[v]);
      hi[v] = fmaf(0.5f, slope, rc[v]);
      sb[v] = sf;
    }
    const bool fa = fprev, fb = C::SF && P.sf_flag[sfrow + (long long)q * sfstride] != 0;
    const long long fidx = frow + (long long)q * fstride;
    float tface = 0.0f;
    if (!C::FAST && C::HELM) {
      tface = 0.5f * (tm + rc[IG]);
      tm = rc[IG];
    }
    face_from_edges<C, D>(P, fidx, q, D == 1 ? q : c[1], hip, lo, tface, fa, fb, smax_s);
#pragma unroll
    for (int v = 0; v < NR; ++v) {
      hip[v] = hi[v];
      rc[v] = rp[v];
    }
    fprev = fb;
  }
}

// Stage, part 1 for LIM2ND along x1: a warp takes 32 neighbouring cells of a row and solves the
// 29 faces whose stencils they hold.  A lane loads one cell (coalesced, all loads at once); the
// differences and edge values of its neighbours come by shuffle, each slope is formed once, and
// nothing is carried between faces, so the kernel needs no shared memory, no barrier and any row
// length fits.  Lanes 0, 1 and 31 hold the stencil's rim: lane l (2 <= l < 31) solves the face
// below its cell.  Bound by issue slots (70% of the cycles issue, 750 instructions a face); 67 us
// for the x1 faces of a 128^3 MHD stage, where tiles staged in shared memory by bulk copies (766
// instructions, two block barriers a tile) took 83 and a walk of 4 faces 1% more per stage.
template <class C>
__global__ void __launch_bounds__(128, ROW_MINB) k_face_split_row(Prm P, FastDiv chunks) {
  static_assert(C::REC == REC_LIM2ND, "the row kernel forms LIM2ND edges");
  if (!*P.active) return;
  using L = WalkCell<C, 0>;
  constexpr int NR = L::NR, IG = L::IG;
  constexpr unsigned ALL = 0xffffffffu;
  const Geo &g = P.g;
  const unsigned w = (unsigned)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  int c[3], ch;
  unflatten3(w, chunks, g.div1[0], ch, c[1], c[2]);
  if (c[2] >= g.nx[2]) return;
  c[0] = 0;
  // this lane's cell, which is also the index of the face below it; past the upper ghost layer
  // the value is not used
  const int i = min(ch * ROW_FACES - 2 + (int)lane, g.nx[0] + 1);
  float rc[NR], hip[NR], lo[NR];
  load_walk_cell<C, 0>(P, c, i, lin(g, 0, c[1], c[2]) + i, rc);
#pragma unroll
  for (int v = 0; v < NR; ++v) {
    const float sf = __shfl_down_sync(ALL, rc[v], 1) - rc[v];
    const float slope = plm_slope_f32(sf, __shfl_up_sync(ALL, sf, 1));
    lo[v] = fmaf(-0.5f, slope, rc[v]);
    hip[v] = __shfl_up_sync(ALL, fmaf(0.5f, slope, rc[v]), 1);
  }
  float tface = 0.0f;
  if (!C::FAST && C::HELM) tface = 0.5f * (__shfl_up_sync(ALL, rc[IG], 1) + rc[IG]);
  if (lane < 2 || lane > 30 || ch * ROW_FACES - 2 + (int)lane > g.nx[0]) return;
  bool fa = false, fb = false;
  if (C::SF) {
    const long long m = sf_flag_index<C>(g, i, c[1], c[2]);
    fa = P.sf_flag[m - 1] != 0;
    fb = P.sf_flag[m] != 0;
  }
  face_from_edges<C, 0>(P, face_lin(g, 0, i, c[1], c[2]), i, c[1], hip, lo, tface, fa, fb,
                        (float)(P.scal[2] * P.inv_v_ref));
}

// FP32 face EMF / sign at a possibly-ghost transverse index (periodic wrap, or the reflective
// EMF BC: the wall-normal component keeps its sign, the others flip; source.F90:11374-11964)
template <class C>
__device__ __forceinline__ void face_emf_split_at(const Prm &P, int d, int comp, int i, int j, int k, float &e,
                                                  float &sgn) {
  const Geo &g = P.g;
  int c[3] = {i, j, k};
  float fac = 1.0f;
#pragma unroll
  for (int d2 = 0; d2 < C::DIM; ++d2) {
    if (d2 == d) continue;
    int n = g.nx[d2];
    if (c[d2] < 0) {
      if (g.bc[d2][0] == BC_PERIODIC) c[d2] += n;
      else { c[d2] = 0; if (comp != d2) fac = -fac; }
    } else if (c[d2] >= n) {
      if (g.bc[d2][1] == BC_PERIODIC) c[d2] -= n;
      else { c[d2] = n - 1; if (comp != d2) fac = -fac; }
    }
  }
  long long f = face_lin(g, d, c[0], c[1], c[2]);
  e = fac * P.femf[d][(long long)comp * nfaces(g, d) + f];
  sgn = P.fsgn[d][f];
}

// cell-centred -v x B (components 0..2) of FP32 velocity v and cell B b (scaled units)
__device__ __forceinline__ void cell_emf3(const float v[3], const float b[3], float e[3]) {
  e[2] = -v[0] * b[1] + v[1] * b[0];
  e[0] = v[2] * b[1] - v[1] * b[2];
  e[1] = v[0] * b[2] - v[2] * b[0];
}
// the stage input's cell EMFs, written by the kernel that produced its FP32 state (2D has corners
// along x3 only)
template <class C>
__device__ __forceinline__ void store_cell_emf(const Prm &P, long long c, const float v[3], const float b[3]) {
  float e[3];
  cell_emf3(v, b, e);
#pragma unroll
  for (int a = C::DIM == 3 ? 0 : 2; a < 3; ++a) P.fecell[(long long)a * P.g.N + c] = e[a];
}

// cell-centred -v x B component a of a (possibly ghost) cell from the stored cell EMFs: a mirror
// in dimension d != a flips one factor of each product of component a
template <class C>
__device__ __forceinline__ float emf_cell_split(const Prm &P, int a, int i, int j, int k) {
  const Geo &g = P.g;
  bool f0 = false, f1 = false, f2 = false;
  int si = map_index(i, g.nx[0], g.bc[0][0], g.bc[0][1], f0);
  int sj = map_index(j, g.nx[1], g.bc[1][0], g.bc[1][1], f1);
  int sk = C::DIM == 3 ? map_index(k, g.nx[2], g.bc[2][0], g.bc[2][1], f2) : 0;
  float e = __ldg(P.fecell + (long long)a * g.N + lin(g, si, sj, sk));
  const bool flip = (a != 0 && f0) != ((a != 1 && f1) != (a != 2 && f2));
  return flip ? -e : e;
}

// corner EMF along axis A (source.F90:11966-12206), FP32, at corner (c[0], c[1], c[2]); INTERIOR:
// all four faces and cells lie inside the domain (linear indices, no wrap or mirror)
template <class C, int A, bool INTERIOR>
__device__ __forceinline__ float corner_emf_split(const Prm &P, const int c[3]) {
  constexpr int a = A, pa = A == 2 ? 0 : (A == 0 ? 1 : 2), qa = A == 2 ? 1 : (A == 0 ? 2 : 0);
  const Geo &g = P.g;
  float emf_N, emf_E, emf_S, emf_W, sgS, sgN, sgW, sgE, emf_SW, emf_NW, emf_NE, emf_SE;
  if (INTERIOR) {
    const long long fp = face_lin(g, pa, c[0], c[1], c[2]), fq = face_lin(g, qa, c[0], c[1], c[2]);
    const int p0 = g.nx[0] + (pa == 0), p1 = g.nx[1] + (pa == 1);  // face array of pa
    const int q0 = g.nx[0] + (qa == 0), q1 = g.nx[1] + (qa == 1);  // face array of qa
    const long long sp_q = qa == 0 ? 1 : (qa == 1 ? (long long)p0 : (long long)p0 * p1);  // step along qa
    const long long sq_p = pa == 0 ? 1 : (pa == 1 ? (long long)q0 : (long long)q0 * q1);  // step along pa
    const float *ep = P.femf[pa] + (long long)a * nfaces(g, pa), *eq = P.femf[qa] + (long long)a * nfaces(g, qa);
    emf_N = __ldg(ep + fp); sgN = __ldg(P.fsgn[pa] + fp);
    emf_S = __ldg(ep + fp - sp_q); sgS = __ldg(P.fsgn[pa] + fp - sp_q);
    emf_E = __ldg(eq + fq); sgE = __ldg(P.fsgn[qa] + fq);
    emf_W = __ldg(eq + fq - sq_p); sgW = __ldg(P.fsgn[qa] + fq - sq_p);
    const long long cc = lin(g, c[0], c[1], c[2]);
    const long long cp = pa == 0 ? 1 : (pa == 1 ? (long long)g.nx[0] : (long long)g.nx[0] * g.nx[1]);
    const long long cq = qa == 0 ? 1 : (qa == 1 ? (long long)g.nx[0] : (long long)g.nx[0] * g.nx[1]);
    const float *ec = P.fecell + (long long)a * g.N;
    emf_NE = __ldg(ec + cc);
    emf_NW = __ldg(ec + cc - cp);
    emf_SE = __ldg(ec + cc - cq);
    emf_SW = __ldg(ec + cc - cp - cq);
  } else {
    int cqm[3] = {c[0], c[1], c[2]}; cqm[qa] -= 1;
    int cpm[3] = {c[0], c[1], c[2]}; cpm[pa] -= 1;
    int cpq[3] = {c[0], c[1], c[2]}; cpq[pa] -= 1; cpq[qa] -= 1;
    face_emf_split_at<C>(P, pa, a, c[0], c[1], c[2], emf_N, sgN);
    face_emf_split_at<C>(P, qa, a, c[0], c[1], c[2], emf_E, sgE);
    face_emf_split_at<C>(P, pa, a, cqm[0], cqm[1], cqm[2], emf_S, sgS);
    face_emf_split_at<C>(P, qa, a, cpm[0], cpm[1], cpm[2], emf_W, sgW);
    emf_SW = emf_cell_split<C>(P, a, cpq[0], cpq[1], cpq[2]);
    emf_NW = emf_cell_split<C>(P, a, cpm[0], cpm[1], cpm[2]);
    emf_NE = emf_cell_split<C>(P, a, c[0], c[1], c[2]);
    emf_SE = emf_cell_split<C>(P, a, cqm[0], cqm[1], cqm[2]);
  }
  float sgn = sgS;
  float demf_S = 0.5f * (1.0f + sgn) * (emf_W - emf_SW) + 0.5f * (1.0f - sgn) * (emf_E - emf_SE);
  sgn = sgN;
  float demf_N = 0.5f * (1.0f + sgn) * (emf_NW - emf_W) + 0.5f * (1.0f - sgn) * (emf_NE - emf_E);
  sgn = sgW;
  float demf_W = 0.5f * (1.0f + sgn) * (emf_S - emf_SW) + 0.5f * (1.0f - sgn) * (emf_N - emf_NW);
  sgn = sgE;
  float demf_E = 0.5f * (1.0f + sgn) * (emf_SE - emf_S) + 0.5f * (1.0f - sgn) * (emf_NE - emf_N);
  return 0.25f * (emf_S + emf_W + emf_N + emf_E + demf_S - demf_N + demf_W - demf_E);
}

// Corner EMFs of every axis, one thread per grid node (i, j, k): the corner of axis a whose lower
// end is the node.  A node's three corners share their index arithmetic, the signs of the node's
// faces and the cache lines of its cells; one launch a stage.  The first nin_blocks blocks take
// the interior nodes (1 <= index < nx in every dimension), which read faces and cells by linear
// index with no branch; the blocks after them take the nodes on the domain's faces, whose corners
// map their ghost indices (threads over all nodes in array order had a quarter of their warps
// diverge into the mapping path, where the rows of nodes, nx + 1 long, straddle the warps).
// Bound by its loads: 36 B of face EMFs and signs, 12 B of cell EMFs in, 12 B out per cell.
template <class C>
__global__ void __launch_bounds__(256) k_corner_split(Prm P, unsigned nin_blocks, FastDiv e0, FastDiv e1) {
  if (!*P.active) return;
  const Geo &g = P.g;
  int c[3];
  if (blockIdx.x < nin_blocks) {
    // e0 and e1 are nx - 1 of x1 and x2
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)e0.d * e1.d * (C::DIM == 3 ? g.nx[2] - 1 : 1)) return;
    unflatten3(t, e0, e1, c[0], c[1], c[2]);
    c[0] += 1;
    c[1] += 1;
    if (C::DIM == 3) {
      c[2] += 1;
      P.fcor[0][cor_lin(g, 0, c[0], c[1], c[2])] = corner_emf_split<C, 0, true>(P, c);
      P.fcor[1][cor_lin(g, 1, c[0], c[1], c[2])] = corner_emf_split<C, 1, true>(P, c);
    }
    P.fcor[2][cor_lin(g, 2, c[0], c[1], c[2])] = corner_emf_split<C, 2, true>(P, c);
    return;
  }
  if (!rim_node<C>(g, (long long)(blockIdx.x - nin_blocks) * blockDim.x + threadIdx.x, c)) return;
  if (C::DIM == 3) {
    if (c[0] < g.nx[0]) P.fcor[0][cor_lin(g, 0, c[0], c[1], c[2])] = corner_emf_split<C, 0, false>(P, c);
    if (c[1] < g.nx[1]) P.fcor[1][cor_lin(g, 1, c[0], c[1], c[2])] = corner_emf_split<C, 1, false>(P, c);
    if (c[2] >= g.nx[2]) return;
  }
  P.fcor[2][cor_lin(g, 2, c[0], c[1], c[2])] = corner_emf_split<C, 2, false>(P, c);
}

// face-B update (source.F90:12208-12437) in FP64 from the FP32 corner EMFs; one thread per grid
// node (i, j, k), which updates the low face of cell (i, j, k) in every direction (the three
// share corner EMFs: 9 loads for the three faces, most of them cache hits).  Bound by memory:
// 12 B of corner EMFs in, and B and B0 in and B out in FP64 (72 B) per cell.
template <class C>
__global__ void __launch_bounds__(256) k_bface_split(Prm P) {
  if (!*P.active) return;
  const Geo &g = P.g;
  const int n0 = g.nx[0], n1 = g.nx[1], n2 = g.nx[2];
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)(n0 + 1) * (n1 + 1) * (C::DIM == 3 ? n2 + 1 : 1)) return;
  int i, j, k;
  unflatten3(t, g.div0[1], g.div1[1], i, j, k);
  const bool in0 = i < n0, in1 = j < n1, in2 = C::DIM == 2 || k < n2;
  const double dt = P.scal[1];
  const double a1 = P.a1, a2 = P.a2, a3 = P.c3 * dt * (P.v_ref * P.b_ref);
  // differences of the FP32 corner EMFs are formed in FP64 (exact), so the discrete divergence
  // of the update cancels to FP64 rounding as in the FP64 form
  auto e = [&](int a, long long q) { return (double)__ldg(P.fcor[a] + q); };
  // where each corner array continues along the other two directions
  const long long q2 = cor_lin(g, 2, i, j, k), q2y = n0 + 1;
  auto update = [&](int d, double tmp) {
    const long long f = face_lin(g, d, i, j, k);
    const double b = P.bf[d][f];
    double b0;
    if (P.first_stage) { b0 = b; P.b0f[d][f] = b; } else { b0 = P.b0f[d][f]; }
    P.bf[d][f] = a1 * b0 + a2 * b + a3 * tmp;
  };
  if (C::DIM == 2) {
    const double E3 = e(2, q2);
    if (in1) update(0, (e(2, q2 + q2y) - E3) * g.inv_dx[1]);
    if (in0) update(1, (E3 - e(2, q2 + 1)) * g.inv_dx[0]);
    return;
  }
  const long long q0 = cor_lin(g, 0, i, j, k), q0y = n0, q0z = (long long)n0 * (n1 + 1);
  const long long q1 = cor_lin(g, 1, i, j, k), q1z = (long long)(n0 + 1) * n1;
  // E1 exists for i < nx1, E2 for j < nx2, E3 for k < nx3
  const double E1 = in0 ? e(0, q0) : 0.0, E2 = in1 ? e(1, q1) : 0.0, E3 = in2 ? e(2, q2) : 0.0;
  if (in1 && in2) update(0, -(e(1, q1 + q1z) - E2) * g.inv_dx[2] + (e(2, q2 + q2y) - E3) * g.inv_dx[1]);
  if (in0 && in2) update(1, (e(0, q0 + q0z) - E1) * g.inv_dx[2] + (E3 - e(2, q2 + 1)) * g.inv_dx[0]);
  if (in0 && in1) update(2, (e(1, q1 + 1) - E2) * g.inv_dx[0] - (e(0, q0 + q0y) - E1) * g.inv_dx[1]);
}

// cells per block of the cons->prim kernels
constexpr int C2P_BLOCK = 128;
// New state of one cell that the EoS part of cons->prim needs (the rest is stored before it)
struct C2pState {
  double rho = 1.0, inv_rho = 1.0, eint = 0.0, ye = 0.0, inv_abar = 1.0;
  double Tw = 0.0;  // the stage input's temperature (the Newton's warm start), loaded up front
  long long bc = 0;
};

// Stage, part 3a: flux divergence from the face fluxes, gravity and the RK combine of U
// (FP64), b_cc from the updated faces (FP64); stores U (U0 in the first stage), scaled b_cc and
// what depends on the conserved state alone (FP32 velocities and scalars, cell EMFs), and
// returns what the EoS part needs
// (given: the flux divergence in scaled units, from the kernel that solved the faces itself)
template <class C>
__device__ __forceinline__ void c2p_split_combine(const Prm &P, long long c, C2pState &cs, const float *given = nullptr) {
  constexpr int NV = C::NV, IP = C::IP, IAS = C::IAS, DIM = C::DIM;
  const Geo &g = P.g;
  double &rho = cs.rho, &inv_rho = cs.inv_rho, &eint = cs.eint, &ye = cs.ye, &inv_abar = cs.inv_abar;
  long long &bc = cs.bc;
  {
    int i, j, k;
    unflatten3(c, g.div0[0], g.div1[0], i, j, k);
    bc = bg_cc(g, i, j, k);
    double bcc[3] = {0, 0, 0}, u[NV];
    // the running and initial conserved state travel to shared memory (each thread its own cell's,
    // so no barrier) while the fluxes are read: with all 56 loads through the 64 to 72 registers a
    // thread has here they went out in small batches, each waiting for the memory
    __shared__ double su[2 * NV][C2P_BLOCK];
    const int tid = threadIdx.x;
#pragma unroll
    for (int iv = 0; iv < NV; ++iv) cp_async8(&su[iv][tid], P.U + (long long)iv * g.N + c);
    if (!P.first_stage) {
#pragma unroll
      for (int iv = 0; iv < NV; ++iv) cp_async8(&su[NV + iv][tid], P.U0 + (long long)iv * g.N + c);
    }
    cp_async_commit();
#pragma unroll
    for (int d = 0; d < DIM && C::MHD; ++d) {
      int ui = i + (d == 0), uj = j + (d == 1), uk = k + (d == 2);
      bcc[d] = 0.5 * (P.bf[d][face_lin(g, d, ui, uj, uk)] + P.bf[d][face_lin(g, d, i, j, k)]);
      P.bccf[(long long)d * g.N + c] = (float)(bcc[d] * P.inv_b_ref);
    }
    // flux divergence (directions in the order of the hydro stage), gravity, RK combine
    float res[NV];
    if (given) {
#pragma unroll
      for (int iv = 0; iv < NV; ++iv) res[iv] = given[iv];
    }
#pragma unroll
    for (int d = 0; d < DIM && !given; ++d) {
      const long long nf = nfaces(g, d);
      float lo[NV], hi[NV];
      FluxPlanes<NV>::load(P.fflux[d], nf, face_lin(g, d, i, j, k), lo);
      FluxPlanes<NV>::load(P.fflux[d], nf, face_lin(g, d, i + (d == 0), j + (d == 1), k + (d == 2)), hi);
      const float inv_dl = (float)g.inv_dx[d];
#pragma unroll
      for (int iv = 0; iv < NV; ++iv) {
        float dd = (hi[iv] - lo[iv]) * inv_dl;
        res[iv] = d == 0 ? dd : res[iv] + dd;
      }
    }
    const double fm = P.rho_ref * P.v_ref, fe = P.p_ref * P.v_ref;
    double rd[NV];
    rd[0] = (double)res[0] * fm;
#pragma unroll
    for (int d = 0; d < DIM; ++d) rd[1 + d] = (double)res[1 + d] * P.p_ref;
    rd[IP] = (double)res[IP] * fe;
#pragma unroll
    for (int iv = IAS; iv < NV; ++iv) rd[iv] = (double)res[iv] * fm;
    if (C::GRAV) {
      const double rho_dev_phys = (double)P.Wf_in[c] * P.rho_ref;
#pragma unroll
      for (int d = 0; d < DIM; ++d)
        rd[1 + d] -= rho_dev_phys * __ldg(P.grav + (long long)d * (g.bg_profile ? g.nx[1] : g.N) + bc);
    }
    {
      const double dt = P.scal[1], a1 = P.a1, a2 = P.a2, a3 = P.c3 * dt;
      double un[NV];
      cp_async_wait_all();
#pragma unroll
      for (int iv = 0; iv < NV; ++iv) un[iv] = su[iv][tid];
      if (g.use_acc) constant_acceleration<DIM, IP>(g, un, rd);
#pragma unroll
      for (int iv = 0; iv < NV; ++iv) {
        double u0;
        if (P.first_stage) {
          u0 = un[iv];
          P.U0[(long long)iv * g.N + c] = un[iv];
        } else {
          u0 = su[NV + iv][tid];
        }
        u[iv] = a1 * u0 + a2 * un[iv] + a3 * rd[iv];
        P.U[(long long)iv * g.N + c] = u[iv];
      }
    }
    rho = u[0];
    inv_rho = 1.0 / rho;
    double ke = u[1] * u[1] + u[2] * u[2] + (DIM == 3 ? u[3] * u[3] : 0.0);
    eint = u[IP] - 0.5 * ke * inv_rho;
    if (C::MHD) eint = eint - 0.5 * (bcc[0] * bcc[0] + bcc[1] * bcc[1] + bcc[2] * bcc[2]);
    if (C::ETOT) eint = eint - rho * __ldg(P.phi_cc + bc);
    float vf[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      vf[d] = (float)(u[1 + d] * inv_rho * P.inv_v_ref);
      P.Wf_out[(long long)(1 + d) * g.N + c] = vf[d];
    }
    if (C::MHD) {
      const float bf3[3] = {(float)(bcc[0] * P.inv_b_ref), (float)(bcc[1] * P.inv_b_ref),
                            DIM == 3 ? (float)(bcc[2] * P.inv_b_ref) : 0.0f};
      store_cell_emf<C>(P, c, vf, bf3);
    }
#pragma unroll
    for (int iv = IAS; iv < NV; ++iv) P.Wf_out[(long long)iv * g.N + c] = (float)(u[iv] * inv_rho);
    if (C::HELM) {
      ye = u[IAS] * inv_rho;
      inv_abar = u[IAS + 1] * inv_rho;
    }
  }
}

// Temperature guess of the split MHD cons->prim Newton
enum { C2P_WARM = 0,    // the previous stage's temperature (the reference's warm start)
       C2P_LEARNED = 1, // the network's guess, judged by <= 3 Newton iterations
       C2P_RESCUE = 2   // the warm start; a cell whose first Newton correction exceeds
                        // RESCUE_STEP * T is queued for the learned guess instead
};
// first warm-start correction (relative) above which a cell is handed to the learned guess: the
// network's guesses are within ~0.2% (0.001 dex); from a start 2% off the warm Newton needs
// ~4 more iterations, from the learned guess ~3 in all
constexpr double RESCUE_STEP = 0.02;

// Stage, part 3b: cons -> prim of the new state with the Helmholtz Newton (FP64) from the
// warm guess (the previous stage's temperature), or (C2P_LEARNED) from the network's guess lT
// (log10 T; NaN for none): the guess is accepted when the reference Newton converges from it
// within 3 iterations without leaving the table, otherwise the Newton starts again from the
// warm guess.  FP32 density and pressure deviations, gammas, T and eint out; last stage the
// cell's CFL speed with the Alfven speed.  C2P_RESCUE: a cell whose warm start is poor stores
// eint, joins P.rescue_q and returns false with nothing else written (the rescue kernels finish
// it from the learned guess); the other cells run the warm-start Newton unchanged.
template <class C, int MODE>
__device__ __forceinline__ bool c2p_split_eos(const Prm &P, long long c, const C2pState &cs, float lT_mlp,
                                                  SplitStat &st) {
  constexpr bool LEARNED = MODE == C2P_LEARNED;
  constexpr int IP = C::IP, DIM = C::DIM;
  const Geo &g = P.g;
  const double rho = cs.rho, inv_rho = cs.inv_rho, eint = cs.eint, ye = cs.ye, inv_abar = cs.inv_abar;
  const long long bc = cs.bc;
  HelmCell hc;
  {
    double p, T, sound2;
    if (C::HELM) {
      int clamped = 0, it = 0;
      bool conv = false;
      if constexpr (LEARNED) {
        // judged guess: at most 3 reference Newton iterations from the learned guess (the
        // density part of the cell is already set)
        const bool have_guess = !isnan(lT_mlp);
        helm_cell_init_rho(P.helm, hc, rho, ye);
        if (have_guess) {
          T = fmin(fmax((double)exp10f(lT_mlp), P.helm.Tl * 1.000001), P.helm.Th * 0.999999);
          helm_cell_contract(P.helm, hc, helm_node_index(P.helm.T, P.helm.nT, P.helm.log10_T1, P.helm.dT, T));
          it = helm_rhoe_fast(P.helm, hc, inv_rho, eint * inv_rho, inv_abar, T, 3, clamped, conv);
        }
        if (have_guess && conv && clamped == 0) {
          st.mlp_acc += 1;
        } else {
          st.mlp_rej += 1;
          st.iters += it;
          clamped = 0;
          conv = false;
          T = cs.Tw;
          helm_cell_contract(P.helm, hc, helm_node_index(P.helm.T, P.helm.nT, P.helm.log10_T1, P.helm.dT, T));
          it = helm_rhoe_fast(P.helm, hc, inv_rho, eint * inv_rho, inv_abar, T, 100, clamped, conv);
        }
      } else if constexpr (MODE == C2P_RESCUE) {
        const double Tw = cs.Tw;
        T = Tw;
        helm_cell_init_rho(P.helm, hc, rho, ye);
        helm_cell_contract(P.helm, hc, helm_node_index(P.helm.T, P.helm.nT, P.helm.log10_T1, P.helm.dT, T));
        it = helm_rhoe_fast_from(P.helm, hc, inv_rho, eint * inv_rho, inv_abar, T, Tw, 1, clamped, conv);
        if (!conv && fabs(T - Tw) > RESCUE_STEP * Tw) {
          // poor warm start: the learned guess finishes this cell (its iteration is counted)
          st.iters += it;
          P.eint[c] = eint;
          const unsigned slot = atomicAdd(P.rescue_q, 1u);
          P.rescue_q[1 + slot] = (unsigned)c;
          return false;
        }
        if (!conv) it += helm_rhoe_fast_from(P.helm, hc, inv_rho, eint * inv_rho, inv_abar, T, Tw, 99, clamped, conv);
      } else {
        T = cs.Tw;
        helm_cell_init_rho(P.helm, hc, rho, ye);
        helm_cell_contract(P.helm, hc, helm_node_index(P.helm.T, P.helm.nT, P.helm.log10_T1, P.helm.dT, T));
        it = helm_rhoe_fast(P.helm, hc, inv_rho, eint * inv_rho, inv_abar, T, 100, clamped, conv);
      }
      st.calls += 1; st.iters += it; st.nonconv += !conv; st.clamp += clamped;
      helm_cell_p_sound2(P.helm, hc, rho, inv_rho, T, inv_abar, p, sound2);
      if (C::FAST) {
        // gamma_e goes to FP32 as a deviation from its equilibrium value, so it is formed in FP64;
        // gamma_c is stored as it is, to FP32 precision
        double ge = p / eint + 1.0;
        const float gc = (float)(sound2 * rho) / (float)p;
        if (C::WB) ge = ge - __ldg(P.eq_ge_cc + bc);
        P.gf_out[c] = (float)ge;
        P.gf_out[g.N + c] = gc;
      } else {
        P.gf_out[c] = (float)T;
      }
    } else {
      p = (g.gm - 1.0) * eint;
      T = p / (rho * CONST_RGAS * (1.0 / g.mu));
      sound2 = g.gm * p / rho;
    }
    double rdev = rho, pdev = p;
    if (C::WB) {
      rdev = rho - __ldg(P.eq_rho_cc + bc);
      pdev = p - __ldg(P.eq_p_cc + bc);
    }
    P.Wf_out[c] = (float)(rdev * P.inv_rho_ref);
    P.Wf_out[(long long)IP * g.N + c] = (float)(pdev * P.inv_p_ref);
    if (!(rho > 0.0) || !(p > 0.0) || !(T > 0.0) || !isfinite(eint)) st.bad += 1;
    // the next stage starts its Newton from T; nothing in a step reads eint back, nor T without one
    if (C::HELM || P.last_stage) P.temp[c] = T;
    if (P.last_stage) {
      P.eint[c] = eint;
      // |v| and b_cc^2 of the new state, read back (U and the face B are this cell's own)
      int i, j, k;
      unflatten3(c, g.div0[0], g.div1[0], i, j, k);
      double vabs[3] = {0.0, 0.0, 0.0}, ca2 = 0.0;
#pragma unroll
      for (int d = 0; d < DIM; ++d) {
        if (C::MHD) {
          const double b = 0.5 * (P.bf[d][face_lin(g, d, i + (d == 0), j + (d == 1), k + (d == 2))] +
                                  P.bf[d][face_lin(g, d, i, j, k)]);
          ca2 = d == 0 ? b * b : ca2 + b * b;
        }
        vabs[d] = fabs(P.U[(long long)(1 + d) * g.N + c] * inv_rho);
      }
      double csnd = sqrt(sound2 + ca2 * inv_rho);
      double sx1 = (vabs[0] + csnd) * g.inv_dx[0];
      double sx2 = (vabs[1] + csnd) * g.inv_dx[1];
      double sm = sx1 + sx2;
      if (DIM == 3) sm = (vabs[2] + csnd) * g.inv_dx[2] + sm;
      st.smax = fmax(st.smax, sm);
    }
  }
  return true;
}

template <class C, int MODE>
__global__ void __launch_bounds__(C2P_BLOCK, C::MINB_C2P32) k_c2p_split(Prm P) {
  if (!*P.active) return;
  SplitStat st;
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c < P.g.N) {
    C2pState cs;
    // the warm start first: its load then overlaps the combine instead of following its stores
    if (C::HELM) cs.Tw = P.temp[c];
    c2p_split_combine<C>(P, c, cs);
    c2p_split_eos<C, MODE>(P, c, cs, 0.0f, st);
  }
  split_stat_flush<C>(P, st);
}

// A whole hydro stage in one kernel, one thread per cell: every face is solved by both of its cells,
// nothing goes through memory but the state.  On small grids, whose kernels are all latency, one
// launch beats the face kernels and cons->prim (SplitRunnerT::face_fluxes has the line).  PPH at four
// blocks per SM (128 registers): a 40^3 box, one wave instead of one and an eighth of three blocks,
// 16.7 us a stage against 24.5.
template <class C>
__global__ void __launch_bounds__(C2P_BLOCK, C::REC == REC_PPH && !C::SF ? 4 : 0) k_stage_split(Prm P) {
  if (!*P.active) return;
  constexpr int NV = C::NV, DIM = C::DIM, SW = C::SW, NS = 2 * SW + 1;
  const Geo &g = P.g;
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  SplitStat st;
  if (c < g.N) {
    C2pState cs;
    if (C::HELM) cs.Tw = P.temp[c];
    int i, j, k;
    unflatten3(c, g.div0[0], g.div1[0], i, j, k);
    float res[NV];
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      // cells c-SW .. c+SW along d: the low face reads the first 2 SW, the high face the last
      float w[NS][NV], gmv[NS][2];
#pragma unroll
      for (int s = 0; s < NS; ++s)
        load_wf<C>(P, i + (d == 0 ? s - SW : 0), j + (d == 1 ? s - SW : 0), k + (d == 2 ? s - SW : 0), w[s], gmv[s]);
      const float none[3] = {0.0f, 0.0f, 0.0f};
      const float *const nb[6] = {none, none, none, none, none, none};
      float F[2][NV], Fb[3], rs;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        // cells m-3 .. m+2 of the face; the outer pair is read by LIM5TH only
        const float *wp[6], *gp[6];
#pragma unroll
        for (int s = 0; s < 6; ++s) {
          const int q = s + e + SW - 3;
          wp[s] = w[q < 0 ? 0 : (q < NS ? q : NS - 1)];
          gp[s] = gmv[q < 0 ? 0 : (q < NS ? q : NS - 1)];
        }
        face_flux_split_rec<C>(P, d, i + (e && d == 0), j + (e && d == 1), k + (e && d == 2), wp, gp, nb, F[e], Fb, rs);
      }
      const float inv_dl = (float)g.inv_dx[d];
#pragma unroll
      for (int iv = 0; iv < NV; ++iv) {
        const float dd = (F[1][iv] - F[0][iv]) * inv_dl;
        res[iv] = d == 0 ? dd : res[iv] + dd;
      }
    }
    c2p_split_combine<C>(P, c, cs, res);
    c2p_split_eos<C, C2P_WARM>(P, c, cs, 0.0f, st);
  }
  split_stat_flush<C>(P, st);
}

// the state of the combine for cell c, read back from U and eint
template <class C>
__device__ __forceinline__ void c2p_state_from_u(const Prm &P, long long c, C2pState &cs) {
  constexpr int IAS = C::IAS;
  const Geo &g = P.g;
  int i, j, k;
  unflatten3(c, g.div0[0], g.div1[0], i, j, k);
  cs.bc = bg_cc(g, i, j, k);
  cs.rho = P.U[c];
  cs.inv_rho = 1.0 / cs.rho;
  cs.eint = P.eint[c];
  if (C::HELM) cs.Tw = P.temp[c];
  cs.ye = P.U[(long long)IAS * g.N + c] * cs.inv_rho;
  cs.inv_abar = P.U[(long long)(IAS + 1) * g.N + c] * cs.inv_rho;
}

// the network's input features of a cell: log10 rho, log10 of the thermal energy (the cold
// energy E(rho, T_lo) from the density row of the table subtracted), Abar, Zbar, each scaled
template <class C>
__device__ __forceinline__ float4 c2p_features(const Prm &P, const C2pState &cs) {
  HelmCell hc;
  const double abar = 1.0 / cs.inv_abar, zbar = cs.ye * abar;
  helm_cell_init_rho(P.helm, hc, cs.rho, cs.ye);
  const double e_th = cs.eint * cs.inv_rho - helm_cell_cold_energy(P.helm, hc, cs.inv_rho, cs.inv_abar);
  float4 f;
  f.x = (log10f((float)cs.rho) - 3.5f) / 5.5f;
  f.y = (log10f((float)fmax(e_th, 1e-30)) - 19.5f) / 8.5f;
  f.z = (float)((abar - 28.5) / 27.5);
  f.w = (float)((zbar - 14.0) / 14.0);
  return f;
}

// Learned guess in the step, in three launches so that the cons->prim kernels keep their
// occupancy (a block-wide tensor-core product inside them would hold all their warps at its
// barriers): (1) the combine, storing eint and the network's features, (2) k_mlp_guess over
// all cells, (3) the EoS part from the stored state and guess.
template <class C>
__global__ void __launch_bounds__(128, C::MINB_C2P32) k_c2p_split_features(Prm P) {
  if (!*P.active) return;
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= P.g.N) return;
  C2pState cs;
  c2p_split_combine<C>(P, c, cs);
  P.eint[c] = cs.eint;
  reinterpret_cast<float4 *>(P.mlp_feat)[c] = c2p_features<C>(P, cs);
}

template <class C>
__global__ void __launch_bounds__(128, C::MINB_C2P32) k_c2p_split_guessed(Prm P) {
  if (!*P.active) return;
  SplitStat st;
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c < P.g.N) {
    // the state of the combine, read back: U and eint
    C2pState cs;
    c2p_state_from_u<C>(P, c, cs);
    st.gevals += 1;
    c2p_split_eos<C, C2P_LEARNED>(P, c, cs, P.mlp_out[c], st);
  }
  split_stat_flush<C>(P, st);
}

// network guesses for n samples (features [n][4] -> log10 T, NaN where the product stalled);
// the FP32 layers come in as a kernel argument (constant-bank operands)
static __global__ void __launch_bounds__(128) k_mlp_guess(const __grid_constant__ MlpSmall w,
                                                          const __nv_bfloat16 *w2bf, long long n, const float *feat,
                                                          float *out, const int *active, unsigned long long *stalled) {
  if (!*active) return;
  extern __shared__ __align__(128) unsigned char mlp_sm[];
  MlpUmmaSmem &S = *reinterpret_cast<MlpUmmaSmem *>(mlp_sm);
  mlp_cta_setup(w2bf, S);
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  float x[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  if (t < n) {
    const float4 f = reinterpret_cast<const float4 *>(feat)[t];
    x[0] = f.x; x[1] = f.y; x[2] = f.z; x[3] = f.w;
  }
  bool ok = true, have = false;
  const float y = mlp_forward_tile(w, x, S, 0u, ok, have, stalled);
  mlp_cta_teardown(S);
  if (t < n) out[t] = have ? y : __int_as_float(0x7fc00000);
}

// ---- learned rescue of poor warm starts (eos_guess = PHL_GUESS_MLP_RESCUE): one kernel on a
// fixed grid over the queue that k_c2p_split<C, C2P_RESCUE> fills.  Tiles of 128 queue
// slots, strided over the blocks: each thread reads its cell's state back (U, eint) and forms
// the network's features, the block runs one tensor-core product for the tile, and each thread
// finishes its cell from the judged guess.  With an empty queue every block reads the count and
// returns; a block without a tile returns before it claims tensor memory.
template <class C>
__global__ void __launch_bounds__(128) k_c2p_rescue(Prm P, const __grid_constant__ MlpSmall w) {
  if (!*P.active) return;
  const long long n = P.rescue_q[0];
  if ((long long)blockIdx.x * blockDim.x >= n) return;
  extern __shared__ __align__(128) unsigned char mlp_sm[];
  MlpUmmaSmem &S = *reinterpret_cast<MlpUmmaSmem *>(mlp_sm);
  mlp_cta_setup(P.mlp_w2bf, S);
  SplitStat st;
  bool ok = true;
  uint32_t parity = 0;
  for (long long t0 = (long long)blockIdx.x * blockDim.x; t0 < n; t0 += (long long)gridDim.x * blockDim.x) {
    const long long q = t0 + threadIdx.x;
    C2pState cs;
    long long c = -1;
    float x[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (q < n) {
      c = P.rescue_q[1 + q];
      c2p_state_from_u<C>(P, c, cs);
      const float4 f = c2p_features<C>(P, cs);
      x[0] = f.x; x[1] = f.y; x[2] = f.z; x[3] = f.w;
    }
    bool have = false;
    const float y = mlp_forward_tile(w, x, S, parity, ok, have, P.stat + STAT_TC_STALLED);
    parity ^= 1u;
    if (c >= 0) {
      st.gevals += 1;
      c2p_split_eos<C, C2P_LEARNED>(P, c, cs, have ? y : __int_as_float(0x7fc00000), st);
    }
  }
  mlp_cta_teardown(S);
  split_stat_flush<C>(P, st);
}

// FP64 primitives (+eint, gammaf) -> U (FP64) and FP32 deviations (prim->cons of
// source.F90:7057-7117)
template <class C>
__global__ void k_split_from_prim(Prm P) {
  constexpr int NV = C::NV, IP = C::IP, IAS = C::IAS, DIM = C::DIM;
  const Geo &g = P.g;
  long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= g.N) return;
  int i, j, k;
  unflatten3(c, g.div0[0], g.div1[0], i, j, k);
  const long long bc = bg_cc(g, i, j, k);
  double w[NV];
#pragma unroll
  for (int iv = 0; iv < NV; ++iv) w[iv] = P.Win[(long long)iv * g.N + c];
  double rho = w[0], vx1 = w[1], vx2 = w[2], vx3 = DIM == 3 ? w[3] : 0.0;
  double u[NV];
  u[0] = rho; u[1] = rho * vx1; u[2] = rho * vx2; if (DIM == 3) u[3] = rho * vx3;
  double rhoe = P.eint[c] + 0.5 * rho * (vx1 * vx1 + vx2 * vx2 + vx3 * vx3);
  if (C::MHD) {
    double b0 = P.bcc_in[c], b1 = P.bcc_in[g.N + c], b2 = DIM == 3 ? P.bcc_in[2 * g.N + c] : 0.0;
    rhoe = rhoe + 0.5 * (b0 * b0 + b1 * b1 + b2 * b2);
    P.bccf[c] = (float)(b0 * P.inv_b_ref);
    P.bccf[g.N + c] = (float)(b1 * P.inv_b_ref);
    if (DIM == 3) P.bccf[2 * g.N + c] = (float)(b2 * P.inv_b_ref);
  }
  if (C::ETOT) rhoe = rhoe + rho * __ldg(P.phi_cc + bc);
  u[IP] = rhoe;
#pragma unroll
  for (int iv = IAS; iv < NV; ++iv) u[iv] = rho * w[iv];
#pragma unroll
  for (int iv = 0; iv < NV; ++iv) P.U[(long long)iv * g.N + c] = u[iv];
  double rdev = rho, pdev = w[IP];
  if (C::WB) {
    rdev = rho - __ldg(P.eq_rho_cc + bc);
    pdev = w[IP] - __ldg(P.eq_p_cc + bc);
  }
  P.Wf_out[c] = (float)(rdev / P.rho_ref);
#pragma unroll
  for (int d = 0; d < DIM; ++d) P.Wf_out[(long long)(1 + d) * g.N + c] = (float)(w[1 + d] / P.v_ref);
  if (C::MHD) {
    const float vf[3] = {(float)(w[1] / P.v_ref), (float)(w[2] / P.v_ref), DIM == 3 ? (float)(w[3] / P.v_ref) : 0.0f};
    const float bf3[3] = {P.bccf[c], P.bccf[g.N + c], DIM == 3 ? P.bccf[2 * g.N + c] : 0.0f};
    store_cell_emf<C>(P, c, vf, bf3);
  }
  P.Wf_out[(long long)IP * g.N + c] = (float)(pdev / P.p_ref);
#pragma unroll
  for (int iv = IAS; iv < NV; ++iv) P.Wf_out[(long long)iv * g.N + c] = (float)w[iv];
  if (C::FAST) {
    double ge = P.gin[c];
    if (C::WB) ge = ge - __ldg(P.eq_ge_cc + bc);
    P.gf_out[c] = (float)ge;
    P.gf_out[g.N + c] = (float)P.gin[g.N + c];
  } else if (C::HELM) {
    P.gf_out[c] = (float)P.temp[c];
  }
}

// U (FP64) + temp -> FP64 primitives and gammaf (for download and the standalone dt)
template <class C>
__global__ void k_split_to_prim(Prm P) {
  constexpr int NV = C::NV, IP = C::IP, IAS = C::IAS, DIM = C::DIM;
  const Geo &g = P.g;
  long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= g.N) return;
  int i, j, k;
  unflatten3(c, g.div0[0], g.div1[0], i, j, k);
  const long long bc = bg_cc(g, i, j, k);
  double u[NV];
#pragma unroll
  for (int iv = 0; iv < NV; ++iv) u[iv] = P.U[(long long)iv * g.N + c];
  double rho = u[0], inv_rho = 1.0 / rho;
  double eint = P.eint[c];
  double p;
  if (C::HELM) {
    // pressure and sound speed at the state's temperature from the contracted table cell (the
    // evaluation of the split form's cons->prim, equal to given_full to rounding)
    const double inv_abar = u[IAS + 1] * inv_rho, ye = u[IAS] * inv_rho, T = P.temp[c];
    HelmCell hc;
    helm_cell_init_rho(P.helm, hc, rho, ye);
    helm_cell_contract(P.helm, hc, helm_node_index(P.helm.T, P.helm.nT, P.helm.log10_T1, P.helm.dT, T));
    double s2;
    helm_cell_p_sound2(P.helm, hc, rho, inv_rho, T, inv_abar, p, s2);
    if (C::FAST) {
      P.gout[c] = p / eint + 1.0;
      P.gout[g.N + c] = s2 * rho / p;
    } else {
      P.gout[c] = P.temp[c];
    }
  } else {
    p = (g.gm - 1.0) * eint;
  }
  if (C::MHD) {
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      int ui = i + (d == 0), uj = j + (d == 1), uk = k + (d == 2);
      P.bcc_out[(long long)d * g.N + c] = 0.5 * (P.bf[d][face_lin(g, d, ui, uj, uk)] + P.bf[d][face_lin(g, d, i, j, k)]);
    }
  }
  P.Wout[c] = rho;
#pragma unroll
  for (int d = 0; d < DIM; ++d) P.Wout[(long long)(1 + d) * g.N + c] = u[1 + d] * inv_rho;
  P.Wout[(long long)IP * g.N + c] = p;
#pragma unroll
  for (int iv = IAS; iv < NV; ++iv) P.Wout[(long long)iv * g.N + c] = u[iv] * inv_rho;
  (void)bc;
}

namespace {
inline unsigned nblk(long long n, int t) { return (unsigned)((n + t - 1) / t); }

}

template <class C>
struct SplitRunnerT : Runner {
  // PHL_FACE_KERNEL=walk runs the walking kernel along x1 as well (comparison)
  const bool walk_x1 = [] {
    const char *e = getenv("PHL_FACE_KERNEL");
    return e && strcmp(e, "walk") == 0;
  }();
  // A hydro stage in one per-cell kernel on grids of up to ONE_KERNEL_WAVES waves of its blocks; with
  // more cells the face kernels, which solve each face once, pay for their launches.  A wave is 38,000
  // cells (without USE_FASTEOS, 254 registers) to 152,000 (2D ideal gas, 64).  Three waves, but one where a
  // cell's edges cost more than its solver (LIM5TH, and PPH with its flattened edges), since a cell's are
  // formed four times here and twice there.  us per stage, one kernel / face kernels, the last size
  // below and the first above the line (a few percent between the two forms on either side of it):
  //   3D Helmholtz FASTEOS LHLLC 60^3 42.5 / 43.1, 62^3 49.6 / 46.1; HLLC 60^3 43.1 / 43.4, 62^3 51.5 / 46.3
  //   without FASTEOS LHLLC      48^3 155 / 170,   50^3 193 / 179
  //   PPH                        60^3 40.9 / 41.9, 62^3 48.6 / 45.2
  //   LIM5TH                     38^3 22.1 / 25.8, 40^3 39.8 / 28.2
  //   PLM flattened              52^3 46.0 / 46.0, 56^3 55.6 / 49.5; PPH flattened 38^3 28.4 / 31.6, 40^3 41.0 / 32.4
  //   3D ideal gas LHLLC         70^3 33.0 / 33.9, 74^3 38.7 / 35.3
  //   2D ideal gas LHLLC         640^2 23.2 / 22.6; bubble 624^2 24.8 / 24.1, 640^2 26.0 / 24.9
  //   2D Helmholtz               528^2 36.6 / 36.7, 544^2 41.3 / 38.9; 2D flattened 576^2 32.1 / 32.2, 600^2 34.5 / 33.4
  // PHL_STAGE_KERNEL=cell / =faces select one of the forms on any grid (comparisons).
  static constexpr int ONE_KERNEL_WAVES = C::REC == REC_LIM2ND || (C::REC == REC_PPH && !C::SF) ? 3 : 1;
  static long long one_kernel_cells() {
    int dev = 0, sms = 0, blocks = 0;
    if constexpr (!C::MHD) {
      if (cudaGetDevice(&dev) != cudaSuccess ||
          cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
          cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, (const void *)k_stage_split<C>, C2P_BLOCK, 0) !=
              cudaSuccess)
        return 0;
    }
    return (long long)ONE_KERNEL_WAVES * blocks * sms * C2P_BLOCK;
  }
  const int stage_kind = [] {
    const char *e = getenv("PHL_STAGE_KERNEL");
    return e && strcmp(e, "cell") == 0 ? 1 : (e && strcmp(e, "faces") == 0 ? 2 : 0);
  }();
  bool face_fluxes(const Geo &g) const override {
    if (C::MHD) return true;
    if (stage_kind) return stage_kind == 2;
    return g.N > one_kernel_cells();
  }
  void stage(const Prm &P, cudaStream_t s) override {
    if constexpr (C::SF) {
      k_sf_mark_split<C><<<nblk(sf_mark_cells<C>(P.g), 256), 256, 0, s>>>(P);
      k_sf_flag<C><<<nblk(sf_flag_cells<C>(P.g), 256), 256, 0, s>>>(P);
    }
    if (!C::MHD && !P.fflux[0]) {  // small grid, or no room for the face fluxes
      if constexpr (!C::MHD) k_stage_split<C><<<nblk(P.g.N, C2P_BLOCK), C2P_BLOCK, 0, s>>>(P);
    } else {
      const Geo &g = P.g;
      auto nfc = [&](int d) {
        return (long long)(g.nx[0] + (d == 0)) * (g.nx[1] + (d == 1)) * (g.nx[2] + (d == 2));
      };
      if constexpr (C::REC == REC_LIM2ND) {
        // threads of the walking kernels: faces along D in chunks of K, times the other extents
        auto nwalk = [&](int d, int k) {
          long long n = (g.nx[d] + 1 + k - 1) / k;
          for (int a = 0; a < C::DIM; ++a)
            if (a != d) n *= g.nx[a];
          return n;
        };
        // without USE_FASTEOS a face is two FP64 (rho, P) -> T solves, and the row kernel's three idle
        // lanes in 32 cost more than its loads save (96^3 MHD step 2.50 ms against 2.28)
        if (walk_x1 || C::EOSM == EOS_GIVEN) {
          k_face_split_walk<C, 0, WALK_K0><<<nblk(nwalk(0, WALK_K0), 128), 128, 0, s>>>(P);
        } else if constexpr (C::EOSM != EOS_GIVEN) {
          const unsigned chunks = nblk(g.nx[0] + 1, ROW_FACES);
          k_face_split_row<C><<<nblk((long long)chunks * g.nx[1] * g.nx[2], 4), 128, 0, s>>>(P, FastDiv::by(chunks));
        }
        k_face_split_walk<C, 1, WALK_K><<<nblk(nwalk(1, WALK_K), 128), 128, 0, s>>>(P);
        if constexpr (C::DIM == 3)
          k_face_split_walk<C, 2, WALK_K><<<nblk(nwalk(2, WALK_K), 128), 128, 0, s>>>(P);
      } else {
        k_face_split<C, 0><<<nblk(nfc(0), 128), 128, 0, s>>>(P);
        k_face_split<C, 1><<<nblk(nfc(1), 128), 128, 0, s>>>(P);
        if constexpr (C::DIM == 3) k_face_split<C, 2><<<nblk(nfc(2), 128), 128, 0, s>>>(P);
      }
      if constexpr (C::MHD) {
        corners(P, s);
        const long long nodes = (long long)(g.nx[0] + 1) * (g.nx[1] + 1) * (C::DIM == 3 ? g.nx[2] + 1 : 1);
        k_bface_split<C><<<nblk(nodes, 256), 256, 0, s>>>(P);
      }
      if constexpr (C::HELM && C::MHD) {
        if (P.mlp_w && P.mlp_small && P.rescue_q) {
          // warm start everywhere; cells with a poor warm start through the learned guess
          cudaMemsetAsync(P.rescue_q, 0, sizeof(unsigned), s);
          k_c2p_split<C, C2P_RESCUE><<<nblk(g.N, C2P_BLOCK), C2P_BLOCK, 0, s>>>(P);
          k_c2p_rescue<C><<<RESCUE_BLOCKS, 128, sizeof(MlpUmmaSmem), s>>>(P, *P.mlp_small);
          return;
        }
        if (P.mlp_w && P.mlp_small && P.mlp_feat && P.mlp_out) {
          k_c2p_split_features<C><<<nblk(g.N, 128), 128, 0, s>>>(P);
          k_mlp_guess<<<nblk(g.N, 128), 128, sizeof(MlpUmmaSmem), s>>>(*P.mlp_small, P.mlp_w2bf, g.N, P.mlp_feat,
                                                                       P.mlp_out, P.active, P.stat + STAT_TC_STALLED);
          k_c2p_split_guessed<C><<<nblk(g.N, 128), 128, 0, s>>>(P);
          return;
        }
      }
      k_c2p_split<C, C2P_WARM><<<nblk(g.N, C2P_BLOCK), C2P_BLOCK, 0, s>>>(P);
    }
  }
  // corner EMFs: the interior nodes' blocks, then those of the nodes on the domain's faces
  void corners(const Prm &P, cudaStream_t s) {
    const Geo &g = P.g;
    const long long n0 = g.nx[0], n1 = g.nx[1], n2 = g.nx[2];
    const long long nin = (n0 - 1) * (n1 - 1) * (C::DIM == 3 ? n2 - 1 : 1);
    const long long nrim = 2 * (n0 + n1) * (C::DIM == 3 ? n2 - 1 : 1) + (C::DIM == 3 ? 2 * (n0 + 1) * (n1 + 1) : 0);
    const unsigned bin = nblk(nin, 256);
    k_corner_split<C><<<bin + nblk(nrim, 256), 256, 0, s>>>(P, bin, FastDiv::by((unsigned)n0 - 1),
                                                            FastDiv::by((unsigned)n1 - 1));
  }
  void split_from_prim(const Prm &P, cudaStream_t s) override {
    k_split_from_prim<C><<<nblk(P.g.N, 256), 256, 0, s>>>(P);
  }
  void split_to_prim(const Prm &P, cudaStream_t s) override {
    k_split_to_prim<C><<<nblk(P.g.N, 256), 256, 0, s>>>(P);
  }
};

#define PHL_SPLIT_LIST(X)                                   \
  X(2, 4, true, false, false, R_HLLD, false, REC_LIM2ND, false) \
  X(2, 4, true, false, false, R_LHLLD, false, REC_LIM2ND, false) \
  X(3, 5, true, false, false, R_HLLD, false, REC_LIM2ND, false) \
  X(3, 5, true, false, false, R_LHLLD, false, REC_LIM2ND, false) \
  X(3, 7, true, true, true, R_LHLLD, true, REC_LIM2ND, false) \
  X(3, 7, true, true, true, R_HLLD, true, REC_LIM2ND, false) \
  X(3, 7, true, true, true, R_LHLLD, false, REC_LIM2ND, false) \
  X(2, 4, false, false, false, R_LHLLC, false, REC_LIM2ND, false) \
  X(2, 4, false, false, false, R_HLLC, false, REC_LIM2ND, false) \
  X(2, 4, false, false, true, R_LHLLC, false, REC_LIM2ND, false) \
  X(2, 6, false, true, true, R_LHLLC, true, REC_LIM2ND, false) \
  X(3, 5, false, false, false, R_LHLLC, false, REC_LIM2ND, false) \
  X(3, 5, false, false, false, R_HLLC, false, REC_LIM2ND, false) \
  X(3, 7, false, true, true, R_LHLLC, true, REC_LIM2ND, false) \
  X(3, 7, false, true, true, R_HLLC, true, REC_LIM2ND, false) \
  X(3, 7, false, true, true, R_LHLLC, false, REC_LIM2ND, false) \
  X(3, 7, false, true, true, R_HLLC, false, REC_LIM2ND, false) \
  X(2, 4, true, false, false, R_HLLD, false, REC_LIM5TH, false) \
  X(3, 7, true, true, true, R_LHLLD, true, REC_PPH, false) \
  X(3, 7, true, true, true, R_LHLLD, true, REC_LIM5TH, false) \
  X(3, 7, false, true, true, R_LHLLC, true, REC_PPH, false) \
  X(3, 7, false, true, true, R_LHLLC, true, REC_LIM5TH, false) \
  X(2, 5, false, false, false, R_HLLC, false, REC_LIM2ND, true) \
  X(2, 4, true, false, false, R_HLLD, false, REC_LIM2ND, true) \
  X(3, 7, false, true, true, R_LHLLC, true, REC_LIM2ND, true) \
  X(3, 7, false, true, true, R_LHLLC, true, REC_PPH, true) \
  X(3, 7, true, true, true, R_LHLLD, true, REC_LIM2ND, true)

Runner *make_split_runner(int dim, int nv, bool mhd, bool helm, bool strat, int riem, bool fast, int rec, bool sf) {
#define X(D, N, M, H, S, R, F, REC, SF)                                                                      \
  if (dim == D && nv == N && mhd == M && helm == H && strat == S && riem == R && (!H || fast == F) &&         \
      rec == REC && sf == SF)                                                                                 \
    return new SplitRunnerT<Cfg<D, N, M, H, S, S, S, R, F, REC, SF>>();
  PHL_SPLIT_LIST(X)
#undef X
  return nullptr;
}

}  // namespace phl
