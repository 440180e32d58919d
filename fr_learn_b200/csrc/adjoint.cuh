// adjoint.cuh -- discrete adjoint (vector-Jacobian products) of one FR
// residual evaluation, and its fusion into the reverse sweep of the explicit
// RK update.  FP64 throughout.  There is no adjoint in the reference; these
// kernels transpose, operation by operation, the forward residual that the
// stage kernels compute (calcResidual, src/solver.cpp:252-291):
//
//   traces   U_f   = sum_j lag[side][j] U[line pt j]              (extrapolateU)
//   fluxes   Fs_d1 = sum_d2 JGinv[d1][d2] F_d2(U)                 (calcInviscidFlux_spts)
//   normal   dis   = +-sum_j lag[side][j] Fs_dir[line pt j]       (extrapolateNormalFlux)
//   common   Fn    = Riemann(U_L, U_R, n); jump J = +-Fn dA - dis (face::calcInviscidFlux)
//   residual divF  = sum_d sum_q dlag[i_d][q] Fs_d[line pt q] + sum_c g_c J[f_c]
//                                                                 (calcDivF_spts, correctDivFlux)
//
// Given gbar = dJ/d(divF) at the solution points, the transposed chain is
//   Jbar[f]      = sum_j g(side, j) gbar[line pt j]               (correction^T)
//   fbar[f]      = +-dA Jbar[f] from this element's copy of the common flux
//                  plus the neighbour's copy (both elements evaluate the same
//                  face flux), gathered from the face-seed pass
//   Ubar_f       = (dFn/dU_own)^T fbar   (reverse-mode products; on boundaries
//                  the ghost state is differentiated with the interior state,
//                  and the freestream parameter's component gives dJ/dtheta)
//   Fsbar_d[s]   = sum_i dlag[i][c_d(s)] gbar[line pt i] - sum_f (+-) lag Jbar[f]
//   Ubar[s]      = sum_d (dF_d/dU)^T (sum_d1 JGinv[d1][d] Fsbar_d1) + sum_f lag Ubar_f
//
// One launch per reversed stage: fr_adj_stage_kernel, in the form of the line
// kernels (kernels_line.cuh).  It reads the traces of its stage state and every
// side's share of the common-flux adjoint, both left by the launch before, and
// leaves them for the stage reversed next; fr_adj_face_kernel makes them for the
// first stage of a sweep segment and for a single product.
#pragma once
#include "dual.cuh"
#include "kernels.cuh"
#include "kernels_line.cuh"

namespace frg {

// Scratch of the viscous adjoint (adjoint_visc.cuh), FP64 [..][point][element].
struct AdjViscBufs {
  double *g;      // forward corrected gradient at the solution points [DIM][NV][NS][L]
  double *fvn;    // each side's projected viscous flux [NV][NF][L] (interior flux points)
  double *fvn2;   // 3D LDG penalty: the left side's projection [NV][NF][L]
  double *ub;     // state adjoint at the solution points [NV][NS][L]
  double *ufb;    // trace adjoint at the flux points [NV][NF][L]
  double *dcb;    // adjoint of the LDG correction Dc = Uc - U_f [NV][NF][L]
  int visc2;
};

struct AdjArgs {
  int nE, nEle;           // element stride (padded) and real element count
  const double *Y;        // stage state [NV][NS][nE]
  const double *gbar;     // seed dJ/d(divF) [NV][NS][nE]
  double *trY;            // traces of Y [NV][NF][nE] (face kernel out)
  double *fnbar;          // this element's common-flux adjoint [NV][NF][nE] (face kernel out)
  const int *nbr;         // [NF][nE]
  const double *nrm, *dA, *JG, *detJ, *invDet;
  int vcjh;
  unsigned *err;
  // outputs of the element kernel
  const double *Ynext;    // state of the stage reversed next, or null: its traces and flux-adjoint shares
  double *trNext, *fnNext;  // go here
  double *ybar;           // (ADJ_PLAIN) Ybar = (d divF / dY)^T gbar
  const double *lam;      // (RK) adjoint of the step's final state
  double *lamNew;         // (RK) adjoint of the step's initial state, accumulated
  double *seedOut;        // (RK) seed of the stage before
  double cLam, cY;        // seedOut = -(cLam * base + cY * ybar) * dt / detJ
  double dt;
  int mode;               // ADJ_* flags
  int pdl;                // launch as a programmatic dependent of the launch before (host side)
  const double *thetaDir; // d(rhoB, vB[0..2], pB) / d(theta) of the boundary state (device, 5)
  const int *grp;         // ensemble mode: group of each element, else null
  const double *dtGrp;    // ensemble mode: fixed dt per group (replaces dt)
  double *thetaBar;       // += fbar . dFn/dtheta over boundary flux points
  AdjViscBufs v;          // viscous runs only
  Phys ph;
  // (the 1D operators of the inviscid stage kernel are a parameter of its own: the
  // viscous kernels keep a copy of this block on each thread's stack, and 560 bytes
  // more of it took their element pass of 150x149 quads, P = 1, from 844 to 928 us)
};
static_assert(sizeof(AdjArgs) <= 464, "copied to each thread's stack by the viscous kernels");

enum : int {
  ADJ_PLAIN = 1,      // write ybar only
  ADJ_RK_FIRST = 2,   // the last RK stage, the first reversed: lamNew = lam + ybar
  ADJ_RK_LAST = 4,    // RK stage 0, the last reversed: seedOut from the finished lamNew
  ADJ_RK = 8          // fused reverse-RK outputs
};

template <class C, typename T>
__device__ __forceinline__ void adj_common(const T *UL, const T *UR, const T *n, int code, T *Fn, const Phys &ph,
                                           int rs) {
  constexpr int NV = C::NV, DIM = C::DIM;
  if constexpr (NV == 1) {
    lax_friedrichs<DIM, T>(UL[0], UR[0], n, Fn, ph);
  } else if constexpr (DIM == 3) {
    rusanov<DIM, NV, T, T>(UL, UR, n, Fn, ph);
  } else {
    // boundary faces always use Rusanov (src/face.cpp:142-145)
    if (rs == 0 || code < 0) rusanov<DIM, NV, T, T>(UL, UR, n, Fn, ph);
    else roe2d<T, T>(UL, UR, n, Fn, ph);
  }
}

// Face-seed pass: one thread per (flux point, element).
template <class C>
__global__ void __launch_bounds__(256) fr_adj_face_kernel(const AdjArgs a) {
  constexpr int NV = C::NV, NF = C::NF, NS = C::NS, N1 = C::N1;
  const OpTab<double> &op = optab<double>(a.vcjh, C::P);
  const long n = (long)NF * a.nE;
  for (long it = blockIdx.x * (long)blockDim.x + threadIdx.x; it < n; it += (long)gridDim.x * blockDim.x) {
    const int f = (int)(it / a.nE), eg = (int)(it - (long)f * a.nE);
    if (eg >= a.nEle) continue;
    int dir, side, s0, st;
    fpt_line<C>(f, dir, side, s0, st);
    const int code = a.nbr[(size_t)f * a.nE + eg];
    const bool right = code >= 0 && (code & 1);
    const double dA = a.dA[(size_t)f * a.nE + eg];
#pragma unroll
    for (int v = 0; v < NV; v++) {
      double t = 0, jb = 0;
#pragma unroll
      for (int j = 0; j < N1; j++) {
        const size_t gi = ((size_t)v * NS + s0 + j * st) * a.nE + eg;
        t += op.lag[side][j] * a.Y[gi];
        jb += (side ? op.gR[j] : -op.gL[j]) * a.gbar[gi];
      }
      a.trY[((size_t)v * NF + f) * a.nE + eg] = t;
      a.fnbar[((size_t)v * NF + f) * a.nE + eg] = (right ? -dA : dA) * jb;
    }
  }
}

// ---- reverse-mode products of the pointwise fluxes, written out

// b^T dF_n/dU, added to ub: the Euler flux along n (any vector; the unit vectors
// give the coordinate fluxes).
template <int DIM>
__device__ __forceinline__ void vjp_normal_flux(const double *U, const double *n, const double *b, double g1,
                                                double *ub) {
  const double ir = 1.0 / U[0];
  double u[DIM], vn = 0, uu = 0, bu = 0, bn = 0;
#pragma unroll
  for (int d = 0; d < DIM; d++) {
    u[d] = U[d + 1] * ir;
    vn += u[d] * n[d];
    uu += u[d] * u[d];
    bu += b[d + 1] * u[d];
    bn += b[d + 1] * n[d];
  }
  const double p = g1 * (U[DIM + 1] - 0.5 * U[0] * uu), H = (U[DIM + 1] + p) * ir, bE = b[DIM + 1];
  const double S = b[0] + bu + bE * H, Q = (bn + bE * vn) * g1;
  ub[0] += Q * 0.5 * uu - vn * (bu + bE * H);
#pragma unroll
  for (int d = 0; d < DIM; d++) ub[d + 1] += S * n[d] + vn * b[d + 1] - Q * u[d];
  ub[DIM + 1] += bE * vn + Q;
}

// Adjoints of one side's derived values -- velocity vb, enthalpy hb, normal
// velocity vnb, sound speed cb, pressure p0b -- to its conservative ones, added
// to ub.
template <int DIM>
__device__ __forceinline__ void vjp_side(const double *u, const double *n, double ir, double vn, double p, double h,
                                         double c, double g1, const double *vb, double hb, double vnb, double cb,
                                         double *ub, double p0b = 0.0) {
  double vu = 0, uu = 0;
#pragma unroll
  for (int d = 0; d < DIM; d++) {
    vu += vb[d] * u[d];
    uu += u[d] * u[d];
  }
  const double pb = p0b + hb * ir + 0.5 * cb * c / p;
  ub[0] += pb * g1 * 0.5 * uu - ir * (vu + vnb * vn + hb * h + 0.5 * cb * c);
#pragma unroll
  for (int d = 0; d < DIM; d++) ub[d + 1] += ir * (vb[d] + vnb * n[d]) - pb * g1 * u[d];
  ub[DIM + 1] += hb * ir + pb * g1;
}

// Rusanov (rusanov_normal): fb^T dFn/dUL and fb^T dFn/dUR.
template <int DIM>
__device__ __forceinline__ void vjp_rusanov(const double *UL, const double *UR, const double *n, const double *fb,
                                            double gamma, double *ubL, double *ubR) {
  constexpr int NV = DIM + 2;
  const double g1 = gamma - 1.0;
  double hb[NV], jump = 0, vn[2], eig[2], c[2], ir[2], p[2], u[2][DIM];
#pragma unroll
  for (int v = 0; v < NV; v++) {
    hb[v] = 0.5 * fb[v];
    jump += hb[v] * (UR[v] - UL[v]);
  }
#pragma unroll
  for (int s = 0; s < 2; s++) {
    const double *U = s ? UR : UL;
    ir[s] = 1.0 / U[0];
    double uu = 0;
    vn[s] = 0;
#pragma unroll
    for (int d = 0; d < DIM; d++) {
      u[s][d] = U[d + 1] * ir[s];
      uu += u[s][d] * u[s][d];
      vn[s] += n[d] * u[s][d];
    }
    p[s] = g1 * (U[DIM + 1] - 0.5 * U[0] * uu);
    c[s] = sqrt(fmax(gamma * p[s] * ir[s], 0.0));
    eig[s] = fabs(vn[s]) + c[s];
  }
  const bool left = eig[0] > eig[1];
  const double e = left ? eig[0] : eig[1];
#pragma unroll
  for (int v = 0; v < NV; v++) {
    ubL[v] = e * hb[v];
    ubR[v] = -e * hb[v];
  }
  vjp_normal_flux<DIM>(UL, n, hb, g1, ubL);
  vjp_normal_flux<DIM>(UR, n, hb, g1, ubR);
  const double zero[DIM] = {};
  if (left) vjp_side<DIM>(u[0], n, ir[0], vn[0], p[0], 0.0, c[0], g1, zero, 0.0, vn[0] < 0 ? jump : -jump, -jump, ubL);
  else vjp_side<DIM>(u[1], n, ir[1], vn[1], p[1], 0.0, c[1], g1, zero, 0.0, vn[1] < 0 ? jump : -jump, -jump, ubR);
}

// Roe with the entropy fix (roe2d, whose names these are; xb: adjoint of x):
// fb^T dFn/dUL and fb^T dFn/dUR.
__device__ __forceinline__ void vjp_roe2d(const double *UL, const double *UR, const double *n, const double *fb,
                                          double gamma, double *ubL, double *ubR) {
  const double g1 = gamma - 1.0;
  double v[2][2], ir[2], p[2], h[2], vn[2], c[2], du[4], db[4], hb[4];
#pragma unroll
  for (int s = 0; s < 2; s++) {
    const double *U = s ? UR : UL;
    ir[s] = 1.0 / U[0];
    v[s][0] = U[1] * ir[s];
    v[s][1] = U[2] * ir[s];
    p[s] = g1 * (U[3] - 0.5 * U[0] * (v[s][0] * v[s][0] + v[s][1] * v[s][1]));
    h[s] = (U[3] + p[s]) * ir[s];
    vn[s] = v[s][0] * n[0] + v[s][1] * n[1];
    c[s] = sqrt(gamma * p[s] * ir[s]);
  }
  const double sq = sqrt(UR[0] * ir[0]), rr = 1.0 / (sq + 1.0);
  const double um[2] = {rr * (v[0][0] + sq * v[1][0]), rr * (v[0][1] + sq * v[1][1])};
  const double usq = 0.5 * (um[0] * um[0] + um[1] * um[1]), unm = um[0] * n[0] + um[1] * n[1];
  const double hm = rr * (h[0] + sq * h[1]), am = sqrt(g1 * (hm - usq)), iam = 1.0 / am;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    du[i] = UR[i] - UL[i];
    hb[i] = 0.5 * fb[i];
    db[i] = -hb[i];
  }
  const double l[3] = {fabs(unm), fabs(unm + am), fabs(unm - am)};
  const double dvn = vn[0] - vn[1], dc = c[0] - c[1], eps = 0.5 * (fabs(dvn) + fabs(dc)), qe = 0.25 / eps;
  double lam[3];
#pragma unroll
  for (int i = 0; i < 3; i++) lam[i] = l[i] < 2.0 * eps ? qe * l[i] * l[i] + eps : l[i];
  const double a2 = 0.5 * (lam[1] + lam[2]) - lam[0], a3 = 0.5 * (lam[1] - lam[2]) * iam;
  const double a1 = a2 * g1 * iam * iam, a4 = a3 * g1;
  const double a5 = usq * du[0] - um[0] * du[1] - um[1] * du[2] + du[3], a6 = unm * du[0] - n[0] * du[1] - n[1] * du[2];
  const double aL1 = a1 * a5 - a3 * a6, bL1 = a4 * a5 - a2 * a6;
  // reverse
  double lamb[3], dub[4];
  lamb[0] = db[0] * du[0] + db[1] * du[1] + db[2] * du[2] + db[3] * du[3];
  const double aL1b = db[0] + db[1] * um[0] + db[2] * um[1] + db[3] * hm;
  const double bL1b = db[1] * n[0] + db[2] * n[1] + db[3] * unm;
  const double a5b = aL1b * a1 + bL1b * a4, a6b = -aL1b * a3 - bL1b * a2;
  const double a1b = aL1b * a5, a2b = a1b * g1 * iam * iam - bL1b * a6, a3b = bL1b * a5 * g1 - aL1b * a6;
  double umb[2] = {aL1 * db[1] - a5b * du[1], aL1 * db[2] - a5b * du[2]};
  double hmb = aL1 * db[3], unmb = bL1 * db[3] + a6b * du[0];
  double usqb = a5b * du[0], iamb = 2.0 * a1b * a2 * g1 * iam + 0.5 * a3b * (lam[1] - lam[2]);
  dub[0] = lam[0] * db[0] + a5b * usq + a6b * unm;
  dub[1] = lam[0] * db[1] - a5b * um[0] - a6b * n[0];
  dub[2] = lam[0] * db[2] - a5b * um[1] - a6b * n[1];
  dub[3] = lam[0] * db[3] + a5b;
  lamb[1] = 0.5 * a3b * iam + 0.5 * a2b;
  lamb[2] = -0.5 * a3b * iam + 0.5 * a2b;
  lamb[0] -= a2b;
  double epsb = 0;
#pragma unroll
  for (int i = 0; i < 3; i++)
    if (l[i] < 2.0 * eps) {
      epsb += lamb[i] * (1.0 - qe * l[i] * l[i] / eps);
      lamb[i] *= 2.0 * qe * l[i];
    }
  const double s0 = unm < 0 ? -lamb[0] : lamb[0], s1 = unm + am < 0 ? -lamb[1] : lamb[1];
  const double s2 = unm - am < 0 ? -lamb[2] : lamb[2];
  unmb += s0 + s1 + s2;
  const double am2b = 0.5 * iam * (s1 - s2 - iamb * iam * iam) * g1;
  hmb += am2b;
  usqb -= am2b;
#pragma unroll
  for (int d = 0; d < 2; d++) umb[d] += usqb * um[d] + unmb * n[d];
  const double rrb = (umb[0] * um[0] + umb[1] * um[1] + hmb * hm) / rr;
  const double sqb = rr * (umb[0] * v[1][0] + umb[1] * v[1][1] + hmb * h[1]) - rrb * rr * rr;
  const double vnb = dvn < 0 ? -0.5 * epsb : 0.5 * epsb, cb = dc < 0 ? -0.5 * epsb : 0.5 * epsb;
  const double vLb[2] = {rr * umb[0], rr * umb[1]}, vRb[2] = {rr * sq * umb[0], rr * sq * umb[1]};
#pragma unroll
  for (int i = 0; i < 4; i++) {
    ubL[i] = -dub[i];
    ubR[i] = dub[i];
  }
  ubL[0] -= 0.5 * sqb * sq * ir[0];
  ubR[0] += 0.5 * sqb * sq * ir[1];
  vjp_side<2>(v[0], n, ir[0], vn[0], p[0], h[0], c[0], g1, vLb, rr * hmb, vnb, cb, ubL);
  vjp_side<2>(v[1], n, ir[1], vn[1], p[1], h[1], c[1], g1, vRb, rr * sq * hmb, -vnb, -cb, ubR);
  vjp_normal_flux<2>(UL, n, hb, g1, ubL);
  vjp_normal_flux<2>(UR, n, hb, g1, ubR);
}

// A ghost state's transpose (bc_ghost_t): rb^T dUR/dU added to ub; returns rb^T
// dUR/dtheta for the direction th of the boundary state (rhoB, vB, pB).
template <int DIM>
__device__ __forceinline__ double vjp_ghost(int bc, const double *U, const double *n, const double *rb, const Phys &ph,
                                            const double *th, double *ub) {
  const double g = ph.gamma, g1 = g - 1.0, ir = 1.0 / U[0], rE = rb[DIM + 1];
  double v[DIM], vv = 0, vn = 0, vBn = 0, vB2 = 0, rv = 0, rvB = 0, rn = 0;
#pragma unroll
  for (int d = 0; d < DIM; d++) {
    v[d] = U[d + 1] * ir;
    vv += v[d] * v[d];
    vn += v[d] * n[d];
    vBn += ph.vB[d] * n[d];
    vB2 += ph.vB[d] * ph.vB[d];
    rv += rb[d + 1] * v[d];
    rvB += rb[d + 1] * ph.vB[d];
    rn += rb[d + 1] * n[d];
  }
  const double p = g1 * (U[DIM + 1] - 0.5 * U[0] * vv);
  double pb = 0, theta = 0;  // adjoint of the interior pressure
  double vb[DIM] = {}, vnb = 0, cb = 0, c = 0;
  switch (bc) {
    case BC_SUB_IN:
      pb = rE / g1;
      theta = th[0] * (rb[0] + rvB + rE * 0.5 * vB2);
#pragma unroll
      for (int d = 0; d < DIM; d++) theta += th[1 + d] * ph.rhoB * (rb[d + 1] + rE * ph.vB[d]);
      break;
    case BC_SUB_OUT:
      ub[0] += rb[0] - rE * 0.5 * vv;
#pragma unroll
      for (int d = 0; d < DIM; d++) ub[d + 1] += rb[d + 1] + rE * v[d];
      theta = th[4] * rE / g1;
      break;
    case BC_SUP_IN:
      theta = th[0] * (rb[0] + rvB + rE * 0.5 * vB2) + th[4] * rE / g1;
#pragma unroll
      for (int d = 0; d < DIM; d++) theta += th[1 + d] * ph.rhoB * (rb[d + 1] + rE * ph.vB[d]);
      break;
    case BC_SUP_OUT:
#pragma unroll
      for (int i = 0; i < DIM + 2; i++) ub[i] += rb[i];
      break;
    case BC_SLIP:
    case BC_SYMMETRY:
      ub[0] += rb[0];
#pragma unroll
      for (int d = 0; d < DIM; d++) ub[d + 1] += rb[d + 1] - 2.0 * rn * n[d];
      ub[DIM + 1] += rE;
      break;
    case BC_ISO_NOSLIP_MOVING:
    case BC_ISO_NOSLIP: {
      double q = rb[0], w2 = 0;
      if (bc == BC_ISO_NOSLIP_MOVING) {
#pragma unroll
        for (int d = 0; d < DIM; d++) {
          q += rb[d + 1] * ph.vWall[d];
          w2 += ph.vWall[d] * ph.vWall[d];
        }
      }
      pb = (q + rE * 0.5 * w2) / (ph.RGas * ph.TWall) + rE / g1;
      break;
    }
    case BC_ADI_NOSLIP:
      ub[0] += rb[0];
      pb = rE / g1;
      break;
    case BC_CHAR: {
      // the forward's intermediate values, then their adjoints
      const bool in = vn < 0;
      c = sqrt(g * p * ir);
      const double cB = sqrt(g * ph.pB / ph.rhoB), k = 2.0 / g1;
      const bool sup = fabs(vBn) >= cB, lB = sup && !in, bL = sup && in;
      const double RL = lB ? vBn + k * cB : vn + k * c, RB = bL ? vn - k * c : vBn - k * cB;
      const double f = 0.25 * g1 * (RL - RB), s0 = in ? pow(ph.rhoB, g) / ph.pB : pow(U[0], g) / p;
      const double rho = pow(f * f / g * s0, 1.0 / g1), VB = 0.5 * (RL + RB);
      double w[DIM], w2 = 0, rw = 0, wb[DIM], wn = 0;
#pragma unroll
      for (int d = 0; d < DIM; d++) {
        w[d] = in ? ph.vB[d] + (VB - vBn) * n[d] : v[d] + (VB - vn) * n[d];
        w2 += w[d] * w[d];
        rw += rb[d + 1] * w[d];
        wb[d] = rho * (rb[d + 1] + rE * w[d]);
        wn += wb[d] * n[d];
      }
      const double rhob = rb[0] + rw + rE * 0.5 * w2 + rE / g1 * f * f / g, y = rhob * rho / g1;
      const double fb = rE / g1 * 2.0 * f * rho / g + 2.0 * y / f;
      const double RLb = 0.25 * g1 * fb + 0.5 * wn, RBb = -0.25 * g1 * fb + 0.5 * wn;
      double vBnb = 0, cBb = 0;
      if (lB) { vBnb += RLb; cBb += k * RLb; }
      else { vnb += RLb; cb += k * RLb; }
      if (bL) { vnb += RBb; cb -= k * RBb; }
      else { vBnb += RBb; cBb -= k * RBb; }
      double rhoBb = -0.5 * cBb * cB / ph.rhoB, pBb = 0.5 * cBb * cB / ph.pB;
      if (in) {
        rhoBb += y * g / ph.rhoB;
        pBb -= y / ph.pB;
        vBnb -= wn;
      } else {
        ub[0] += y * g * ir;
        pb = -y / p;
        vnb -= wn;
      }
      theta = th[0] * rhoBb + th[4] * pBb;
#pragma unroll
      for (int d = 0; d < DIM; d++) {
        theta += th[1 + d] * ((in ? wb[d] : 0.0) + vBnb * n[d]);
        vb[d] = in ? 0.0 : wb[d];
      }
      break;
    }
    default:
      break;
  }
  vjp_side<DIM>(v, n, ir, vn, p, 0.0, c, g1, vb, 0.0, vnb, cb, ub, pb);
  return theta;
}

// Block of the stage kernel: narrow tiles and a thread per flux point.  What
// bounds it is the latency of one block's chain (the adjoint's meshes are small):
// loads, the Riemann solver's transpose with its dependent FP64 divisions and
// roots, barriers.  Per reversed stage of 3,072 quads, P = 3, walls, Roe (one
// B200): 27.3 us with the face-seed and dual-number element kernels this replaces,
// 16.2 with a thread per line that took both ends (3,133 instructions in a row: a
// warp waited 3.6 of its 10.4 cycles per instruction for the instruction cache),
// 13.4 in this form.
template <class C>
struct AdjTile {
  static constexpr int TE = C::DIM == 2 ? 8 : C::P == 1 ? 8 : C::P < 4 ? 4 : 2;
  static constexpr int NC = C::DIM == 2 ? C::N1 : C::N1 * C::N1;
  static constexpr int NT = (C::NF * TE + 31) & ~31;
  using T = LineT<C, double, TE, NT>;
  static constexpr int BUF = C::DIM * T::BUF;      // values of one set of line buffers
  static constexpr int ENDS = C::NF * C::NV * TE;  // one value per field and line end
  static constexpr int SMEM = (2 * BUF + 2 * ENDS) * 8;
  static constexpr int MINB = NT <= 128 ? 3 : NT <= 192 ? 2 : 1;  // at most 168 registers
};

template <class C, bool BC, int RS>
__global__ void __launch_bounds__(AdjTile<C>::NT, AdjTile<C>::MINB) fr_adj_stage_kernel(const AdjArgs a, const OpTab<double> op) {
  using A = AdjTile<C>;
  using T = typename A::T;
  constexpr int TE = A::TE, NT = A::NT, NS = C::NS, NF = C::NF, NV = C::NV, DIM = C::DIM, N1 = C::N1;
  constexpr int NLN = DIM * A::NC;  // lines of an element
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double *G = reinterpret_cast<double *>(smem_raw);  // the seed's lines, then the contravariant flux's adjoint
  double *W = G + A::BUF;                            // the traces' part of the state's adjoint
  double *JB = W + A::BUF, *UB = JB + A::ENDS;       // [side][NV][line][TE]: jump and trace adjoints at the ends
  __shared__ double red[NT / 32];
  const Phys &ph = a.ph;
  const int e0 = blockIdx.x * TE, L = a.nE;
  StageArgs sa{};  // the size line_point reads
  sa.nEle = a.nEle;
  // this thread's line end
  const int it = threadIdx.x / TE, e = threadIdx.x - it * TE, eg = e0 + e;
  const int side = it >= NLN, ln = it - side * NLN, dir = ln / A::NC, c = ln - dir * A::NC;
  const int p = DIM == 2 ? c : c % N1, q = DIM == 2 ? 0 : c / N1;
  const bool act = eg < a.nEle && it < 2 * NLN;
  const int base = dir * T::BUF + c * T::N1P * TE + e, end = (side * NV * NLN + ln) * TE + e;
  pdl_wait();
  pdl_launch_dependents();

  // ---- the seed's points into lines, and this thread's end
  const size_t fl = (size_t)NF * L, at = (size_t)(act ? line_fpt<C>(dir, side, p, q) : 0) * L + eg;
  int code = 0;
  if (act) code = __ldg(a.nbr + at);
#pragma unroll
  for (int r = 0; r < T::NP; r++) {
    int s, ep;
    if (!line_point<T, NS>(sa, r, e0, s, ep)) continue;
    double gb[NV];
#pragma unroll
    for (int v = 0; v < NV; v++) gb[v] = __ldcg(a.gbar + ((size_t)v * NS + s) * L + e0 + ep);
    line_put_state<C, double, T>(G, gb, s % N1, (s / N1) % N1, DIM == 3 ? s / (N1 * N1) : 0, ep);
  }
  double n[DIM], dA = 0, own[NV], oth[NV], fb[NV];
  if (act) {
    const size_t o = code >= 0 ? (size_t)(code >> 1) : at;
    dA = __ldg(a.dA + at);
#pragma unroll
    for (int d = 0; d < DIM; d++) n[d] = __ldg(a.nrm + d * fl + at);
#pragma unroll
    for (int v = 0; v < NV; v++) {
      own[v] = __ldcg(a.trY + v * fl + at);
      oth[v] = __ldcg(a.trY + v * fl + o);
      fb[v] = __ldcg(a.fnbar + v * fl + o);
    }
  }
  const bool right = code >= 0 && (code & 1);
  const double sA = right ? -dA : dA;
  __syncthreads();

  // ---- per end: the correction's and the face flux's transposes
  double theta = 0;
  if (act) {
    double ub[NV];
#pragma unroll
    for (int v = 0; v < NV; v++) {
      double jb = 0;
#pragma unroll
      for (int j = 0; j < N1; j++) jb += (side ? op.gR[j] : -op.gL[j]) * G[base + (v * T::NL + j) * TE];
      JB[end + v * NLN * TE] = jb;
      fb[v] = code >= 0 ? sA * jb + fb[v] : sA * jb;
    }
    if constexpr (NV == 1) {
      double vN = 0;
#pragma unroll
      for (int d = 0; d < DIM; d++) vN += ph.adv[d] * n[d];
      const double up = 0.5 * ph.lambda * fabs(vN);
      ub[0] = fb[0] * (0.5 * vN + (right ? -up : up));  // a boundary's ghost state stays zero
      if (!BC && code < 0) atomicOr(a.err, ERRF_BC);
    } else {
      double UL[NV], UR[NV], bR[NV];
      bool wall = false;
      if constexpr (BC) {
        wall = code < 0;
        if (wall && !bc_ghost<DIM>(-1 - code, own, n, oth, ph)) atomicOr(a.err, ERRF_BC);
      } else if (code < 0) {
        atomicOr(a.err, ERRF_BC);
      }
#pragma unroll
      for (int v = 0; v < NV; v++) {
        UL[v] = right ? oth[v] : own[v];
        UR[v] = right ? own[v] : oth[v];
      }
      // boundary faces always use Rusanov (src/face.cpp:142-145)
      if (RS == 1 && DIM == 2 && !wall) {
        if constexpr (DIM == 2) vjp_roe2d(UL, UR, n, fb, ph.gamma, ub, bR);
      } else if (RS == 0 || DIM == 3 || BC) {
        vjp_rusanov<DIM>(UL, UR, n, fb, ph.gamma, ub, bR);
      }
      if constexpr (BC)
        if (wall) theta = vjp_ghost<DIM>(-1 - code, own, n, bR, ph, a.thetaDir, ub);
#pragma unroll
      for (int v = 0; v < NV; v++) ub[v] = right ? bR[v] : ub[v];
    }
#pragma unroll
    for (int v = 0; v < NV; v++) UB[end + v * NLN * TE] = ub[v];
  }
  if constexpr (BC) {
    for (int o = 16; o > 0; o >>= 1) theta += __shfl_xor_sync(0xffffffffu, theta, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = theta;
  }
  __syncthreads();
  if constexpr (BC) {
    if (a.thetaBar && threadIdx.x == 0) {
      double x = 0;
      for (int w = 0; w < NT / 32; w++) x += red[w];
      if (x != 0) atomicAdd(a.thetaBar, x);
    }
  }

  // ---- per line: side 0's thread the derivative's transpose less the
  // extrapolated normal flux's (over the seed), side 1's the traces' transpose
  if (act) {
    const double *E = side ? UB : JB;
    const int en = ln * TE + e;
#pragma unroll
    for (int v = 0; v < NV; v++) {
      const double lo = E[en + v * NLN * TE], hi = E[en + (NV + v) * NLN * TE];
      if (side) {
#pragma unroll
        for (int i = 0; i < N1; i++) W[base + (v * T::NL + i) * TE] = op.lag[0][i] * lo + op.lag[1][i] * hi;
      } else {
        double g[N1];
#pragma unroll
        for (int i = 0; i < N1; i++) g[i] = G[base + (v * T::NL + i) * TE];
#pragma unroll
        for (int i = 0; i < N1; i++) {
          double x = op.lag[0][i] * lo - op.lag[1][i] * hi;
#pragma unroll
          for (int j = 0; j < N1; j++) x += op.dlag[j][i] * g[j];
          G[base + (v * T::NL + i) * TE] = x;
        }
      }
    }
  }
  __syncthreads();

  // ---- per point: the metric's and the flux Jacobians' transposes, the reverse
  // RK update, and the next stage's seed and state over the lines
  const bool next = a.Ynext != nullptr, rk = a.mode & ADJ_RK, first = a.mode & ADJ_RK_FIRST;
#pragma unroll 1
  for (int r = 0; r < T::NP; r++) {
    int s, ep;
    if (!line_point<T, NS>(sa, r, e0, s, ep)) continue;
    const int i = s % N1, j = (s / N1) % N1, k = DIM == 3 ? s / (N1 * N1) : 0;
    double u[NV], lam[NV], lnew[NV], yn[NV], JG[DIM][DIM];
    const size_t g0 = (size_t)s * L + e0 + ep, gs = (size_t)NS * L;
#pragma unroll
    for (int v = 0; v < NV; v++) u[v] = __ldcg(a.Y + g0 + v * gs);
    if (rk) {
#pragma unroll
      for (int v = 0; v < NV; v++) {
        lam[v] = __ldcg(a.lam + g0 + v * gs);
        lnew[v] = first ? lam[v] : __ldcg(a.lamNew + g0 + v * gs);
      }
    }
    if (next) {
#pragma unroll
      for (int v = 0; v < NV; v++) yn[v] = __ldcg(a.Ynext + g0 + v * gs);
    }
#pragma unroll
    for (int d1 = 0; d1 < DIM; d1++)
#pragma unroll
      for (int d2 = 0; d2 < DIM; d2++) JG[d1][d2] = __ldg(a.JG + (size_t)(d1 * DIM + d2) * gs + g0);
    const double D = (a.grp ? a.dtGrp[a.grp[e0 + ep]] : a.dt) * __ldg(a.invDet + g0);
    int o[DIM];
#pragma unroll
    for (int d = 0; d < DIM; d++) o[d] = d * T::BUF + line_slot<T>(d, i, j, k, ep);
    double yb[NV], Fs[DIM][NV];
#pragma unroll
    for (int v = 0; v < NV; v++) {
      yb[v] = 0;
#pragma unroll
      for (int d = 0; d < DIM; d++) {
        Fs[d][v] = G[o[d] + v * T::NL * TE];
        yb[v] += W[o[d] + v * T::NL * TE];
      }
    }
#pragma unroll
    for (int d2 = 0; d2 < DIM; d2++) {
      double Fb[NV];
#pragma unroll
      for (int v = 0; v < NV; v++) {
        Fb[v] = 0;
#pragma unroll
        for (int d1 = 0; d1 < DIM; d1++) Fb[v] += JG[d1][d2] * Fs[d1][v];
      }
      if constexpr (NV == 1) {
        yb[0] += ph.adv[d2] * Fb[0];
      } else {
        double ed[DIM] = {};
        ed[d2] = 1.0;
        vjp_normal_flux<DIM>(u, ed, Fb, ph.gamma - 1.0, yb);
      }
    }
    double sd[NV];
#pragma unroll
    for (int v = 0; v < NV; v++) {
      const size_t gi = g0 + v * gs;
      sd[v] = 0;
      if (a.mode & ADJ_PLAIN) a.ybar[gi] = yb[v];
      if (rk) {
        // the adjoint of the step's initial state collects every stage's ybar
        const double x = lnew[v] + yb[v];
        a.lamNew[gi] = x;
        sd[v] = (a.mode & ADJ_RK_LAST) ? -a.cLam * x * D : -(a.cLam * lam[v] + a.cY * yb[v]) * D;
        a.seedOut[gi] = sd[v];
      }
    }
    if (next) {
      line_put_state<C, double, T>(G, sd, i, j, k, ep);
      line_put_state<C, double, T>(W, yn, i, j, k, ep);
    }
  }
  if (!next) return;
  __syncthreads();
  if (act) {
#pragma unroll
    for (int v = 0; v < NV; v++) {
      double x = 0, y = 0;
#pragma unroll
      for (int j = 0; j < N1; j++) {
        x += (side ? op.lag[1][j] : op.lag[0][j]) * W[base + (v * T::NL + j) * TE];
        y += (side ? op.gR[j] : -op.gL[j]) * G[base + (v * T::NL + j) * TE];
      }
      a.trNext[v * fl + at] = x;
      a.fnNext[v * fl + at] = sA * y;
    }
  }
}

// ---------------------------------------------------------------------------
// Objectives and their gradients with respect to the solution-point state.
// ---------------------------------------------------------------------------

// Entropy error integral, sum_e sum_s w_s detJ (p rhoB^gamma / (rho^gamma pB) - 1)
// (integrateError with the freestream entropy error, src/solver.cpp:1507-1531;
// src/funcs.cpp:1891-1901).  Per-block partial sums in `part`.
template <int DIM, int NV>
__global__ void __launch_bounds__(256) fr_obj_entropy_kernel(const double *U, const double *detJ,
                                                             const double *wvol, int NS, int nE, int L,
                                                             Phys ph, double *grad, double *part) {
  using D0 = ad::Dual<NV>;
  __shared__ double red[8];
  double acc = 0;
  const long n = (long)NS * L;
  const double rfg = pow(ph.rhoB, ph.gamma);
  for (long it = blockIdx.x * (long)blockDim.x + threadIdx.x; it < n; it += (long)gridDim.x * blockDim.x) {
    const int s = (int)(it / L), e = (int)(it - (long)s * L);
    if (e >= nE) {
      for (int v = 0; v < NV; v++) grad[(size_t)v * NS * L + it] = 0;
      continue;
    }
    D0 u[NV];
    for (int v = 0; v < NV; v++) {
      u[v] = D0(U[(size_t)v * NS * L + it]);
      u[v].d[v] = 1.0;
    }
    D0 ke = 0;
    for (int d = 0; d < DIM; d++) ke += u[d + 1] * u[d + 1];
    const D0 p = (ph.gamma - 1.) * (u[DIM + 1] - .5 * ke / u[0]);
    const D0 err = p * rfg / (ad::pow(u[0], ph.gamma) * ph.pB) - 1.;
    const double wj = wvol[s] * detJ[it];
    acc += err.v * wj;
    for (int v = 0; v < NV; v++) grad[(size_t)v * NS * L + it] = err.d[v] * wj;
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += red[w];
    part[blockIdx.x] = t;
  }
}

// Pressure integrated over the slip-wall faces with the face quadrature of
// boundFace::computeWallForce (src/boundFace.cpp:330-378): sum w_f p(U_f) dA_f
// over wall flux points, U_f the element's trace.  One thread per element;
// `grad` must be zero on entry (only wall elements write).
template <class C>
__global__ void __launch_bounds__(128) fr_obj_wallp_kernel(const double *U, const int *nbr, const double *dA,
                                                           const double *wsurf, int vcjh, int nE, int L, int bcWall,
                                                           Phys ph, double *grad, double *part) {
  constexpr int NV = C::NV, NS = C::NS, NF = C::NF, N1 = C::N1, DIM = C::DIM;
  using D0 = ad::Dual<NV>;
  const OpTab<double> &op = optab<double>(vcjh, C::P);
  __shared__ double red[4];
  double acc = 0;
  const int eg = blockIdx.x * blockDim.x + threadIdx.x;
  if (eg < nE) {
    for (int f = 0; f < NF; f++) {
      const int code = nbr[(size_t)f * L + eg];
      if (code >= 0 || -1 - code != bcWall) continue;
      int dir, side, s0, st;
      fpt_line<C>(f, dir, side, s0, st);
      D0 u[NV];
      for (int v = 0; v < NV; v++) {
        double t = 0;
        for (int j = 0; j < N1; j++) t += op.lag[side][j] * U[((size_t)v * NS + s0 + j * st) * L + eg];
        u[v] = D0(t);
        u[v].d[v] = 1.0;
      }
      D0 ke = 0;
      for (int d = 0; d < DIM; d++) ke += u[d + 1] * u[d + 1] / (u[0] * u[0]);
      const D0 p = (ph.gamma - 1) * (u[DIM + 1] - 0.5 * u[0] * ke);
      const double wd = wsurf[f % C::NFF] * dA[(size_t)f * L + eg];
      acc += p.v * wd;
      for (int v = 0; v < NV; v++)
        for (int j = 0; j < N1; j++) grad[((size_t)v * NS + s0 + j * st) * L + eg] += op.lag[side][j] * p.d[v] * wd;
    }
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += red[w];
    part[blockIdx.x] = t;
  }
}

}  // namespace frg
