// kernels.cuh -- what the FR kernels share for sm_100a: operator tables, sizes
// and point numbering of one configuration, the arguments of a stage launch, the
// common inviscid flux, and the trace and wave-speed kernels.
//
// Data layout in HBM: every per-point array is [field][point][element] with
// the element index fastest, so a warp's lanes (consecutive elements at one
// point) issue coalesced accesses.
//
// The stage kernels do a whole RK stage in one launch per tile of elements
// (kernels_line.cuh: a thread per coordinate line; kernels_tma.cuh: the 2D
// inviscid update over tiles moved by TMA):
//
//   A  stage state, pointwise flux + metric transform
//        (solver::calcInviscidFlux_spts, src/solver.cpp:514-539)
//   B  per flux point: own trace (extrapolateU, :401-412), neighbour trace
//        (gathered from the previous launch's trace buffer), common flux
//        (face::calcInviscidFlux, src/face.cpp:132-175), the extrapolated
//        normal flux (extrapolateNormalFlux, :729-787) and the jump
//        Fn*dA - disFn (correctDivFlux, :789-806)
//   C  divergence + correction (calcDivF_spts :707-727, correctDivFlux), then
//        the RK stage update (timeStepA/B, :307-385) in FP64
//   D  traces of the new state for the next launch
//
// The spts->fpts, gradient and correction operators are Kronecker products
// of 1D tables, so they are applied by sum factorisation along one
// coordinate line: (P+1) terms per output instead of nSpts or nFpts.  Each
// face's common flux is evaluated by both elements that share it, in the
// reference's left/right order with the left element's normal, so both get the
// reference's values; this removes the separate face pass and its flux round
// trip through HBM.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "physics.cuh"

namespace frg {

constexpr int KMAXP = 5;

// 1D operator tables (see setup.h Ops1D), per VCJH scheme and order.
template <typename R>
struct OpTab {
  R lag[2][KMAXP + 1];
  R dlag[KMAXP + 1][KMAXP + 1];
  R gL[KMAXP + 1], gR[KMAXP + 1];
  R w[KMAXP + 1];
};
// Each CUDA translation unit that includes this header holds its own copy of
// the tables (internal linkage) and uploads it through its own entry point.
static __constant__ OpTab<double> c_opd[4][KMAXP + 1];
static __constant__ OpTab<float> c_opf[4][KMAXP + 1];

template <typename R>
__device__ __forceinline__ const OpTab<R> &optab(int vcjh, int P);
template <>
__device__ __forceinline__ const OpTab<double> &optab<double>(int vcjh, int P) { return c_opd[vcjh][P]; }
template <>
__device__ __forceinline__ const OpTab<float> &optab<float>(int vcjh, int P) { return c_opf[vcjh][P]; }

// Error flag bits written by kernels; the host reads the word after a step.
enum : unsigned { ERRF_NAN = 1u, ERRF_DT = 2u, ERRF_BC = 4u };

// Compile-time sizes of one (dimension, order, fields) configuration.
template <int DIM_, int P_, int NV_>
struct Cfg {
  static constexpr int DIM = DIM_, P = P_, NV = NV_, N1 = P_ + 1;
  static constexpr int NS = DIM == 2 ? N1 * N1 : N1 * N1 * N1;
  static constexpr int NFF = DIM == 2 ? N1 : N1 * N1;
  static constexpr int NF = 2 * DIM * NFF;
};
// Geometry of flux point f: normal direction, side (0: -1 face, 1: +1 face),
// first solution point of the coordinate line through it and that line's stride.
template <class C>
__device__ __forceinline__ void fpt_line(int f, int &dir, int &side, int &s0, int &stride) {
  constexpr int P = C::P, N1 = C::N1;
  if constexpr (C::DIM == 2) {
    int face = f / N1, k = f - face * N1;
    switch (face) {
      case 0: dir = 1; side = 0; s0 = k; stride = N1; break;
      case 1: dir = 0; side = 1; s0 = k * N1; stride = 1; break;
      case 2: dir = 1; side = 1; s0 = P - k; stride = N1; break;
      default: dir = 0; side = 0; s0 = (P - k) * N1; stride = 1; break;
    }
  } else {
    constexpr int P12 = N1 * N1;
    int face = f / P12, k = f - face * P12, a = k % N1, b = k / N1;
    switch (face) {
      case 0: dir = 2; side = 0; s0 = a + N1 * b; stride = P12; break;
      case 1: dir = 2; side = 1; s0 = (P - a) + N1 * b; stride = P12; break;
      case 2: dir = 0; side = 0; s0 = N1 * a + P12 * b; stride = 1; break;
      case 3: dir = 0; side = 1; s0 = N1 * (P - a) + P12 * b; stride = 1; break;
      case 4: dir = 1; side = 0; s0 = (P - a) + P12 * b; stride = N1; break;
      default: dir = 1; side = 1; s0 = a + P12 * b; stride = N1; break;
    }
  }
}

// Flux points whose correction reaches solution point (i,j[,k]), in face
// order, with the sign of the correction-function derivative they carry
// (divVCJH_quad / divVCJH_hex, src/operators.cpp:1544-1619).
template <class C>
__device__ __forceinline__ void corr_fpts(int i, int j, int k, int fp[2 * C::DIM], int side[2 * C::DIM],
                                          int at[2 * C::DIM]) {
  constexpr int P = C::P, N1 = C::N1;
  if constexpr (C::DIM == 2) {
    fp[0] = i;                  side[0] = 0; at[0] = j;
    fp[1] = N1 + j;             side[1] = 1; at[1] = i;
    fp[2] = 2 * N1 + (P - i);   side[2] = 1; at[2] = j;
    fp[3] = 3 * N1 + (P - j);   side[3] = 0; at[3] = i;
  } else {
    constexpr int P12 = N1 * N1;
    fp[0] = i + N1 * j;                 side[0] = 0; at[0] = k;
    fp[1] = P12 + (P - i) + N1 * j;     side[1] = 1; at[1] = k;
    fp[2] = 2 * P12 + j + N1 * k;       side[2] = 0; at[2] = i;
    fp[3] = 3 * P12 + (P - j) + N1 * k; side[3] = 1; at[3] = i;
    fp[4] = 4 * P12 + (P - i) + N1 * k; side[4] = 0; at[4] = j;
    fp[5] = 5 * P12 + i + N1 * k;       side[5] = 1; at[5] = j;
  }
}

// Stage modes
enum : int {
  SF_WAVESP = 1,    // store Rusanov / LF wave speeds of left-side flux points
  SF_FIRST = 2,     // first RK stage: accumulator = U0 - b t
  SF_LAST = 4,      // last RK stage: U = accumulator - b t
  SF_RESIDUAL = 8,  // solver::calcResidual only: write divF, no update
  SF_JAMESON = 16,  // timeType 5: every stage U = U0 - a t
  SF_TIME = 32,     // advance the device time by dt (block 0)
  SF_DIVF = 64,     // also store divF (residual monitoring) during an update
  SF_DTNEXT = 128,  // last stage: compute the next step's CFL dt
  SF_PDL = 256,     // launch as a programmatic dependent of the previous kernel (host side)
  SF_DTUSED = 512   // last stage: dt is checked in the step that uses it, not where it is computed
};

// Arguments of one stage launch.  Arrays of the stored type S (double, or
// float in the mixed mode) are passed untyped and cast in the kernel.
struct StageArgs {
  int nE;    // element stride of the mesh arrays (geometry, traces), a multiple of 32
  int nEle;  // number of real elements
  int ldU;   // element stride of the state arrays (U, U0, Acc, W, divF)
  const double *Uin_d;  // stage input when stored in double (else null)
  const void *Uin_s;    // stage input in the stored type
  const double *U0;     // state at the start of the step
  double *Acc;          // running final combination U0 - sum_s b_s t_s
  double *Uout;         // final state (last stage); may alias U0
  void *Wout;           // next stage state (S)
  const void *trIn;     // traces of the input state (S), [NV][NF][nE]
  void *trOut;          // traces of the output state (S)
  double *divF;         // residual, [NV][NS][nE] (SF_RESIDUAL / SF_DIVF)
  const int *nbr;       // [NF][nE]
  const void *nrm;      // (S) [DIM][NF][nE] normal of the face's left element
  const void *dA;       // (S) [NF][nE]
  const void *JG;       // (S) [DIM][DIM][NS][nE]
  const void *invDet;   // (S) [NS][nE] 1 / detJ
  double *waveSp;       // [NF][nE]
  const double *dt;     // scalar, [nE] when dtLocal, or one per group when grp is set
  const int *grp;       // ensemble mode: group (independent case) of each element, else null
  double *time;         // device time (SF_TIME)
  const double *dtTime; // what it advances by: the global dt, with dtLocal the smallest of the elements'
  unsigned *err;
  double aNext, bCur;
  int dtLocal, flags, vcjh;
  // viscous path: this side's projected viscous flux per flux point (S),
  // [NV][NF][nE]; the second array only for the 3D LDG penalty term
  void *fvnOut, *fvn2Out;
  const void *fvnIn, *fvn2In;
  int visc2;
  // optional output of the gradient pass: the corrected physical gradient at the
  // solution points (S), [DIM][NV][NS][nE], for the boundary integrals and the adjoint
  void *dUg;
  // SF_DTNEXT: the next step's dt (ele::calcDt + the global minimum)
  const double *vol, *dAd, *wsurf;
  double *blockMin, *dtNext, *eleDt;
  // first stage of a step with the fused dt: the next step's dt
  // slot, set here to a huge value before the last stage minimises into it
  double *dtReset;
  unsigned *ticket;
  double cflFac;
  int nff;
  Phys ph;
  // the run's 1D operator tables (order, VCJH scheme), in the launch
  // parameters so the kernels' unrolled loops read them as constant-bank
  // operands rather than by indexed loads
  OpTab<float> opf;
  OpTab<double> opd;
};

template <typename R>
__device__ __forceinline__ const OpTab<R> &stage_op(const StageArgs &a);
template <>
__device__ __forceinline__ const OpTab<double> &stage_op<double>(const StageArgs &a) { return a.opd; }
template <>
__device__ __forceinline__ const OpTab<float> &stage_op<float>(const StageArgs &a) { return a.opf; }
// Host: fill a launch's tables from the 1D operators (setup.h Ops1D), cast
// as the constant-memory copies are.
template <class Ops>
inline void set_stage_ops(StageArgs &a, const Ops &o) {
  for (int i = 0; i <= KMAXP; i++) {
    for (int h = 0; h < 2; h++) {
      a.opd.lag[h][i] = o.lag[h][i];
      a.opf.lag[h][i] = (float)o.lag[h][i];
    }
    a.opd.gL[i] = o.gL[i];
    a.opd.gR[i] = o.gR[i];
    a.opd.w[i] = o.w[i];
    a.opf.gL[i] = (float)o.gL[i];
    a.opf.gR[i] = (float)o.gR[i];
    a.opf.w[i] = (float)o.w[i];
    for (int j = 0; j <= KMAXP; j++) {
      a.opd.dlag[i][j] = o.dlag[i][j];
      a.opf.dlag[i][j] = (float)o.dlag[i][j];
    }
  }
}

// ----------------------------------------------------------------------------
// The fused stage kernels and the block-level phases they share.
// R: arithmetic type; S: stored type of stage states, traces and metrics.
// BC: the mesh has boundary faces (else the ghost-state code is not built);
// RS: interior Riemann solver, 0 Rusanov, 1 Roe (boundaries always Rusanov,
// src/face.cpp:142-145).
// ----------------------------------------------------------------------------

// Common inviscid flux of face::calcInviscidFlux (src/face.cpp:132-175).
// Returns the wave speed the reference stores (negative for Roe).
template <class C, typename R, bool BC, int RS>
__device__ __forceinline__ R inviscid_common(const R *UL, const R *UR, const R *n, int code, R *Fn,
                                             const Phys &ph) {
  constexpr int NV = C::NV, DIM = C::DIM;
  if constexpr (NV == 1) {
    return lax_friedrichs<DIM, R>(UL[0], UR[0], n, Fn, ph);
  } else if constexpr (RS == 0 || DIM == 3) {
    return rusanov_normal<DIM, R, double>(UL, UR, n, Fn, ph);
  } else if constexpr (BC) {
    if (code < 0) return rusanov_normal<DIM, R, double>(UL, UR, n, Fn, ph);
    roe2d<R, double>(UL, UR, n, Fn, ph);
    return -1;
  } else {
    roe2d<R, double>(UL, UR, n, Fn, ph);
    return -1;
  }
}

// The jump Fn dA - disFn at a flux point (extrapolateNormalFlux, correctDivFlux):
// Fn along the left element's normal, ext the contravariant flux extrapolated
// along its coordinate.
template <typename R>
__device__ __forceinline__ R face_jump(R Fn, bool right, R dA, int side, R ext) {
  return Fn * (right ? -dA : dA) - (side ? ext : -ext);
}

// RK update of one value (timeStepA/B, src/solver.cpp:307-385) from dj = divF /
// detJ; base is the accumulator (first stage, Jameson form: U0).  Returns the new
// state, and in accNew the new accumulator.
__device__ __forceinline__ double rk_update(int flags, double dj, double base, double u0, double cb, double ca,
                                            double &accNew) {
  accNew = 0;
  if (flags & SF_JAMESON) return base - ca * dj;
  accNew = base - cb * dj;
  if (flags & SF_LAST) return accNew;
  return ((flags & SF_FIRST) ? base : u0) - ca * dj;
}

// LDG penalty sign: face::ldgSolution (src/face.cpp:590-598).
template <int DIM, typename R>
__device__ __forceinline__ R ldg_pen(const R *n, double penFact) {
  if constexpr (DIM == 2) return (n[0] + n[1] < (R)0) ? (R)-penFact : (R)penFact;
  else return (n[0] + n[1] + (R)1.4142135623730951 * n[2] < (R)0) ? (R)-penFact : (R)penFact;
}

// Viscous flux [DIM][NV] of a state and its physical gradient.
template <class C, typename R>
__device__ __forceinline__ void visc_flux(const R *u, const R *g, R Fv[C::DIM][C::NV], const Phys &ph) {
  if constexpr (C::NV == 1) {
    R t[C::DIM][1];
    viscous_flux_ad<C::DIM, R>(g, t, ph);
#pragma unroll
    for (int d = 0; d < C::DIM; d++) Fv[d][0] = t[d][0];
  } else {
    viscous_flux<C::DIM, R>(u, g, Fv, ph);
  }
}

// ----------------------------------------------------------------------------
// Traces of a double state (solver::extrapolateU), one thread per
// (flux point, element).
// ----------------------------------------------------------------------------
template <class C, typename R, typename S>
__global__ void fr_trace_kernel(const double *__restrict__ U, S *__restrict__ tr, int nE, int nEle, int ldU,
                                int vcjh) {
  constexpr int NS = C::NS, NF = C::NF, NV = C::NV, N1 = C::N1;
  const OpTab<R> &op = optab<R>(vcjh, C::P);
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long)NF * nE) return;
  const int f = (int)(idx / nE), eg = (int)(idx - (long)f * nE);
  if (eg >= nEle) return;
  int dir, side, s0, st;
  fpt_line<C>(f, dir, side, s0, st);
#pragma unroll
  for (int v = 0; v < NV; v++) {
    R t = 0;
#pragma unroll
    for (int j = 0; j < N1; j++) t += op.lag[side][j] * (R)U[((size_t)v * NS + s0 + j * st) * ldU + eg];
    tr[((size_t)v * NF + f) * nE + eg] = (S)t;
  }
}

// A state in the reference's layout [spt][ele][field] into the device's, and the
// traces of it, in one launch: block row y < NS converts solution point y, the
// others form flux point y - NS's traces straight from the reference layout.
template <class C, typename R, typename S>
__global__ void __launch_bounds__(128) fr_import_kernel(const double *__restrict__ ref, double *__restrict__ U,
                                                        S *__restrict__ tr, int nEle, int L, int vcjh) {
  constexpr int NS = C::NS, NF = C::NF, NV = C::NV, N1 = C::N1;
  const int e = blockIdx.x * 128 + threadIdx.x, y = blockIdx.y;
  if (e >= nEle) return;
  if (y < NS) {
    const double *r = ref + ((size_t)y * nEle + e) * NV;
#pragma unroll
    for (int v = 0; v < NV; v++) U[(size_t)(v * NS + y) * L + e] = r[v];
    return;
  }
  const OpTab<R> &op = optab<R>(vcjh, C::P);
  const int f = y - NS;
  int dir, side, s0, st;
  fpt_line<C>(f, dir, side, s0, st);
  R t[NV];
#pragma unroll
  for (int v = 0; v < NV; v++) t[v] = 0;
#pragma unroll
  for (int j = 0; j < N1; j++) {
    const double *r = ref + ((size_t)(s0 + j * st) * nEle + e) * NV;
    const R l = op.lag[side][j];
#pragma unroll
    for (int v = 0; v < NV; v++) t[v] += l * (R)r[v];
  }
#pragma unroll
  for (int v = 0; v < NV; v++) tr[(size_t)(v * NF + f) * L + e] = (S)t[v];
}

// ele::calcWaveSpFpts (src/ele.cpp:1031-1084) for every flux point.
template <int DIM, int NV, typename S>
__global__ void fr_wavesp_kernel(const S *__restrict__ tr, const double *__restrict__ nrmOwn, double *waveSp,
                                 int NF, int nE, Phys ph) {
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long)NF * nE) return;
  const int f = (int)(idx / nE), e = (int)(idx - (long)f * nE);
  double n[DIM];
  for (int d = 0; d < DIM; d++) n[d] = nrmOwn[((size_t)d * NF + f) * nE + e];
  double ws;
  if constexpr (NV == 1) {
    double vN = ph.adv[0] * n[0] + ph.adv[1] * n[1];
    if constexpr (DIM == 3) vN += ph.adv[2] * n[2];
    double vTot = fabs(vN - 0.0);
    vN = fabs(vN);
    ws = fmax(vTot, fmax(vN, 0.0));
  } else {
    double U[NV];
    for (int v = 0; v < NV; v++) U[v] = (double)tr[((size_t)v * NF + f) * nE + e];
    double rho = U[0], u = U[1] / rho, v = U[2] / rho, w = 0;
    if constexpr (DIM == 3) w = U[3] / rho;
    double rhoVSq = rho * (u * u + v * v + w * w);
    double p = (ph.gamma - 1) * (U[DIM + 1] - 0.5 * rhoVSq);
    double vN = u * n[0] + v * n[1];
    if constexpr (DIM == 3) vN += w * n[2];
    double csq = fmax(ph.gamma * p / rho, 0.0);
    ws = (fabs(vN - 0.0) + sqrt(csq));
  }
  waveSp[(size_t)f * nE + e] = ws;
}

}  // namespace frg
