// kernels_line.cuh -- RK stage and residual kernels in which one thread owns
// one coordinate line of an element.
//
// A block holds TE elements and one thread per (direction, line, element).
// Point-wise work (fluxes, RK update) goes over the tile's solution points;
// everything that couples points of a line -- the extrapolation to its two
// ends, both end fluxes, the derivative, the correction, the traces of the new
// state -- is done by the line's thread with the line in registers.  Between
// the two the values pass once through shared memory, in one buffer per
// direction in which each line is contiguous and is replaced in place by its
// result.  Operator entries are launch parameters with compile-time indices.
//
// What bounds it: the point-per-thread kernels this replaces were bound by
// instruction issue (every output re-read its lines from shared memory and
// indexed the operators by thread).  Here it is the latency of the loads, which
// are plain coalesced loads (element index fastest): long-scoreboard stalls are
// 4.4 of the 15.8 cycles a warp spends per instruction (barriers 1.9), DRAM is at 35 %.  Per step,
// us, before and after (one B200):
//   3D Euler 31x29x27   P = 3 FP32 1184 -> 572   FP64 1684 -> 882
//   3D Euler 16x16x16   P = 3 FP32  172 ->  97   FP64  300 -> 180
//   3D NS    32x32x32   P = 3 FP32 1840 -> 1471  FP64 3947 -> 3017 (before: a TMA pair)
//   3D NS    28x28x28   P = 2 FP32  854 -> 556   FP64 2147 -> 1045
//   2D NS    150x96     P = 3 FP32  198 -> 117;  75x48 P = 4 FP64 127 -> 82.5
// Tried and not kept: a thread per column of an element that takes the three
// directions in turn, its own column in registers (573 on the first line, twice
// the latency on small meshes); L2 prefetch of the next wave's tile (5-12 %
// slower: the requests queue with the loads).
#pragma once
#include "kernels_tma.cuh"

namespace frg {

// A block lets the next launch start only behind its own wait.  Signalled ahead of
// it, all the launches of a step (of a run of steps) start at once, and the blocks
// that wait hold the threads and shared memory of SMs that the running launch's
// blocks are then not spread over: 3D NS 7x7x6, P = 3 FP32, 117.8 us a step against
// 78.3 (79.4 without programmatic launches), 2D NS 48x47, P = 3 FP64, 73.5 against
// 50.5 (53.2); on meshes of a few blocks per SM and more no difference.
//
// Loads: metrics with the read-only path; what a stage writes (states, traces,
// the RK arrays) from L2, since with programmatic dependent launch this grid may
// have started before the previous one wrote them.

// Flux point at end `side` of the line with cross coordinates (p, q) along
// direction dir: 3D dir 0 (p, q) = (j, k), dir 1 (i, k), dir 2 (i, j); 2D
// dir 0 p = j, dir 1 p = i (the inverse of fpt_line).
template <class C>
__device__ __forceinline__ int line_fpt(int dir, int side, int p, int q) {
  constexpr int P = C::P, N1 = C::N1;
  if constexpr (C::DIM == 2) {
    if (dir == 0) return side ? N1 + p : 3 * N1 + P - p;
    return side ? 2 * N1 + P - p : p;
  } else {
    constexpr int P12 = N1 * N1;
    const int face = dir == 0 ? 2 : dir == 1 ? 4 : 0;
    const bool flip = (dir == 1) != (side == 1);
    return (face + side) * P12 + (flip ? P - p : p) + N1 * q;
  }
}

// What one end of a line reads: the face's normal (of its left element), area,
// neighbour code and this element's own trace; then the other side's trace.
// The viscous stage also reads both sides' projected viscous fluxes (vo this
// side's, vx the other's) and, with the 3D LDG penalty, the left side's second
// projection (vl).
template <class C, typename R, bool VISC = false>
struct LineEnd {
  R n[C::DIM], dA, own[C::NV], oth[C::NV];
  R vo[VISC ? C::NV : 1], vx[VISC ? C::NV : 1], vl[VISC ? C::NV : 1];
  int f, code;
};
// In three steps, so that both ends' loads are in flight together: the code,
// what lies at the flux point itself, and the gather (of the own values at a
// boundary, so it needs no branch).
template <class C, typename R, bool VISC>
__device__ __forceinline__ void line_end_code(const StageArgs &a, LineEnd<C, R, VISC> &L, int f, int eg) {
  L.f = f;
  L.code = __ldg(a.nbr + (size_t)f * (unsigned)a.nE + eg);
}
template <class C, typename R, typename S, bool VISC>
__device__ __forceinline__ void line_end_own(const StageArgs &a, LineEnd<C, R, VISC> &L, int eg) {
  constexpr int NF = C::NF, NV = C::NV, DIM = C::DIM;
  const size_t at = (size_t)L.f * (unsigned)a.nE + eg, fl = (size_t)NF * (unsigned)a.nE;
  const S *tr = static_cast<const S *>(a.trIn) + at, *nr = static_cast<const S *>(a.nrm) + at;
#pragma unroll
  for (int d = 0; d < DIM; d++) L.n[d] = (R)__ldg(nr + d * fl);
  L.dA = (R)__ldg(static_cast<const S *>(a.dA) + at);
#pragma unroll
  for (int v = 0; v < NV; v++) L.own[v] = (R)__ldcg(tr + v * fl);
  if constexpr (VISC) {
    const S *fv = static_cast<const S *>(a.fvnIn) + at;
#pragma unroll
    for (int v = 0; v < NV; v++) L.vo[v] = (R)__ldcg(fv + v * fl);
  }
}
template <class C, typename R, typename S, bool VISC>
__device__ __forceinline__ void line_end_gather(const StageArgs &a, LineEnd<C, R, VISC> &L, int eg) {
  constexpr int NF = C::NF, NV = C::NV, DIM = C::DIM;
  const size_t at = (size_t)L.f * (unsigned)a.nE + eg, fl = (size_t)NF * (unsigned)a.nE;
  const size_t t = L.code >= 0 ? (size_t)(L.code >> 1) : at;
  const S *tr = static_cast<const S *>(a.trIn) + t;
#pragma unroll
  for (int v = 0; v < NV; v++) L.oth[v] = (R)__ldcg(tr + v * fl);
  if constexpr (VISC) {
    const S *fv = static_cast<const S *>(a.fvnIn) + t;
#pragma unroll
    for (int v = 0; v < NV; v++) L.vx[v] = (R)__ldcg(fv + v * fl);
    const bool right = L.code & 1;
    if (DIM == 3 && a.visc2) {
      const S *f2 = static_cast<const S *>(a.fvn2In) + (right ? t : at);
#pragma unroll
      for (int v = 0; v < NV; v++) L.vl[v] = (R)__ldcg(f2 + v * fl);
    } else {
      // without a penalty the term is multiplied by zero: any finite value
#pragma unroll
      for (int v = 0; v < NV; v++) L.vl[v] = right ? L.vx[v] : L.vo[v];
    }
  }
}
// Both ends of a thread's line, in flight together.  Issued where they are used:
// ahead of the point-wise phase, steps were 1-6 % slower at P >= 2 (2D NS 75x48 P = 4
// FP64 86.0 against 82.5 us) and 2-4 % faster at P = 1, and 5-28 % slower where a block
// takes its lines in rounds: the registers they hold cost more than the latency
// they hide.
template <class C, typename R, typename S, bool VISC, class LT>
__device__ __forceinline__ void line_ends_load(const StageArgs &a, LineEnd<C, R, VISC> *E, const LT &t) {
#pragma unroll
  for (int s = 0; s < 2; s++) line_end_code<C, R>(a, E[s], t.fpt(s), t.eg);
#pragma unroll
  for (int s = 0; s < 2; s++) line_end_own<C, R, S>(a, E[s], t.eg);
#pragma unroll
  for (int s = 0; s < 2; s++) line_end_gather<C, R, S>(a, E[s], t.eg);
}
// Ghost state at a boundary end (in double, as other_side).
template <class C, typename R, bool BC, bool VISC>
__device__ __forceinline__ void line_end_ghost(const StageArgs &a, LineEnd<C, R, VISC> &L) {
  constexpr int NV = C::NV, DIM = C::DIM;
  if (L.code >= 0) return;
  if constexpr (NV == 1 || !BC) {
    // advection boundaries keep a zero ghost state (src/boundFace.cpp:274)
#pragma unroll
    for (int v = 0; v < NV; v++) L.oth[v] = 0;
    if constexpr (!BC) atomicOr(a.err, ERRF_BC);
  } else {
    double ul[NV], ur[NV], nd[DIM];
#pragma unroll
    for (int v = 0; v < NV; v++) ul[v] = L.own[v];
#pragma unroll
    for (int d = 0; d < DIM; d++) nd[d] = L.n[d];
    if (!bc_ghost<DIM>(-1 - L.code, ul, nd, ur, a.ph)) atomicOr(a.err, ERRF_BC);
#pragma unroll
    for (int v = 0; v < NV; v++) L.oth[v] = (R)ur[v];
  }
}

// Common flux at one end and the jump Fn dA - disFn; keeps the wave speed and,
// with SF_DTNEXT, leaves the end's term of ele::calcDt's sum in Ws.
template <class C, typename R, bool BC, int RS, int TE, bool VISC>
__device__ __forceinline__ void line_end_jump(const StageArgs &a, const LineEnd<C, R, VISC> &L, int side, const R *ext,
                                              double *Ws, int e, int eg, R *jump) {
  constexpr int NV = C::NV;
  const bool right = L.code >= 0 && (L.code & 1);
  R UL[NV], UR[NV], Fn[NV];
#pragma unroll
  for (int v = 0; v < NV; v++) {
    UL[v] = right ? L.oth[v] : L.own[v];
    UR[v] = right ? L.own[v] : L.oth[v];
  }
  const R ws = inviscid_common<C, R, BC, RS>(UL, UR, L.n, L.code, Fn, a.ph);
  const bool upd = !right && ws >= 0;
  if (a.flags & (SF_WAVESP | SF_DTNEXT)) {
    const size_t at = (size_t)L.f * a.nE + eg;
    if ((a.flags & SF_WAVESP) && upd) a.waveSp[at] = (double)ws;
    if (a.flags & SF_DTNEXT) Ws[L.f * TE + e] = (upd ? (double)ws : a.waveSp[at]) * a.wsurf[L.f % C::NFF] * a.dAd[at];
  }
  if constexpr (VISC) {
    // LDG viscous flux of the two sides (face::calcViscousFlux,
    // src/face.cpp:177-287); at a boundary the part the gradient pass formed
    R nn = 0;
#pragma unroll
    for (int d = 0; d < C::DIM; d++) nn += L.n[d] * L.n[d];
    const R tau = (R)a.ph.tau, pf = ldg_pen<C::DIM, R>(L.n, a.ph.penFact);
#pragma unroll
    for (int v = 0; v < NV; v++) {
      if (L.code >= 0) {
        const R FL = right ? L.vx[v] : L.vo[v], FR = right ? L.vo[v] : L.vx[v];
        if constexpr (NV == 1) Fn[v] += (R)0.5 * (FL + FR);  // centralFlux (src/flux.cpp:379-387)
        else Fn[v] += (R)0.5 * (FL + FR) + pf * nn * (L.vl[v] - FR) + tau * nn * (UL[v] - UR[v]);
      } else {
        Fn[v] += NV == 1 ? L.vo[v] : L.vo[v] + tau * nn * (UL[v] - UR[v]);
      }
    }
  }
#pragma unroll
  for (int v = 0; v < NV; v++) jump[v] = face_jump(Fn[v], right, L.dA, side, ext[v]);
}

// Both ends of a line and its part of the divergence, in place: on entry
// F[v][q] the contravariant flux along the line, on exit derivative plus
// correction.
template <class C, typename R, bool BC, int RS, int TE, bool VISC>
__device__ __forceinline__ void line_divergence(const StageArgs &a, const OpTab<R> &op, LineEnd<C, R, VISC> *E,
                                                R F[C::NV][C::N1], double *Ws, int e, int eg) {
  constexpr int NV = C::NV, N1 = C::N1;
  R jump[2][NV];
#pragma unroll
  for (int side = 0; side < 2; side++) {
    R ext[NV];
#pragma unroll
    for (int v = 0; v < NV; v++) {
      R q = 0;
#pragma unroll
      for (int j = 0; j < N1; j++) q += op.lag[side][j] * F[v][j];
      ext[v] = q;
    }
    if constexpr (BC || NV == 1) line_end_ghost<C, R, BC>(a, E[side]);
    line_end_jump<C, R, BC, RS, TE>(a, E[side], side, ext, Ws, e, eg, jump[side]);
  }
#pragma unroll
  for (int v = 0; v < NV; v++) {
    R d[N1];
#pragma unroll
    for (int i = 0; i < N1; i++) {
      R acc = 0;
#pragma unroll
      for (int q = 0; q < N1; q++) acc += op.dlag[i][q] * F[v][q];
      acc += -op.gL[i] * jump[0][v];
      acc += op.gR[i] * jump[1][v];
      d[i] = acc;
    }
#pragma unroll
    for (int i = 0; i < N1; i++) F[v][i] = d[i];
  }
}

// Sizes of the line kernels' blocks.
template <class C, typename R, int TE_, int NT_>
struct LineT {
  static constexpr int N1 = C::N1, NV = C::NV, DIM = C::DIM, TE = TE_;
  static constexpr int NC = DIM == 2 ? N1 : N1 * N1;  // lines per direction
  // slots per line: odd, so the lines a warp reads start on different banks (a
  // warp whose lanes read one line needs no padding)
  static constexpr int N1P = TE * (int)sizeof(R) >= 128 ? N1 : N1 | 1;
  static constexpr int NL = NC * N1P;
  static constexpr int NT = NT_;
  static constexpr int LR = (DIM * NC * TE + NT - 1) / NT;  // rounds of the line-wise phases
  static constexpr int BUF = NV * NL * TE;  // values of one direction's buffer
  static constexpr int NP = (C::NS * TE + NT - 1) / NT;  // rounds of the point-wise phases
  static constexpr int WS = (C::NF * TE * 8 + 15) & ~15;
  static constexpr int SMEM = WS + DIM * BUF * (int)sizeof(R);
};
// Slot of point (x[0], x[1], x[2]) in direction d's buffer (one field).
template <class T>
__device__ __forceinline__ int line_slot(int d, int i, int j, int k, int e) {
  const int x = d == 0 ? i : d == 1 ? j : k;
  const int l = T::DIM == 2 ? (d == 0 ? j : i) : d == 0 ? j + T::N1 * k : d == 1 ? i + T::N1 * k : i + T::N1 * j;
  return (l * T::N1P + x) * T::TE + e;
}
// A thread's line in round r of the line-wise phases.
template <class C, class T>
struct LineThread {
  int e, eg, d, c, p, q;  // line: element, direction, line number, cross coordinates
  bool act;
  __device__ __forceinline__ LineThread(const StageArgs &a, int e0, int r) {
    const int it = threadIdx.x + r * T::NT, l = it / T::TE;
    e = it - l * T::TE;
    eg = e0 + e;
    d = l / T::NC;
    c = l - d * T::NC;
    p = T::DIM == 2 ? c : c % T::N1;
    q = T::DIM == 2 ? 0 : c / T::N1;
    act = eg < a.nEle && l < T::DIM * T::NC;
  }
  __device__ __forceinline__ int fpt(int side) const { return line_fpt<C>(d, side, p, q); }
  __device__ __forceinline__ int base() const { return d * T::BUF + c * T::N1P * T::TE + e; }
};
// Round r of the point-wise phases: false where the thread has no point.
template <class T, int NS>
__device__ __forceinline__ bool line_point(const StageArgs &a, int r, int e0, int &s, int &e) {
  const int it = threadIdx.x + r * T::NT;
  s = it / T::TE;
  e = it - s * T::TE;
  return it < NS * T::TE && e0 + e < a.nEle;
}

// The RK update of one value (timeStepA/B, src/solver.cpp:307-385); base is
// the accumulator (first stage: U0).
template <class C, typename R, typename S>
__device__ __forceinline__ R line_rk_update(const StageArgs &a, R acc, R idet, double base, double u0, size_t gi,
                                            double cb, double ca, bool check) {
  const bool last = a.flags & SF_LAST;
  double accNew;
  const double unew = rk_update(a.flags, (double)(acc * idet), base, u0, cb, ca, accNew);  // acc / detJ
  if (!last && !(a.flags & SF_JAMESON)) a.Acc[gi] = accNew;
  if (last) {
    a.Uout[gi] = unew;
    if (check && isnan(unew)) atomicOr(a.err, ERRF_NAN);
    return (R)unew;
  }
  static_cast<S *>(a.Wout)[gi] = (S)unew;
  return (R)(S)unew;
}

// A point's row offset into a [field][point][element] array.
template <class C>
__device__ __forceinline__ size_t line_row(int v, int s, int ld, int eg) {
  return (size_t)(v * C::NS + s) * (unsigned)ld + eg;
}
// The stage input at a point.
template <class C, typename R, typename S>
__device__ __forceinline__ void line_load_point(const StageArgs &a, int s, int eg, R *u) {
  if (a.Uin_d) {
#pragma unroll
    for (int v = 0; v < C::NV; v++) u[v] = (R)__ldcg(a.Uin_d + line_row<C>(v, s, a.ldU, eg));
  } else {
#pragma unroll
    for (int v = 0; v < C::NV; v++) u[v] = (R)__ldcg(static_cast<const S *>(a.Uin_s) + line_row<C>(v, s, a.ldU, eg));
  }
}
// JGinv at a point.
template <class C, typename R, typename S>
__device__ __forceinline__ void line_load_jg(const StageArgs &a, int s, int eg, R G[C::DIM][C::DIM]) {
  const S *JG = static_cast<const S *>(a.JG);
#pragma unroll
  for (int d1 = 0; d1 < C::DIM; d1++)
#pragma unroll
    for (int d2 = 0; d2 < C::DIM; d2++) G[d1][d2] = (R)__ldg(JG + (size_t)((d1 * C::DIM + d2) * C::NS + s) * (unsigned)a.nE + eg);
}
// Physical to contravariant flux at a point, into the buffers.
template <class C, typename R, class T>
__device__ __forceinline__ void line_put_flux(R *B, const R F[C::DIM][C::NV], const R G[C::DIM][C::DIM], int i, int j,
                                              int k, int e) {
#pragma unroll
  for (int d1 = 0; d1 < C::DIM; d1++) {
    const int o = d1 * T::BUF + line_slot<T>(d1, i, j, k, e);
#pragma unroll
    for (int v = 0; v < C::NV; v++) {
      R t = 0;
#pragma unroll
      for (int d2 = 0; d2 < C::DIM; d2++) t += G[d1][d2] * F[d2][v];
      B[o + v * T::NL * T::TE] = t;
    }
  }
}
// One value per field at a point, into every direction's buffer.
template <class C, typename R, class T>
__device__ __forceinline__ void line_put_state(R *B, const R *u, int i, int j, int k, int e) {
#pragma unroll
  for (int d1 = 0; d1 < C::DIM; d1++) {
    const int o = d1 * T::BUF + line_slot<T>(d1, i, j, k, e);
#pragma unroll
    for (int v = 0; v < C::NV; v++) B[o + v * T::NL * T::TE] = u[v];
  }
}
template <class C, typename R, class T>
__device__ __forceinline__ void line_get(const R *Bl, R F[C::NV][C::N1]) {
#pragma unroll
  for (int v = 0; v < C::NV; v++)
#pragma unroll
    for (int i = 0; i < C::N1; i++) F[v][i] = Bl[(v * T::NL + i) * T::TE];
}
template <class C, typename R, class T>
__device__ __forceinline__ void line_set(R *Bl, const R F[C::NV][C::N1]) {
#pragma unroll
  for (int v = 0; v < C::NV; v++)
#pragma unroll
    for (int i = 0; i < C::N1; i++) Bl[(v * T::NL + i) * T::TE] = F[v][i];
}
// The end of a stage: every line's part of the divergence, the point-wise sum
// and RK update, the traces of the new state and the next step's dt.  On entry
// the buffers hold the contravariant flux.
template <class C, typename R, typename S, bool BC, int RS, int TE, class T, bool VISC>
__device__ __forceinline__ void line_stage_end(const StageArgs &a, const OpTab<R> &op, R *B, double *Ws,
                                               int e0) {
  constexpr int NF = C::NF, NV = C::NV, DIM = C::DIM, N1 = C::N1, NL = T::NL;
  const bool resid = a.flags & SF_RESIDUAL;
#pragma unroll 1
  for (int r = 0; r < T::LR; r++) {
    const LineThread<C, T> t(a, e0, r);
    if (!t.act) continue;
    LineEnd<C, R, VISC> E[2];
    line_ends_load<C, R, S>(a, E, t);
    R F[NV][N1];
    line_get<C, R, T>(B + t.base(), F);
    line_divergence<C, R, BC, RS, TE>(a, op, E, F, Ws, t.e, t.eg);
    line_set<C, R, T>(B + t.base(), F);
  }
  // the FP64 operands of the RK update, loaded ahead of the barrier
  const bool first = a.flags & (SF_FIRST | SF_JAMESON), last = a.flags & SF_LAST;
  double base[T::NP][NV], u0[T::NP][NV], dtl[T::NP];
  R idet[T::NP];
  if (!resid) {
    const double *bs = first ? a.U0 : a.Acc;
    const size_t gs = (size_t)C::NS * (unsigned)a.ldU;
#pragma unroll
    for (int r = 0; r < T::NP; r++) {
      int s, e;
      if (!line_point<T, C::NS>(a, r, e0, s, e)) continue;
      const size_t g0 = line_row<C>(0, s, a.ldU, e0 + e);
#pragma unroll
      for (int v = 0; v < NV; v++) base[r][v] = __ldcg(bs + g0 + v * gs);
      if (!first && !last) {
#pragma unroll
        for (int v = 0; v < NV; v++) u0[r][v] = __ldcg(a.U0 + g0 + v * gs);
      }
      idet[r] = (R)__ldg(static_cast<const S *>(a.invDet) + (size_t)s * (unsigned)a.nE + e0 + e);
      dtl[r] = a.grp ? a.dt[a.grp[e0 + e]] : a.dtLocal ? a.dt[e0 + e] : stage_dt(a);
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < T::NP; r++) {
    int s, e;
    if (!line_point<T, C::NS>(a, r, e0, s, e)) continue;
    const int i = s % N1, j = (s / N1) % N1, k = DIM == 3 ? s / (N1 * N1) : 0;
    const size_t g0 = line_row<C>(0, s, a.ldU, e0 + e), gs = (size_t)C::NS * (unsigned)a.ldU;
    const double cb = a.bCur * dtl[r], ca = a.aNext * dtl[r];
    int o[DIM];
#pragma unroll
    for (int d = 0; d < DIM; d++) o[d] = d * T::BUF + line_slot<T>(d, i, j, k, e);
#pragma unroll
    for (int v = 0; v < NV; v++) {
      R acc = B[o[0] + v * NL * TE];
#pragma unroll
      for (int d = 1; d < DIM; d++) acc += B[o[d] + v * NL * TE];
      if (a.flags & (SF_RESIDUAL | SF_DIVF)) a.divF[g0 + v * gs] = (double)acc;
      if (resid) continue;
      const R un = line_rk_update<C, R, S>(a, acc, idet[r], base[r][v], u0[r][v], g0 + v * gs, cb, ca, v == 0 || v == NV - 1);
#pragma unroll
      for (int d = 0; d < DIM; d++) B[o[d] + v * NL * TE] = un;
    }
  }
  if (resid) return;
  if ((a.flags & SF_TIME) && !a.grp && blockIdx.x == 0 && threadIdx.x == 0) stage_time(a, stage_dt(a));
  __syncthreads();
#pragma unroll 1
  for (int r = 0; r < T::LR; r++) {
    const LineThread<C, T> t(a, e0, r);
    if (!t.act) continue;
    S *trO = static_cast<S *>(a.trOut);
    R U[NV][N1];
    line_get<C, R, T>(B + t.base(), U);
#pragma unroll
    for (int side = 0; side < 2; side++) {
      const size_t at = (size_t)t.fpt(side) * (unsigned)a.nE + t.eg;
#pragma unroll
      for (int v = 0; v < NV; v++) {
        R x = 0;
#pragma unroll
        for (int m = 0; m < N1; m++) x += op.lag[side][m] * U[v][m];
        trO[(size_t)(v * NF) * (unsigned)a.nE + at] = (S)x;
      }
    }
  }
  if ((a.flags & SF_DTNEXT) && threadIdx.x < 32) tma_dt_reduce(a, tma_tile_dt<NF, TE>(a, Ws, e0, threadIdx.x));
}

// ----------------------------------------------------------------------------
// Inviscid RK stage / residual (Euler or scalar advection, 2D and 3D).
// ----------------------------------------------------------------------------
template <class C, typename R, typename S, bool BC, int RS, int TE, int NT, int MB>
__global__ void __launch_bounds__(NT, MB) fr_line_stage_kernel(const StageArgs a) {
  using T = LineT<C, R, TE, NT>;
  constexpr int NV = C::NV, DIM = C::DIM, N1 = C::N1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double *Ws = reinterpret_cast<double *>(smem_raw);  // [NF][TE]
  R *B = reinterpret_cast<R *>(smem_raw + T::WS);     // [DIM][NV][NL][TE]
  const OpTab<R> &op = stage_op<R>(a);
  const int e0 = blockIdx.x * TE;
  pdl_wait();
  pdl_launch_dependents();
  stage_dt_reset(a);
  R u[T::NP][NV], G[T::NP][DIM][DIM];
#pragma unroll
  for (int r = 0; r < T::NP; r++) {
    int s, e;
    if (!line_point<T, C::NS>(a, r, e0, s, e)) continue;
    line_load_point<C, R, S>(a, s, e0 + e, u[r]);
    line_load_jg<C, R, S>(a, s, e0 + e, G[r]);
  }
  // contravariant flux at the solution points (calcInviscidFlux_spts)
#pragma unroll
  for (int r = 0; r < T::NP; r++) {
    int s, e;
    if (!line_point<T, C::NS>(a, r, e0, s, e)) continue;
    R F[DIM][NV];
    inviscid_flux<DIM, NV, R>(u[r], F, a.ph);
    line_put_flux<C, R, T>(B, F, G[r], s % N1, (s / N1) % N1, DIM == 3 ? s / (N1 * N1) : 0, e);
  }
  __syncthreads();
  line_stage_end<C, R, S, BC, RS, TE, T, false>(a, op, B, Ws, e0);
}

// ----------------------------------------------------------------------------
// Viscous path (solver::calcResidual with viscous = 1, src/solver.cpp:252-291):
// a gradient pass that leaves each side's projected viscous flux, then the
// stage, which forms the gradient again (cheaper than a round trip through HBM).
// ----------------------------------------------------------------------------

// viscousFlux (src/flux.cpp:90-226) with one reciprocal of the density; the
// reference's index slips kept: tauxz = mu(du/dz + dv/dx), tauyz =
// mu(du/dz + dv/dy) (:197-198), Fvis[0][3] = -tauzz, Fvis[1][3] = -tauyz
// (:216-217).  g is the physical gradient [DIM][NV].
template <class C, typename R>
__device__ __forceinline__ void line_visc_flux(const R *U, const R *g, R Fv[C::DIM][C::NV], const Phys &ph) {
  constexpr int DIM = C::DIM, NV = C::NV;
  if constexpr (NV == 1) {
#pragma unroll
    for (int d = 0; d < DIM; d++) Fv[d][0] = -(R)ph.diffD * g[d];
  } else {
    const R rho = U[0], ir = (R)1 / rho;
    R w[DIM], vv = 0;
#pragma unroll
    for (int d = 0; d < DIM; d++) {
      w[d] = U[d + 1] * ir;
      vv += w[d] * w[d];
    }
    const R e = U[DIM + 1] * ir - (R)0.5 * vv;
    R mu = (R)ph.mu;
    if (!ph.fixVis) {  // Sutherland's law
      const R rt = ((R)ph.gamma - (R)1.0) * e / (R)ph.rt_inf;
      mu *= pow(rt, (R)1.5) * ((R)1. + (R)ph.c_sth) / (rt + (R)ph.c_sth);
    }
    const R kap = (mu / (R)ph.prandtl) * (R)ph.gamma;
    R dw[DIM][DIM], q[DIM];  // dw[a][k] = d w_k / d x_a, q = -kappa grad e
#pragma unroll
    for (int x = 0; x < DIM; x++) {
      const R *gx = g + x * NV;
      R dk = 0;
#pragma unroll
      for (int k = 0; k < DIM; k++) {
        dw[x][k] = (gx[k + 1] - gx[0] * w[k]) * ir;
        dk += w[k] * dw[x][k];
      }
      dk = (R)0.5 * vv * gx[0] + rho * dk;
      q[x] = -kap * ((gx[DIM + 1] - dk - gx[0] * e) * ir);
    }
    R diag = 0;
#pragma unroll
    for (int d = 0; d < DIM; d++) diag += dw[d][d];
    diag = diag / (R)3.0;
    R t[DIM][DIM];
#pragma unroll
    for (int d = 0; d < DIM; d++) t[d][d] = (R)2.0 * mu * (dw[d][d] - diag);
    t[0][1] = t[1][0] = mu * (dw[1][0] + dw[0][1]);
    if constexpr (DIM == 3) {
      t[0][2] = t[2][0] = mu * (dw[2][0] + dw[0][1]);
      t[1][2] = t[2][1] = mu * (dw[2][0] + dw[1][1]);
    }
#pragma unroll
    for (int d = 0; d < DIM; d++) {
      Fv[d][0] = 0;
      R en = 0;
#pragma unroll
      for (int k = 0; k < DIM; k++) {
        Fv[d][k + 1] = -t[d][k];
        en += w[k] * t[d][k];
      }
      Fv[d][DIM + 1] = q[d] - en;
    }
    if constexpr (DIM == 3) Fv[0][3] = -t[2][2];
  }
}

// Common solution minus own trace at one end (face::ldgSolution,
// src/face.cpp:583-606).
template <class C, typename R, bool BC>
__device__ __forceinline__ void line_end_ldg(const StageArgs &a, LineEnd<C, R> &L, R *dc) {
  if constexpr (BC || C::NV == 1) line_end_ghost<C, R, BC>(a, L);
  const bool right = L.code >= 0 && (L.code & 1);
  const R pf = L.code < 0 ? (R)0 : ldg_pen<C::DIM, R>(L.n, a.ph.penFact);
#pragma unroll
  for (int v = 0; v < C::NV; v++) {
    const R UL = right ? L.oth[v] : L.own[v], UR = right ? L.own[v] : L.oth[v];
    dc[v] = (R)0.5 * (UL + UR) - pf * (UL - UR) - L.own[v];
  }
}
// Corrected reference-space derivative of every field along a line, in place.
template <class C, typename R, bool BC>
__device__ __forceinline__ void line_gradient(const StageArgs &a, const OpTab<R> &op, LineEnd<C, R> *E,
                                              R U[C::NV][C::N1]) {
  constexpr int NV = C::NV, N1 = C::N1;
  R dc[2][NV];
  line_end_ldg<C, R, BC>(a, E[0], dc[0]);
  line_end_ldg<C, R, BC>(a, E[1], dc[1]);
#pragma unroll
  for (int v = 0; v < NV; v++) {
    R d[N1];
#pragma unroll
    for (int i = 0; i < N1; i++) {
      R acc = 0;
#pragma unroll
      for (int q = 0; q < N1; q++) acc += op.dlag[i][q] * U[v][q];
      acc += op.gL[i] * dc[0][v];
      acc += op.gR[i] * dc[1][v];
      d[i] = acc;
    }
#pragma unroll
    for (int i = 0; i < N1; i++) U[v][i] = d[i];
  }
}
// Reference-space gradient of the tile into the buffers: each direction's
// derivative of the state plus the correction by the common solution
// (calcGradU_spts, correctGradU src/solver.cpp:808-879).
template <class C, typename R, typename S, bool BC, class T>
__device__ __forceinline__ void line_tile_gradient(const StageArgs &a, const OpTab<R> &op, R *B,
                                                   int e0) {
  constexpr int NV = C::NV, DIM = C::DIM, N1 = C::N1;
  R u[T::NP][NV];
#pragma unroll
  for (int r = 0; r < T::NP; r++) {
    int s, e;
    if (line_point<T, C::NS>(a, r, e0, s, e)) line_load_point<C, R, S>(a, s, e0 + e, u[r]);
  }
#pragma unroll
  for (int r = 0; r < T::NP; r++) {
    int s, e;
    if (!line_point<T, C::NS>(a, r, e0, s, e)) continue;
    line_put_state<C, R, T>(B, u[r], s % N1, (s / N1) % N1, DIM == 3 ? s / (N1 * N1) : 0, e);
  }
  __syncthreads();
#pragma unroll 1
  for (int r = 0; r < T::LR; r++) {
    const LineThread<C, T> t(a, e0, r);
    if (!t.act) continue;
    LineEnd<C, R> E[2];
    line_ends_load<C, R, S>(a, E, t);
    R U[NV][N1];
    line_get<C, R, T>(B + t.base(), U);
    line_gradient<C, R, BC>(a, op, E, U);
    line_set<C, R, T>(B + t.base(), U);
  }
  __syncthreads();
}
// Physical gradient [DIM][NV] at a point from the buffers.
template <class C, typename R, typename S, class T>
__device__ __forceinline__ void line_point_gradient(const StageArgs &a, const R *B, const R G[C::DIM][C::DIM], int s,
                                                    int i, int j, int k, int e, int eg, R *g) {
  constexpr int NV = C::NV, DIM = C::DIM;
  const R idet = (R)__ldg(static_cast<const S *>(a.invDet) + (size_t)s * (unsigned)a.nE + eg);
  int o[DIM];
#pragma unroll
  for (int d = 0; d < DIM; d++) o[d] = d * T::BUF + line_slot<T>(d, i, j, k, e);
#pragma unroll
  for (int v = 0; v < NV; v++) {
    R gr[DIM];
#pragma unroll
    for (int d = 0; d < DIM; d++) gr[d] = B[o[d] + v * T::NL * T::TE];
#pragma unroll
    for (int d1 = 0; d1 < DIM; d1++) {
      R x = 0;
#pragma unroll
      for (int d2 = 0; d2 < DIM; d2++) x += gr[d2] * G[d2][d1];
      g[d1 * NV + v] = idet * x;
    }
  }
}
// This side's viscous flux at one end from its gradient trace g, projected on
// the face normal; at a boundary the whole viscous part of the boundary flux.
template <class C, typename R, typename S, bool BC>
__device__ __forceinline__ void line_end_visc(const StageArgs &a, int f, int eg, const R *g) {
  constexpr int NF = C::NF, NV = C::NV, DIM = C::DIM;
  const size_t at = (size_t)f * (unsigned)a.nE + eg, fl = (size_t)NF * (unsigned)a.nE;
  const S *tr = static_cast<const S *>(a.trIn), *nr = static_cast<const S *>(a.nrm);
  S *out = static_cast<S *>(a.fvnOut);
  R u[NV], n[DIM], Fv[DIM][NV];
  const int code = __ldg(a.nbr + at);
#pragma unroll
  for (int v = 0; v < NV; v++) u[v] = (R)__ldcg(tr + (size_t)v * fl + at);
#pragma unroll
  for (int d = 0; d < DIM; d++) n[d] = (R)__ldg(nr + (size_t)d * fl + at);
  line_visc_flux<C, R>(u, g, Fv, a.ph);
  if constexpr (BC && NV > 1) {
    if (-1 - code == BC_ADI_NOSLIP) {
      double ul[NV], ur[NV], nd[DIM];
#pragma unroll
      for (int v = 0; v < NV; v++) ul[v] = u[v];
#pragma unroll
      for (int d = 0; d < DIM; d++) nd[d] = n[d];
      bc_ghost<DIM>(-1 - code, ul, nd, ur, a.ph);
      R UR[NV], gR[DIM * NV];
#pragma unroll
      for (int v = 0; v < NV; v++) UR[v] = (R)ur[v];
      adiabatic_gradient<DIM, R>(u, UR, g, gR, a.ph);
      line_visc_flux<C, R>(UR, gR, Fv, a.ph);
    }
  }
#pragma unroll
  for (int v = 0; v < NV; v++) {
    R fn = 0;
#pragma unroll
    for (int d = 0; d < DIM; d++) fn += Fv[d][v] * n[d];
    // advection-diffusion: centralFlux with a zero ghost gradient
    if (NV == 1 && code < 0) fn *= (R)0.5;
    out[(size_t)v * fl + at] = (S)fn;
    if constexpr (DIM == 3) {
      // the LDG penalty term of the reference reads FL[1] where FL[2] is
      // meant (src/face.cpp:245): the left side contributes n0 F0 + n1 F1 + n2 F1
      if (a.visc2)
        static_cast<S *>(a.fvn2Out)[(size_t)v * fl + at] = (S)(n[0] * Fv[0][v] + n[1] * Fv[1][v] + n[2] * Fv[1][v]);
    }
  }
}

template <class C, typename R, typename S, bool BC, int TE, int NT, int MB>
__global__ void __launch_bounds__(NT, MB) fr_line_grad_kernel(const StageArgs a) {
  using T = LineT<C, R, TE, NT>;
  constexpr int NS = C::NS, NV = C::NV, DIM = C::DIM, N1 = C::N1, NL = T::NL;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  R *B = reinterpret_cast<R *>(smem_raw + T::WS);  // [DIM][NV][NL][TE]
  const OpTab<R> &op = stage_op<R>(a);
  const int e0 = blockIdx.x * TE;
  pdl_wait();
  pdl_launch_dependents();
  line_tile_gradient<C, R, S, BC, T>(a, op, B, e0);
  // physical gradient in the place of the reference-space one: d/dx_d of the
  // fields in direction d's buffer (a point's slots are read and written by its
  // own thread)
#pragma unroll
  for (int r = 0; r < T::NP; r++) {
    int s, e;
    if (!line_point<T, NS>(a, r, e0, s, e)) continue;
    const int eg = e0 + e, i = s % N1, j = (s / N1) % N1, k = DIM == 3 ? s / (N1 * N1) : 0;
    R G[DIM][DIM], g[DIM * NV];
    line_load_jg<C, R, S>(a, s, eg, G);
    line_point_gradient<C, R, S, T>(a, B, G, s, i, j, k, e, eg, g);
#pragma unroll
    for (int d = 0; d < DIM; d++) {
      const int o = d * T::BUF + line_slot<T>(d, i, j, k, e);
#pragma unroll
      for (int v = 0; v < NV; v++) B[o + v * NL * TE] = g[d * NV + v];
    }
    if (a.dUg) {
#pragma unroll
      for (int m = 0; m < DIM * NV; m++)
        static_cast<S *>(a.dUg)[(size_t)(m * NS + s) * (unsigned)a.nE + eg] = (S)g[m];
    }
  }
  __syncthreads();
#pragma unroll 1
  for (int r = 0; r < T::LR; r++) {
    const LineThread<C, T> t(a, e0, r);
    if (!t.act) continue;
    // gradient traces at both ends of the line, through every buffer
    R gt[2][DIM * NV];
#pragma unroll
    for (int d = 0; d < DIM; d++) {
      // the line's first point and step in direction d's layout
      const int x0[3] = {t.d == 0 ? 0 : t.p, DIM == 2 ? (t.d == 0 ? t.p : 0) : t.d == 0 ? t.p : t.d == 1 ? 0 : t.q,
                         DIM == 3 && t.d != 2 ? t.q : 0};
      const int x1[3] = {x0[0] + (t.d == 0), x0[1] + (t.d == 1), x0[2] + (t.d == 2)};
      const int o = line_slot<T>(d, x0[0], x0[1], x0[2], t.e), st = line_slot<T>(d, x1[0], x1[1], x1[2], t.e) - o;
#pragma unroll
      for (int v = 0; v < NV; v++) {
        const R *x = B + d * T::BUF + v * NL * TE + o;
        R lo = 0, hi = 0;
#pragma unroll
        for (int i = 0; i < N1; i++) {
          const R y = x[i * st];
          lo += op.lag[0][i] * y;
          hi += op.lag[1][i] * y;
        }
        gt[0][d * NV + v] = lo;
        gt[1][d * NV + v] = hi;
      }
    }
    line_end_visc<C, R, S, BC>(a, t.fpt(0), t.eg, gt[0]);
    line_end_visc<C, R, S, BC>(a, t.fpt(1), t.eg, gt[1]);
  }
}

template <class C, typename R, typename S, bool BC, int RS, int TE, int NT, int MB>
__global__ void __launch_bounds__(NT, MB)
    fr_line_visc_stage_kernel(const StageArgs a) {
  using T = LineT<C, R, TE, NT>;
  constexpr int NS = C::NS, NV = C::NV, DIM = C::DIM, N1 = C::N1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double *Ws = reinterpret_cast<double *>(smem_raw);
  R *B = reinterpret_cast<R *>(smem_raw + T::WS);  // [DIM][NV][NL][TE]
  const OpTab<R> &op = stage_op<R>(a);
  const int e0 = blockIdx.x * TE;
  pdl_wait();
  pdl_launch_dependents();
  stage_dt_reset(a);
  line_tile_gradient<C, R, S, BC, T>(a, op, B, e0);
  // inviscid + viscous flux at the solution points, transformed
  // (calcInviscidFlux_spts, calcViscousFlux_spts src/solver.cpp:562-596), over
  // the gradient
#pragma unroll
  for (int r = 0; r < T::NP; r++) {
    int s, e;
    if (!line_point<T, NS>(a, r, e0, s, e)) continue;
    const int eg = e0 + e, i = s % N1, j = (s / N1) % N1, k = DIM == 3 ? s / (N1 * N1) : 0;
    R u[NV], G[DIM][DIM], g[DIM * NV], F[DIM][NV], Fv[DIM][NV];
    line_load_point<C, R, S>(a, s, eg, u);
    line_load_jg<C, R, S>(a, s, eg, G);
    line_point_gradient<C, R, S, T>(a, B, G, s, i, j, k, e, eg, g);
    inviscid_flux<DIM, NV, R>(u, F, a.ph);
    line_visc_flux<C, R>(u, g, Fv, a.ph);
#pragma unroll
    for (int d = 0; d < DIM; d++)
#pragma unroll
      for (int v = 0; v < NV; v++) F[d][v] += Fv[d][v];
    line_put_flux<C, R, T>(B, F, G, i, j, k, e);
  }
  __syncthreads();
  line_stage_end<C, R, S, BC, RS, TE, T, true>(a, op, B, Ws, e0);
}

}  // namespace frg
