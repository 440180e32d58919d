// stage_impl.cuh -- launchers and the instantiation switch shared by the
// per-configuration translation units.  Include once per unit after defining
// FRG_UNIT_DIM (2 or 3), FRG_UNIT_R / FRG_UNIT_S (arithmetic / stored type)
// and FRG_UNIT_NAME (suffix of the exported functions).
#pragma once
#include "dispatch.h"
#include "kernels.cuh"
#include "kernels_line.cuh"
#include "kernels_tma.cuh"
#include "optab_upload.cuh"

namespace frg {
namespace {

// A TMA stage kernel's launch; with SF_PDL it is a programmatic dependent of
// the previous kernel in the stream (its blocks may start while that kernel's
// last blocks run, see pdl_wait).
template <class K>
void launch_tma_stage(K kernel, const void *args, const void *maps, int nBlk, int nt, size_t smem, cudaStream_t st) {
  const StageArgs &a = *static_cast<const StageArgs *>(args);
  const TmaMaps &m = *static_cast<const TmaMaps *>(maps);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(nBlk);
  cfg.blockDim = dim3(nt);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = (a.flags & SF_PDL) ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, a, m);
}
template <class C, typename R, typename S, bool BC, int RS, int TEV, int NTV>
void launch_stage_tma(const void *args, const void *maps, int nBlk, size_t smem, cudaStream_t st) {
  launch_tma_stage(fr_stage_tma_kernel<C, R, S, BC, RS, TEV, NTV>, args, maps, nBlk, NTV, smem, st);
}
template <class C, typename R, typename S, bool BC, int RS, int TEV, int NTV>
cudaError_t add_tma_variant(KernelSet &k) {
  using TT = TileT<C, R, S, TEV, NTV>;
  if (k.nTma >= KernelSet::kMaxTma) return cudaErrorInvalidValue;  // the variant table is full
  KernelSet::TmaVariant &v = k.tma[k.nTma++];
  v.launch = &launch_stage_tma<C, R, S, BC, RS, TEV, NTV>;
  v.TE = TT::TE;
  v.NT = NTV;
  v.smem = TT::SMEM;
  auto ft = fr_stage_tma_kernel<C, R, S, BC, RS, TEV, NTV>;
  cudaError_t e = cudaFuncSetAttribute(ft, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TT::SMEM);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(ft, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
  return e;
}
template <class C, typename R, typename S, bool BC, int RS, int TEV, int NTV, int NB>
void launch_stage_pipe(const void *args, const void *maps, int nBlk, size_t smem, cudaStream_t st) {
  launch_tma_stage(fr_stage_tma_pipe_kernel<C, R, S, BC, RS, TEV, NTV, NB>, args, maps, nBlk, NTV, smem, st);
}
template <class C, typename R, typename S, bool BC, int RS, int TEV, int NTV, int NB>
cudaError_t add_pipe_variant(KernelSet &k) {
  using TT = PipeT<C, R, S, TEV, NTV, NB>;
  if (k.nTma >= KernelSet::kMaxTma) return cudaErrorInvalidValue;  // the variant table is full
  KernelSet::TmaVariant &v = k.tma[k.nTma++];
  v.launch = &launch_stage_pipe<C, R, S, BC, RS, TEV, NTV, NB>;
  v.TE = TT::TE;
  v.NT = NTV;
  v.smem = TT::SMEM;
  v.persistent = 1;
  auto ft = fr_stage_tma_pipe_kernel<C, R, S, BC, RS, TEV, NTV, NB>;
  cudaError_t e = cudaFuncSetAttribute(ft, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TT::SMEM);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(ft, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v.occ, ft, NTV, TT::SMEM);
  if (e == cudaSuccess && v.occ < 1) e = cudaErrorInvalidConfiguration;
  return e;
}
template <class C, typename R, typename S, bool BC, int RS, int TEV, int NTV>
void launch_stage_split(const void *args, const void *maps, int nBlk, size_t smem, cudaStream_t st) {
  launch_tma_stage(fr_stage_tma_split_kernel<C, R, S, BC, RS, TEV, NTV>, args, maps, nBlk, NTV, smem, st);
}
template <class C, typename R, typename S, bool BC, int RS, int TEV, int NTV>
cudaError_t add_split_variant(KernelSet &k) {
  using TT = SplitT<C, R, S, TEV, NTV>;
  if (k.nTma >= KernelSet::kMaxTma) return cudaErrorInvalidValue;  // the variant table is full
  KernelSet::TmaVariant &v = k.tma[k.nTma++];
  v.launch = &launch_stage_split<C, R, S, BC, RS, TEV, NTV>;
  v.TE = TT::TE;
  v.NT = NTV;
  v.smem = TT::SMEM;
  v.persistent = 1;
  auto ft = fr_stage_tma_split_kernel<C, R, S, BC, RS, TEV, NTV>;
  cudaError_t e = cudaFuncSetAttribute(ft, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TT::SMEM);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(ft, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v.occ, ft, NTV, TT::SMEM);
  if (e == cudaSuccess && v.occ < 1) e = cudaErrorInvalidConfiguration;
  return e;
}
template <class C, typename R, typename S>
void launch_trace(const double *U, void *tr, int nE, int nEle, int ldU, int vcjh, cudaStream_t st) {
  long n = (long)C::NF * nE;
  fr_trace_kernel<C, R, S><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(U, static_cast<S *>(tr), nE, nEle, ldU,
                                                                         vcjh);
}
template <class C, typename R, typename S>
void launch_import(const double *ref, double *U, void *tr, int nEle, int L, int vcjh, cudaStream_t st) {
  fr_import_kernel<C, R, S><<<dim3((nEle + 127) / 128, C::NS + C::NF), 128, 0, st>>>(ref, U, static_cast<S *>(tr), nEle,
                                                                                   L, vcjh);
}
template <int DIM, int NV, typename S>
void launch_wavesp(const void *tr, const double *nrmOwn, double *ws, int NF, int nE, const Phys &ph, cudaStream_t st) {
  long n = (long)NF * nE;
  fr_wavesp_kernel<DIM, NV, S><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(static_cast<const S *>(tr), nrmOwn, ws,
                                                                             NF, nE, ph);
}

// A line kernel's launch; with SF_PDL a programmatic dependent of the previous
// kernel in the stream (see pdl_wait).
template <class K>
void launch_line(K kernel, const StageArgs &a, int nBlk, int nt, size_t smem, cudaStream_t st) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(nBlk);
  cfg.blockDim = dim3(nt);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = (a.flags & SF_PDL) ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, a);
}
template <class C, typename R, typename S, bool BC, int RS, int TE, int NT, int MB, bool VISC>
void launch_line_stage(const void *args, int nBlk, size_t smem, cudaStream_t st) {
  const StageArgs &a = *static_cast<const StageArgs *>(args);
  if constexpr (VISC) launch_line(fr_line_visc_stage_kernel<C, R, S, BC, RS, TE, NT, MB>, a, nBlk, NT, smem, st);
  else launch_line(fr_line_stage_kernel<C, R, S, BC, RS, TE, NT, MB>, a, nBlk, NT, smem, st);
}
template <class C, typename R, typename S, bool BC, int TE, int NT, int MB>
void launch_line_grad(const void *args, int nBlk, size_t smem, cudaStream_t st) {
  launch_line(fr_line_grad_kernel<C, R, S, BC, TE, NT, MB>, *static_cast<const StageArgs *>(args), nBlk, NT,
              smem, st);
}
template <class K>
cudaError_t prepare_kernel(K f, size_t smem) {
  cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
  return e;
}
template <class C, typename R, typename S, bool BC, int RS, bool VISC, int TE, int NT, int MB>
cudaError_t add_line(KernelSet &k) {
  using T = LineT<C, R, TE, NT>;
  static_assert(NT % 32 == 0 && NT <= 1024 && T::SMEM <= 227 * 1024, "block shape");
  KernelSet::LineVariant &v = k.line[k.nLine++];
  v.stage = &launch_line_stage<C, R, S, BC, RS, TE, NT, MB, VISC>;
  v.TE = TE;
  v.rounds = T::LR;
  v.smem = T::SMEM;
  if constexpr (VISC) {
    v.grad = &launch_line_grad<C, R, S, BC, TE, NT, MB>;
    const cudaError_t e = prepare_kernel(fr_line_grad_kernel<C, R, S, BC, TE, NT, MB>, T::SMEM);
    return e == cudaSuccess ? prepare_kernel(fr_line_visc_stage_kernel<C, R, S, BC, RS, TE, NT, MB>, T::SMEM) : e;
  } else {
    return prepare_kernel(fr_line_stage_kernel<C, R, S, BC, RS, TE, NT, MB>, T::SMEM);
  }
}
// The line kernel among the tile shapes of the 2D inviscid update (it takes no
// tensor maps).
template <class C, typename R, typename S, bool BC, int RS, int TE, int NT, int MB>
void launch_line_tile(const void *args, const void *, int nBlk, size_t smem, cudaStream_t st) {
  launch_line(fr_line_stage_kernel<C, R, S, BC, RS, TE, NT, MB>, *static_cast<const StageArgs *>(args), nBlk, NT, smem,
              st);
}
template <class C, typename R, typename S, bool BC, int RS, int TE, int NT, int MB>
cudaError_t add_line_tile(KernelSet &k) {
  if (k.nTma >= KernelSet::kMaxTma) return cudaErrorInvalidValue;  // the variant table is full
  using T = LineT<C, R, TE, NT>;
  KernelSet::TmaVariant &v = k.tma[k.nTma++];
  v.launch = &launch_line_tile<C, R, S, BC, RS, TE, NT, MB>;
  v.TE = TE;
  v.NT = NT;
  v.smem = T::SMEM;
  auto f = fr_line_stage_kernel<C, R, S, BC, RS, TE, NT, MB>;
  const cudaError_t e = prepare_kernel(f, T::SMEM);
  return e == cudaSuccess ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v.occ, f, NT, T::SMEM) : e;
}
// Block shapes of a configuration (elements and threads per block, resident
// blocks per SM), in the order pick_line tries them.  The first is for meshes that
// fill the GPU several times: elements as many as keep a warp's accesses whole
// 128-byte lines where shared memory allows it, threads as many as leave the FP64
// (FP32) line phase its ~168 (~80) registers, the lines taken in rounds.  Per step
// of 24,273 (P = 4: 8,000, P = 2: 21,952) periodic hexes, inviscid, us:
//   P = 2 FP32  32 x 288 x 2: 239   32 x 864: 257   16 x 448 x 2: 260
//   P = 2 FP64  16 x 224 x 2: 359   32 x 448: 374   32 x 864: 437
//   P = 3 FP32  32 x 768: 572   16 x 384 x 2: 587   16 x 768: 723   8 x 384 x 2: 799
//   P = 3 FP64  16 x 384: 882   16 x 256 x 2: 1160  16 x 768: 1214  8 x 384: 1271
//   P = 4 FP32  16 x 608: 443   8 x 320 x 2: 490    8 x 608: 531
//   P = 4 FP64  8 x 320: 716    8 x 608: 775 (viscous: 1491 and 1389)
// The others have a thread for every line of the tile, which is faster where each
// SM gets one block or none (1,287 hexes, P = 2, FP64, viscous: 16 x 448: 116,
// 16 x 224: 176), and the last is the narrowest, for meshes too small to give every
// other SM a wider tile (216 hexes, P = 3, FP64: 4 x 192: 40, 8 x 384: 45,
// 16 x 384: 76).  Viscous passes on such meshes are a chain of point-wise and
// line-wise phases, so their narrowest shapes have a thread for every point too
// (48 / 294 hexes: P = 3 FP64 4 x 192: 80.5 / 89.1, 4 x 256: 76.0 / 83.1; FP32 71.9 /
// 81.6, 65.3 / 74.2; P = 4 FP32 4 x 320: 100 / 112, 4 x 512: 95 / 108; FP64 4 x 320:
// 130.7 / 142.3, 2 x 256: 108.0 / 116.1, but 448 hexes, 1.5 blocks of 2 elements to an
// SM, 148 against 226; 900 hexes, P = 3 FP32: 16 x 768: 105, 8 x 512: 80, 4 x 256: 110).
// P = 1 FP64, inviscid, 31,744 / 83,248 hexes: 16 x 192 x 2: 230 / 596, 32 x 192 x 2:
// 205 / 494 (a residual 51.9 / 130, 45.8 / 110).
struct LineShape {
  int TE, NT, MB;
};
template <class C, typename R, bool VISC>
constexpr LineShape line_shape(int tier) {
  constexpr bool f32 = sizeof(R) == 4;
  constexpr int n = 2 * C::N1;  // 2D: lines per element
  constexpr LineShape none{0, 0, 0};
  using Shapes = LineShape[KernelSet::kMaxLine];
  constexpr Shapes two = {{32, 32 * n, (f32 ? 768 : 384) / (32 * n)}, {8, (8 * n + 31) & ~31, 1}, none, none};
  constexpr LineShape p1w = f32 ? LineShape{32, 384, 2} : LineShape{16, 192, 2}, p1n = {8, 96, 1};
  constexpr bool wide1 = !f32 && !VISC;
  constexpr Shapes p1 = {wide1 ? LineShape{32, 192, 2} : p1w, wide1 ? p1w : p1n, wide1 ? p1n : none, none};
  constexpr Shapes p2 = {f32 ? LineShape{32, 288, 2} : LineShape{16, 224, 2}, {16, 448, 1}, {8, 224, 1}, none};
  constexpr LineShape p3n = {4, VISC ? 256 : 192, 1};
  constexpr Shapes p3 = {f32 ? LineShape{32, 768, 1} : LineShape{16, 384, 1},
                         f32 ? LineShape{16, 768, 1} : LineShape{8, 384, 1},
                         VISC && f32 ? LineShape{8, 512, 1} : p3n, VISC && f32 ? p3n : none};
  constexpr Shapes p4 = {f32 ? LineShape{16, 608, 1} : LineShape{8, VISC ? 608 : 320, 1}, {8, 608, 1},
                         {4, VISC && f32 ? 512 : 320, 1}, VISC && !f32 ? LineShape{2, 256, 1} : none};
  return C::DIM == 2 ? two[tier] : C::P == 1 ? p1[tier] : C::P == 2 ? p2[tier] : C::P == 3 ? p3[tier] : p4[tier];
}
template <class C, typename R, typename S, bool BC, int RS, bool VISC, int TIER = 0>
cudaError_t add_lines(KernelSet &k) {
  if constexpr (TIER < KernelSet::kMaxLine) {
    constexpr LineShape sh = line_shape<C, R, VISC>(TIER);
    if constexpr (sh.TE > 0) {
      const cudaError_t e = add_line<C, R, S, BC, RS, VISC, sh.TE, sh.NT, (sh.MB > 1 ? sh.MB : 1)>(k);
      return e == cudaSuccess ? add_lines<C, R, S, BC, RS, VISC, TIER + 1>(k) : e;
    }
  }
  return cudaSuccess;
}
template <class C, typename R, typename S, bool BC, int RS, bool VISC>
bool make_set(KernelSet &k, std::string &err) {
  k.trace = &launch_trace<C, R, S>;
  k.import = &launch_import<C, R, S>;
  k.wavesp = &launch_wavesp<C::DIM, C::NV, S>;
  k.nLine = 0;
  cudaError_t e = add_lines<C, R, S, BC, RS, VISC>(k);
  if (e == cudaSuccess) {
    // load the trace kernel now (lazy module loading would otherwise load it
    // at its first launch, e.g. inside frg_calc_residual_noalloc)
    cudaFuncAttributes fa;
    e = cudaFuncGetAttributes(&fa, fr_trace_kernel<C, R, S>);
  }
  if constexpr (C::DIM == 2 && !VISC) {
    // the shapes frg_autotune tries and pick_tile chooses from, in the order of
    // KernelSet's tile names
    k.nTma = 0;
    if (e == cudaSuccess) e = add_tma_variant<C, R, S, BC, RS, 0, 128>(k);
    if (e == cudaSuccess) e = add_tma_variant<C, R, S, BC, RS, 0, 256>(k);
    if (e == cudaSuccess) e = add_tma_variant<C, R, S, BC, RS, -1, 128>(k);
    if (e == cudaSuccess) e = add_tma_variant<C, R, S, BC, RS, -1, 64>(k);
    if (e == cudaSuccess) e = add_tma_variant<C, R, S, BC, RS, -2, 64>(k);
    // a thread per line, loads straight to registers: FP32 a thread for every
    // line of 32 elements, FP64 half as many
    constexpr int n = 2 * C::N1;
    constexpr bool f32 = sizeof(R) == 4;
    constexpr int NT = f32 ? 32 * n : 16 * n, MB = f32 ? (C::P < 4 ? 1024 : 768) / NT : 384 / NT;
    if (e == cudaSuccess) e = add_line_tile<C, R, S, BC, RS, 32, NT, (MB > 1 ? MB : 1)>(k);
    // persistent, ring-buffered variants
    if (e == cudaSuccess) e = add_pipe_variant<C, R, S, BC, RS, 0, 160, 2>(k);
    if (e == cudaSuccess) e = add_pipe_variant<C, R, S, BC, RS, 0, 160, 3>(k);
    if (e == cudaSuccess) e = add_pipe_variant<C, R, S, BC, RS, 0, 256, 2>(k);
    if (e == cudaSuccess) e = add_pipe_variant<C, R, S, BC, RS, 0, 128, 2>(k);
    // persistent, FP64 buffers outside the ring (four blocks per SM)
    if (e == cudaSuccess) e = add_split_variant<C, R, S, BC, RS, 0, 160>(k);
    if (e == cudaSuccess) e = add_split_variant<C, R, S, BC, RS, 0, 128>(k);
  }
  if (e != cudaSuccess) { err = std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e); return false; }
  return true;
}

template <class C, typename R, typename S, bool BC, int RS>
bool make_one(const KernelKey &key, KernelSet &k, std::string &err) {
  return key.viscous ? make_set<C, R, S, BC, RS, true>(k, err) : make_set<C, R, S, BC, RS, false>(k, err);
}

template <int DIM, int P, int NV, typename R, typename S>
bool make_variant(const KernelKey &key, KernelSet &k, std::string &err) {
  using C = Cfg<DIM, P, NV>;
  if constexpr (NV == 1 || DIM == 3) {
    return key.bc ? make_one<C, R, S, true, 0>(key, k, err) : make_one<C, R, S, false, 0>(key, k, err);
  } else {
    if (key.riemann == 1)
      return key.bc ? make_one<C, R, S, true, 1>(key, k, err) : make_one<C, R, S, false, 1>(key, k, err);
    return key.bc ? make_one<C, R, S, true, 0>(key, k, err) : make_one<C, R, S, false, 0>(key, k, err);
  }
}

template <int DIM, int NV, typename R, typename S>
bool select_order(const KernelKey &key, KernelSet &k, std::string &err) {
  switch (key.P) {
    case 1: return make_variant<DIM, 1, NV, R, S>(key, k, err);
    case 2: return make_variant<DIM, 2, NV, R, S>(key, k, err);
    case 3: return make_variant<DIM, 3, NV, R, S>(key, k, err);
    case 4: return make_variant<DIM, 4, NV, R, S>(key, k, err);
    case 5:
      if constexpr (DIM == 2) return make_variant<DIM, 5, NV, R, S>(key, k, err);
      break;
  }
  err = "order not available for this dimension (2D: 1..5, 3D: 1..4)";
  return false;
}

}  // namespace
}  // namespace frg

#define FRG_CAT2(a, b) a##b
#define FRG_CAT(a, b) FRG_CAT2(a, b)

namespace frg {
bool FRG_CAT(select_, FRG_UNIT_NAME)(const KernelKey &key, KernelSet &k, std::string &err) {
  using R = FRG_UNIT_R;
  using S = FRG_UNIT_S;
  if (key.NV == 1) return select_order<FRG_UNIT_DIM, 1, R, S>(key, k, err);
  if (key.NV == FRG_UNIT_DIM + 2) return select_order<FRG_UNIT_DIM, FRG_UNIT_DIM + 2, R, S>(key, k, err);
  err = "unsupported field count";
  return false;
}
cudaError_t FRG_CAT(upload_tables_, FRG_UNIT_NAME)() { return upload_tables_impl(); }
}  // namespace frg
