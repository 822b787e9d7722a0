// bx_stage_unit_launch.cuh -- launcher templates of the explicit 3D stage
// kernel (bx_stage_unit.cuh); one translation unit per flux instantiates them
// (bx_stage_unit_*.cu).
#pragma once
#include "bx_stage_unit.cuh"
#include "bx_tune.h"

namespace bx {

// block size 8 or 4, one flux (instantiated in bx_stage_unit_*.cu)
template <int FLUX>
cudaError_t launch_unit(int shape, int kind, const TmaMaps &maps, const StageArgs &a, int nSM, cudaStream_t st);

#ifdef BX_UNIT_INSTANTIATE
template <int N, int MINB, typename TileT, typename Real, typename OutT, int FLUX, int LIM, bool RC>
static cudaError_t launch_unit_rc(const TmaMaps &maps, const StageArgs &a, int nSM, cudaStream_t st) {
  using W = Unit<N, TileT, Real, MINB>;
  auto k = stage_unit_kernel<W, TileT, Real, OutT, FLUX, LIM, RC>;
  constexpr size_t sm = W::smem_bytes;
  static int fit = 0;
  if (!fit) {
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    int n = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, W::NTHR, sm);
    if (e != cudaSuccess) return e;
    fit = n < 1 ? 1 : n;
  }
  // persistent grid: the CTAs of an SM that are resident together, at most
  // the knob's
  const int perSM = tune_value(kTuneStageGrid) < fit ? tune_value(kTuneStageGrid) : fit;
  const int nUnit = N == 8 ? W::PARTS * a.nBlock : (a.nBlock + W::NT - 1) / W::NT;
  const int want = nSM * perSM;
  k<<<nUnit < want ? nUnit : want, W::NTHR, sm, st>>>(maps, a);
  return cudaGetLastError();
}

// without the resolution-change code where no block needs it
template <int N, int MINB, typename TileT, typename Real, typename OutT, int FLUX, int LIM>
static cudaError_t launch_unit_lim(const TmaMaps &maps, const StageArgs &a, int nSM, cudaStream_t st) {
  if (a.anySpecial) return launch_unit_rc<N, MINB, TileT, Real, OutT, FLUX, LIM, true>(maps, a, nSM, st);
  return launch_unit_rc<N, MINB, TileT, Real, OutT, FLUX, LIM, false>(maps, a, nSM, st);
}

template <int N, int MINB, typename TileT, typename Real, typename OutT, int FLUX>
static cudaError_t launch_unit_t(const TmaMaps &maps, const StageArgs &a, int nSM, cudaStream_t st) {
  switch (a.limiter) {
    case kLimMinmod: return launch_unit_lim<N, MINB, TileT, Real, OutT, FLUX, kLimMinmod>(maps, a, nSM, st);
    case kLimMc: return launch_unit_lim<N, MINB, TileT, Real, OutT, FLUX, kLimMc>(maps, a, nSM, st);
    case kLimMc3: return launch_unit_lim<N, MINB, TileT, Real, OutT, FLUX, kLimMc3>(maps, a, nSM, st);
  }
  return cudaErrorInvalidValue;
}

// MINB64, MINB32: CTAs per SM that the register limit allows for
template <int N, int MINB64, int MINB32, int FLUX>
static cudaError_t launch_unit_kind(int kind, const TmaMaps &maps, const StageArgs &a, int nSM, cudaStream_t st) {
  switch (kind) {
    case kKindFp64: return launch_unit_t<N, MINB64, double, double, double, FLUX>(maps, a, nSM, st);
    case kKindFp32In64: return launch_unit_t<N, MINB32, double, float, float, FLUX>(maps, a, nSM, st);
    case kKindFp32In32: return launch_unit_t<N, MINB32, float, float, double, FLUX>(maps, a, nSM, st);
  }
  return cudaErrorInvalidValue;
}

template <int FLUX>
cudaError_t launch_unit(int shape, int kind, const TmaMaps &maps, const StageArgs &a, int nSM, cudaStream_t st) {
  // CTAs per SM: 3 of 128 registers in FP64, 4 of 96 in FP32 (160^3 Linde:
  // FP64 1286 us per step, 1460 with 2; FP32-bulk 748, 815 with 3 and 812 with 5)
  if (shape == kShape444) return launch_unit_kind<4, 3, 4, FLUX>(kind, maps, a, nSM, st);
  if constexpr (FLUX == kFluxRoe) return cudaErrorInvalidValue;  // launch_stage8
  else return launch_unit_kind<8, 3, 4, FLUX>(kind, maps, a, nSM, st);
}
#endif  // BX_UNIT_INSTANTIATE

}  // namespace bx
