// bx_stage8_launch.cuh -- launcher templates of the single-face-phase stage
// kernel for 8^3 blocks (bx_stage3d_v2.cuh): grids with resolution changes
// (stage3d_units), the Roe flux, the residual of the implicit step and
// stage_variant 3; one translation unit per flux instantiates them (bx_stage8_*.cu).  Roe's long
// face code runs better here, with one set of barriers per block and 128
// registers (96^3: 665 us per FP64 step and 368 per FP32-bulk step, against
// 800 and 420 in units of 128 cells).
#pragma once
#include "bx_stage3d_v2.cuh"
#include "bx_tune.h"

namespace bx {

// one flux (instantiated in bx_stage8_*.cu)
template <int FLUX>
cudaError_t launch_stage8(int kind, const TmaMaps &maps, const StageArgs &a, int nSM, cudaStream_t st);

#ifdef BX_STAGE8_INSTANTIATE
template <int NTHR, int MINB, typename TileT, typename Real, typename OutT, int FLUX, int LIM, bool RC>
static cudaError_t launch8_rc(const TmaMaps &maps, const StageArgs &a, int nSM, cudaStream_t st) {
  using B = Blk8<TileT, Real, NTHR, MINB>;
  auto k = stage8_kernel<B, TileT, Real, OutT, FLUX, LIM, RC>;
  constexpr size_t sm = B::smem_bytes;
  static bool attr = false;
  if (!attr) {
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    attr = true;
  }
  // persistent grid of MINB CTAs per SM (what the shared memory and the
  // registers of the instantiation hold together)
  const int want = nSM * MINB;
  const int grid = a.nBlock < want ? a.nBlock : want;
  k<<<grid, NTHR, sm, st>>>(maps, a);
  return cudaGetLastError();
}

// without the resolution-change face code where no block needs it
template <int NTHR, int MINB, typename TileT, typename Real, typename OutT, int FLUX, int LIM>
static cudaError_t launch8_lim(const TmaMaps &maps, const StageArgs &a, int nSM, cudaStream_t st) {
  if (a.anySpecial) return launch8_rc<NTHR, MINB, TileT, Real, OutT, FLUX, LIM, true>(maps, a, nSM, st);
  return launch8_rc<NTHR, MINB, TileT, Real, OutT, FLUX, LIM, false>(maps, a, nSM, st);
}

template <int NTHR, int MINB, typename TileT, typename Real, typename OutT, int FLUX>
static cudaError_t launch8_flux(const TmaMaps &maps, const StageArgs &a, int nSM, cudaStream_t st) {
  switch (a.limiter) {
    case kLimMinmod: return launch8_lim<NTHR, MINB, TileT, Real, OutT, FLUX, kLimMinmod>(maps, a, nSM, st);
    case kLimMc: return launch8_lim<NTHR, MINB, TileT, Real, OutT, FLUX, kLimMc>(maps, a, nSM, st);
    case kLimMc3: return launch8_lim<NTHR, MINB, TileT, Real, OutT, FLUX, kLimMc3>(maps, a, nSM, st);
  }
  return cudaErrorInvalidValue;
}

template <int FLUX>
cudaError_t launch_stage8(int kind, const TmaMaps &maps, const StageArgs &a, int nSM, cudaStream_t st) {
  // FP64: one CTA per SM (the FP64 tile and face slots fill the shared
  // memory) of 512 threads, or 576 (three face groups per warp, 96 registers)
  // with stage_variant 3 and on grids with resolution changes (us per step,
  // 8^3 roots and three levels: HLLD 1498 against 2180, Linde 1249 against
  // 1696).  FP32-bulk: one CTA of 512 per SM or, for stage_ctas_per_sm >= 2,
  // two CTAs of 256, each on its own block
  const bool two = tune_value(kTuneStageGrid) >= 2;
  switch (kind) {
    case kKindFp64:
      if (tune_value(kTuneStageVariant) == 3 || (FLUX != kFluxRoe && a.nRcBlock > 0))
        return launch8_flux<576, 1, double, double, double, FLUX>(maps, a, nSM, st);
      return launch8_flux<512, 1, double, double, double, FLUX>(maps, a, nSM, st);
    case kKindFp32In64:
      if (two) return launch8_flux<256, 2, double, float, float, FLUX>(maps, a, nSM, st);
      return launch8_flux<512, 1, double, float, float, FLUX>(maps, a, nSM, st);
    case kKindFp32In32:
      if (two) return launch8_flux<256, 2, float, float, double, FLUX>(maps, a, nSM, st);
      return launch8_flux<512, 1, float, float, double, FLUX>(maps, a, nSM, st);
  }
  return cudaErrorInvalidValue;
}
#endif  // BX_STAGE8_INSTANTIATE

}  // namespace bx
