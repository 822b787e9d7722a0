// bx_stage3d.cu -- dispatch of the 3D stage kernels, and the instantiations
// of the one that runs one direction at a time (bx_stage3d.cuh).  FP64 mode:
// FP64 tile, fluxes and update.  FP32-bulk mode: stage 1 reads the FP64
// state and writes an FP32 intermediate state, stage 2 reads that FP32 state
// and writes FP64; the reconstruction and fluxes run in FP32, the
// conserved-state update and the pressure recovery in FP64.
#include "bx_stage3d_launch.cuh"
#include "bx_stage8_launch.cuh"
#include "bx_stage_unit_launch.cuh"

namespace bx {

bool stage3d_units(int shape, int flux) {
  return shape == kShape444 || (flux != kFluxRoe && tune_value(kTuneStageVariant) == 0);
}

namespace {

template <int FLUX>
cudaError_t launch_blocks(int shape, int kind, const TmaMaps &maps, const StageArgs &a, int nSM, cudaStream_t st) {
  // the implicit residual, whose finite-difference products amplify
  // rounding, keeps the reference's order of operations (flux_lean)
  if (shape == kShape888 && (a.outputResidual || !stage3d_units(shape, FLUX)))
    return launch_stage8<FLUX>(kind, maps, a, nSM, st);
  if (a.outputResidual) return launch_one<4, 1, double, double, double, FLUX>(maps, a, nSM, st);
  return launch_unit<FLUX>(shape, kind, maps, a, nSM, st);
}

}  // namespace

cudaError_t launch_stage3d(int shape, int flux, int kind, const TmaMaps &maps, const StageArgs &a, int nSM,
                           cudaStream_t st) {
  const int variant = shape == kShape888 ? tune_value(kTuneStageVariant) : 0;
  if (variant == 1) return launch_kind<8, 1>(flux, kind, maps, a, nSM, st);
  if (variant == 2) return launch_stage3d_fpt2(flux, kind, maps, a, nSM, st);
  switch (flux) {
    case kFluxRusanov: return launch_blocks<kFluxRusanov>(shape, kind, maps, a, nSM, st);
    case kFluxLinde: return launch_blocks<kFluxLinde>(shape, kind, maps, a, nSM, st);
    case kFluxHlld: return launch_blocks<kFluxHlld>(shape, kind, maps, a, nSM, st);
    case kFluxRoe: return launch_blocks<kFluxRoe>(shape, kind, maps, a, nSM, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace bx
