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

// 8^3 blocks in units or whole (bx_stage8_launch.cuh).  Uniform grids gain by
// units with Rusanov, Linde and HLLD (160^3 Linde, us per step: FP64 1238 against
// 1694, FP32-bulk 756 against 789).  With resolution changes the faces of
// their blocks take a long branch, which costs more among the three or four
// CTAs of an SM than in one set of barriers per block (refined blasts, us per
// step in units / whole, s the share of blocks at a resolution change):
//   FP64 (whole: 576 threads)    HLLD        Linde       Rusanov
//     14^3 roots, s = 0.07     770 / 944   724 / 850   595 / 693
//      9^3 roots, s = 0.21     328 / 352   304 / 302   256 / 246
//     14^3 roots, s = 0.31    1462 / 1420 1356 / 1229 1123 / 1023
//      8^3 roots, s = 0.53     695 / 568   612 / 499   525 / 433
//      8^3 roots, s = 0.68    2039 / 1498 1809 / 1249 1482 / 1052
//   FP32-bulk
//    272 blocks, s = 0.29      113 / 116    98 / 110    93 / 104
//    664 blocks, s = 0.65      327 / 298   255 / 267   234 / 239
//    855 blocks, s = 0.21      200 / 192   176 / 178   165 / 166
//   1296 blocks, s = 0.53      470 / 403   388 / 368   367 / 343
//   4088 blocks, s = 0.31      944 / 823   794 / 752   738 / 690
// So FP64 runs whole from a share of 0.3 on (Rusanov 0.2), FP32-bulk from five
// blocks per SM on.  In FP64 the two kernels' fluxes differ in rounding; a
// rank of a partitioned grid does not know the other ranks' shares, and
// takes units there.
bool stage3d_units(int shape, int flux, int kind, const StageArgs &a, int nSM) {
  if (shape == kShape444) return true;
  if (flux == kFluxRoe || tune_value(kTuneStageVariant) != 0) return false;
  if (a.nRcBlock == 0) return true;
  if (kind != kKindFp64) return a.nBlock < 5 * nSM;
  return a.isRank || a.nRcBlock < (flux == kFluxRusanov ? 0.2 : 0.3) * a.nBlock;
}

namespace {

template <int FLUX>
cudaError_t launch_blocks(int shape, int kind, const TmaMaps &maps, const StageArgs &a, int nSM, cudaStream_t st) {
  // the implicit residual, whose finite-difference products amplify
  // rounding, keeps the reference's order of operations (flux_lean)
  if (shape == kShape888 && (a.outputResidual || !stage3d_units(shape, FLUX, kind, a, nSM)))
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
