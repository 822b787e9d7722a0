// bx_stage_flat.cu -- instantiations and launcher of the stage kernel of 2D
// blocks (bx_stage_flat.cuh); compiled with --fmad=false.
#include "bx_stage_flat.cuh"

namespace bx {

namespace {

template <int FLUX>
cudaError_t launch_flat_flux(const StageArgs &a, cudaStream_t st) {
  stage_flat_kernel<FLUX><<<a.nBlock, Flat::NTHREAD, 0, st>>>(a);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_stage_flat(int flux, const StageArgs &a, cudaStream_t st) {
  switch (flux) {
    case kFluxRusanov: return launch_flat_flux<kFluxRusanov>(a, st);
    case kFluxLinde: return launch_flat_flux<kFluxLinde>(a, st);
    case kFluxHlld: return launch_flat_flux<kFluxHlld>(a, st);
    case kFluxRoe: return launch_flat_flux<kFluxRoe>(a, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace bx
