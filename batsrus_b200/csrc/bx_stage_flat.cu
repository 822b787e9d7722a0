// bx_stage_flat.cu -- instantiations and launcher of the stage kernel of 2D
// blocks (bx_stage_flat.cuh); compiled with --fmad=false.
#include "bx_stage_flat.cuh"

namespace bx {

namespace {

template <int FLUX, int CTAS>
cudaError_t launch_flat_flux(const StageArgs &a, cudaStream_t st) {
  stage_flat_kernel<FLUX, CTAS><<<a.nBlock, Flat::NTHREAD, 0, st>>>(a);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_stage_flat(int flux, const StageArgs &a, int nSM, cudaStream_t st) {
  switch (flux) {
    case kFluxRusanov: return launch_flat_flux<kFluxRusanov, 5>(a, st);
    case kFluxLinde: {
      const auto waves = [&](int ctas) { return (a.nBlock + ctas * nSM - 1) / (ctas * nSM); };
      return waves(5) < waves(4) ? launch_flat_flux<kFluxLinde, 5>(a, st) : launch_flat_flux<kFluxLinde, 4>(a, st);
    }
    case kFluxHlld: return launch_flat_flux<kFluxHlld, 5>(a, st);
    case kFluxRoe: return launch_flat_flux<kFluxRoe, 5>(a, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace bx
