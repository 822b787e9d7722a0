// bx_stage_flat.cu -- instantiations and launcher of the stage kernel of 1D
// and 2D blocks (bx_stage_flat.cuh).
#include "bx_stage_flat.cuh"

namespace bx {

namespace {

template <class S, int FLUX>
cudaError_t launch_flat_flux(const StageArgs &a, cudaStream_t st) {
  switch (a.limiter) {
    case kLimMinmod: stage_flat_kernel<S, FLUX, kLimMinmod><<<a.nBlock, S::NTHR, 0, st>>>(a); break;
    case kLimMc: stage_flat_kernel<S, FLUX, kLimMc><<<a.nBlock, S::NTHR, 0, st>>>(a); break;
    case kLimMc3: stage_flat_kernel<S, FLUX, kLimMc3><<<a.nBlock, S::NTHR, 0, st>>>(a); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

template <class S>
cudaError_t launch_flat_shape(int flux, const StageArgs &a, cudaStream_t st) {
  switch (flux) {
    case kFluxRusanov: return launch_flat_flux<S, kFluxRusanov>(a, st);
    case kFluxLinde: return launch_flat_flux<S, kFluxLinde>(a, st);
    case kFluxHlld: return launch_flat_flux<S, kFluxHlld>(a, st);
    case kFluxRoe: return launch_flat_flux<S, kFluxRoe>(a, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace

cudaError_t launch_stage_flat(int shape, int flux, const StageArgs &a, cudaStream_t st) {
  switch (shape) {
    case kShape881: return launch_flat_shape<Flat<8, 8>>(flux, a, st);
    case kShape811: return launch_flat_shape<Flat<8, 1>>(flux, a, st);
    case kShape6411: return launch_flat_shape<Flat<64, 1>>(flux, a, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace bx
