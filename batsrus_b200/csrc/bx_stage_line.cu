// bx_stage_line.cu -- instantiations and launcher of the stage kernel of 1D
// blocks (bx_stage_line.cuh); compiled with --fmad=false.
#include "bx_stage_line.cuh"

namespace bx {

namespace {

template <class S, int FLUX>
cudaError_t launch_line_flux(const StageArgs &a, cudaStream_t st) {
  switch (a.limiter) {
    case kLimMinmod: return launch_dependent(stage_line_kernel<S, FLUX, kLimMinmod>, a.nBlock, S::NTHR, 0, st, a);
    case kLimMc: return launch_dependent(stage_line_kernel<S, FLUX, kLimMc>, a.nBlock, S::NTHR, 0, st, a);
    case kLimMc3: return launch_dependent(stage_line_kernel<S, FLUX, kLimMc3>, a.nBlock, S::NTHR, 0, st, a);
  }
  return cudaErrorInvalidValue;
}

template <class S>
cudaError_t launch_line_shape(int flux, const StageArgs &a, cudaStream_t st) {
  switch (flux) {
    case kFluxRusanov: return launch_line_flux<S, kFluxRusanov>(a, st);
    case kFluxLinde: return launch_line_flux<S, kFluxLinde>(a, st);
    case kFluxHlld: return launch_line_flux<S, kFluxHlld>(a, st);
    case kFluxRoe: return launch_line_flux<S, kFluxRoe>(a, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace

cudaError_t launch_stage_line(int shape, int flux, const StageArgs &a, cudaStream_t st) {
  switch (shape) {
    case kShape811: return launch_line_shape<Line<8>>(flux, a, st);
    case kShape6411: return launch_line_shape<Line<64>>(flux, a, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace bx
