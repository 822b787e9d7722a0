// bx_stage_flat.cu -- instantiations and launcher of the stage kernel of 2D
// blocks (bx_stage_flat.cuh).
#include "bx_stage_flat.cuh"

namespace bx {

namespace {

// as many CTAs as are resident together, each working through its blocks
inline int sm_count() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) n = 148;
  }
  return n;
}

template <class S, int FLUX>
cudaError_t launch_flat_flux(const StageArgs &a, cudaStream_t st) {
  const int want = S::minb(FLUX) * sm_count(), grid = a.nBlock < want ? a.nBlock : want;
  switch (a.limiter) {
    case kLimMinmod: return launch_dependent(stage_flat_kernel<S, FLUX, kLimMinmod>, grid, S::NTHR, 0, st, a);
    case kLimMc: return launch_dependent(stage_flat_kernel<S, FLUX, kLimMc>, grid, S::NTHR, 0, st, a);
    case kLimMc3: return launch_dependent(stage_flat_kernel<S, FLUX, kLimMc3>, grid, S::NTHR, 0, st, a);
  }
  return cudaErrorInvalidValue;
}

}  // namespace

cudaError_t launch_stage_flat(int flux, const StageArgs &a, cudaStream_t st) {
  using S = Flat<8, 8>;
  switch (flux) {
    case kFluxRusanov: return launch_flat_flux<S, kFluxRusanov>(a, st);
    case kFluxLinde: return launch_flat_flux<S, kFluxLinde>(a, st);
    case kFluxHlld: return launch_flat_flux<S, kFluxHlld>(a, st);
    case kFluxRoe: return launch_flat_flux<S, kFluxRoe>(a, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace bx
