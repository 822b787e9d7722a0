// bx_stage3d_v2.cu -- instantiations and launchers of the single-face-phase
// stage kernel for 8^3 blocks (bx_stage3d_v2.cuh): the residual of the
// implicit step in FP64, and the explicit stages with the Roe flux, whose
// long face code runs better with one set of barriers per block and 128
// registers (96^3: 665 us per FP64 step and 368 per FP32-bulk step, against
// 800 and 420 in units of 128 cells).
#include "bx_stage3d_launch.cuh"
#include "bx_stage3d_v2.cuh"

namespace bx {

namespace {

// one CTA of 512 threads per SM in FP64 (the tile and the face slots fill the
// shared memory), two of 256 in FP32
template <int NTHR, int MINB, typename TileT, typename Real, typename OutT, int FLUX, int LIM, bool RC>
cudaError_t launch8(const TmaMaps &maps, const StageArgs &a, int nSM, cudaStream_t st) {
  using B = Blk8<TileT, Real, NTHR, MINB>;
  auto k = stage8_kernel<B, TileT, Real, OutT, FLUX, LIM, RC>;
  constexpr size_t sm = B::smem_bytes;
  static bool attr = false;
  if (!attr) {
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    attr = true;
  }
  const int want = nSM * MINB;
  k<<<a.nBlock < want ? a.nBlock : want, NTHR, sm, st>>>(maps, a);
  return cudaGetLastError();
}

template <int NTHR, int MINB, typename TileT, typename Real, typename OutT, int FLUX, bool RC>
cudaError_t launch8_lim(const TmaMaps &maps, const StageArgs &a, int nSM, cudaStream_t st) {
  switch (a.limiter) {
    case kLimMinmod: return launch8<NTHR, MINB, TileT, Real, OutT, FLUX, kLimMinmod, RC>(maps, a, nSM, st);
    case kLimMc: return launch8<NTHR, MINB, TileT, Real, OutT, FLUX, kLimMc, RC>(maps, a, nSM, st);
    case kLimMc3: return launch8<NTHR, MINB, TileT, Real, OutT, FLUX, kLimMc3, RC>(maps, a, nSM, st);
  }
  return cudaErrorInvalidValue;
}

template <bool RC>
cudaError_t launch8_residual(int flux, const TmaMaps &maps, const StageArgs &a, int nSM, cudaStream_t st) {
  switch (flux) {
    case kFluxRusanov: return launch8_lim<512, 1, double, double, double, kFluxRusanov, RC>(maps, a, nSM, st);
    case kFluxLinde: return launch8_lim<512, 1, double, double, double, kFluxLinde, RC>(maps, a, nSM, st);
    case kFluxHlld: return launch8_lim<512, 1, double, double, double, kFluxHlld, RC>(maps, a, nSM, st);
    case kFluxRoe: return launch8_lim<512, 1, double, double, double, kFluxRoe, RC>(maps, a, nSM, st);
  }
  return cudaErrorInvalidValue;
}

template <bool RC>
cudaError_t launch8_roe(int kind, const TmaMaps &maps, const StageArgs &a, int nSM, cudaStream_t st) {
  switch (kind) {
    case kKindFp64: return launch8_lim<512, 1, double, double, double, kFluxRoe, RC>(maps, a, nSM, st);
    case kKindFp32In64: return launch8_lim<256, 2, double, float, float, kFluxRoe, RC>(maps, a, nSM, st);
    case kKindFp32In32: return launch8_lim<256, 2, float, float, double, kFluxRoe, RC>(maps, a, nSM, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace

cudaError_t launch_stage8_residual(int flux, const TmaMaps &maps, const StageArgs &a, int nSM, cudaStream_t st) {
  if (a.anySpecial) return launch8_residual<true>(flux, maps, a, nSM, st);
  return launch8_residual<false>(flux, maps, a, nSM, st);
}

cudaError_t launch_stage8_roe(int kind, const TmaMaps &maps, const StageArgs &a, int nSM, cudaStream_t st) {
  return a.anySpecial ? launch8_roe<true>(kind, maps, a, nSM, st) : launch8_roe<false>(kind, maps, a, nSM, st);
}

}  // namespace bx
