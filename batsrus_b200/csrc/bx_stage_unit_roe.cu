// bx_stage_unit_roe.cu -- the explicit 3D stage kernel with the Roe flux.
#define BX_UNIT_INSTANTIATE
#include "bx_stage_unit_launch.cuh"

namespace bx {
template cudaError_t launch_unit<kFluxRoe>(int, int, const TmaMaps &, const StageArgs &, int, cudaStream_t);
}
