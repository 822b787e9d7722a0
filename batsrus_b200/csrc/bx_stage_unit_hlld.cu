// bx_stage_unit_hlld.cu -- the explicit 3D stage kernel with the Hlld flux.
#define BX_UNIT_INSTANTIATE
#include "bx_stage_unit_launch.cuh"

namespace bx {
template cudaError_t launch_unit<kFluxHlld>(int, int, const TmaMaps &, const StageArgs &, int, cudaStream_t);
}
