// bx_stage_unit_rusanov.cu -- the explicit 3D stage kernel with the Rusanov flux.
#define BX_UNIT_INSTANTIATE
#include "bx_stage_unit_launch.cuh"

namespace bx {
template cudaError_t launch_unit<kFluxRusanov>(int, int, const TmaMaps &, const StageArgs &, int, cudaStream_t);
}
