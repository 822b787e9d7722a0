// bx_stage8_linde.cu -- the stage kernel of whole 8^3 blocks with the Linde flux.
#define BX_STAGE8_INSTANTIATE
#include "bx_stage8_launch.cuh"

namespace bx {
template cudaError_t launch_stage8<kFluxLinde>(int, const TmaMaps &, const StageArgs &, int, cudaStream_t);
}
