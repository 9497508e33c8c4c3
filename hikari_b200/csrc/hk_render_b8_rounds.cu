// Megakernel instantiation: 8-wide tree, texture lookups compiled out, paths dealt to blocks in rounds.
#include "hk_megakernel.cuh"

namespace hk {
template cudaError_t launch_render_t<kAccelBvh8, false, true>(const DevScene &, const RenderLaunch &, int, cudaStream_t);
}  // namespace hk
