// Megakernel instantiation: binary tree, texture lookups compiled in, paths dealt to blocks in rounds.
#include "hk_megakernel.cuh"

namespace hk {
template cudaError_t launch_render_t<kAccelBvh2, true, true>(const DevScene &, const RenderLaunch &, int, cudaStream_t);
}  // namespace hk
