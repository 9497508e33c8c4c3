// Megakernel instantiation: binary tree, texture lookups compiled out, paths dealt to blocks in rounds.
#include "hk_megakernel.cuh"

namespace hk {
template cudaError_t launch_render_t<kAccelBvh2, false, true>(const DevScene &, const RenderLaunch &, int, cudaStream_t);
}  // namespace hk
