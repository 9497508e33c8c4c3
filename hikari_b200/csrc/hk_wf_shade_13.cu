// Wavefront shade kernels: queues 35 (bumpMap / normalMap over coating), 36 (over roughDiffuse).
#include "hk_wf_kernels.cuh"

namespace hk {
template cudaError_t wf_launch_shade_t<35>(const DevScene &, const WfState &, const WfLaunchConfig &, int, cudaStream_t);
template int wf_shade_occupancy_t<35>(int, bool);
template cudaError_t wf_launch_shade_t<36>(const DevScene &, const WfState &, const WfLaunchConfig &, int, cudaStream_t);
template int wf_shade_occupancy_t<36>(int, bool);
}  // namespace hk
