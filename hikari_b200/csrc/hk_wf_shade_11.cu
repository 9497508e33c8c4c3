// Wavefront shade kernels: queues 23 (textured coating), 24 (textured roughDiffuse).
#include "hk_wf_kernels.cuh"

namespace hk {
template cudaError_t wf_launch_shade_t<23>(const DevScene &, const WfState &, const WfLaunchConfig &, int, cudaStream_t);
template int wf_shade_occupancy_t<23>(int, bool);
template cudaError_t wf_launch_shade_t<24>(const DevScene &, const WfState &, const WfLaunchConfig &, int, cudaStream_t);
template int wf_shade_occupancy_t<24>(int, bool);
}  // namespace hk
