// Wavefront shade kernels: queues 11 (coating), 12 (roughDiffuse).
#include "hk_wf_kernels.cuh"

namespace hk {
template cudaError_t wf_launch_shade_t<11>(const DevScene &, const WfState &, const WfLaunchConfig &, int, cudaStream_t);
template int wf_shade_occupancy_t<11>(int, bool);
template cudaError_t wf_launch_shade_t<12>(const DevScene &, const WfState &, const WfLaunchConfig &, int, cudaStream_t);
template int wf_shade_occupancy_t<12>(int, bool);
}  // namespace hk
