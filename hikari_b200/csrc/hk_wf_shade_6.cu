// Wavefront shade kernels: queues 25 (bumpMap / normalMap over diffuse), 26 (over roughConductor).
#include "hk_wf_kernels.cuh"

namespace hk {
template cudaError_t wf_launch_shade_t<25>(const DevScene &, const WfState &, const WfLaunchConfig &, int, cudaStream_t);
template int wf_shade_occupancy_t<25>(int, bool);
template cudaError_t wf_launch_shade_t<26>(const DevScene &, const WfState &, const WfLaunchConfig &, int, cudaStream_t);
template int wf_shade_occupancy_t<26>(int, bool);
}  // namespace hk
