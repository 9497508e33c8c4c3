// Wavefront shade kernels: queues 30-33 (bumpMap / normalMap over mirror, conductor, dielectric, plastic).
#include "hk_wf_kernels.cuh"

namespace hk {
template cudaError_t wf_launch_shade_t<30>(const DevScene &, const WfState &, const WfLaunchConfig &, int, cudaStream_t);
template int wf_shade_occupancy_t<30>(int, bool);
template cudaError_t wf_launch_shade_t<31>(const DevScene &, const WfState &, const WfLaunchConfig &, int, cudaStream_t);
template int wf_shade_occupancy_t<31>(int, bool);
template cudaError_t wf_launch_shade_t<32>(const DevScene &, const WfState &, const WfLaunchConfig &, int, cudaStream_t);
template int wf_shade_occupancy_t<32>(int, bool);
template cudaError_t wf_launch_shade_t<33>(const DevScene &, const WfState &, const WfLaunchConfig &, int, cudaStream_t);
template int wf_shade_occupancy_t<33>(int, bool);
}  // namespace hk
