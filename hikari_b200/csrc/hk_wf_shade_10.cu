// Wavefront shade kernels: queues 18-21 (textured mirror, conductor, dielectric, plastic).
#include "hk_wf_kernels.cuh"

namespace hk {
template cudaError_t wf_launch_shade_t<18>(const DevScene &, const WfState &, const WfLaunchConfig &, int, cudaStream_t);
template int wf_shade_occupancy_t<18>(int, bool);
template cudaError_t wf_launch_shade_t<19>(const DevScene &, const WfState &, const WfLaunchConfig &, int, cudaStream_t);
template int wf_shade_occupancy_t<19>(int, bool);
template cudaError_t wf_launch_shade_t<20>(const DevScene &, const WfState &, const WfLaunchConfig &, int, cudaStream_t);
template int wf_shade_occupancy_t<20>(int, bool);
template cudaError_t wf_launch_shade_t<21>(const DevScene &, const WfState &, const WfLaunchConfig &, int, cudaStream_t);
template int wf_shade_occupancy_t<21>(int, bool);
}  // namespace hk
