// Wavefront shade kernels: queues 16 (textured roughPlastic), 17 (textured roughCoating).
#include "hk_wf_kernels.cuh"

namespace hk {
template cudaError_t wf_launch_shade_t<16>(const DevScene &, const WfState &, const WfLaunchConfig &, int, cudaStream_t);
template int wf_shade_occupancy_t<16>(int, bool);
template cudaError_t wf_launch_shade_t<17>(const DevScene &, const WfState &, const WfLaunchConfig &, int, cudaStream_t);
template int wf_shade_occupancy_t<17>(int, bool);
}  // namespace hk
