// Wavefront shade kernels: queues 27-29 (bumpMap / normalMap over roughDielectric, roughPlastic, roughCoating).
#include "hk_wf_kernels.cuh"

namespace hk {
template cudaError_t wf_launch_shade_t<27>(const DevScene &, const WfState &, const WfLaunchConfig &, int, cudaStream_t);
template int wf_shade_occupancy_t<27>(int, bool);
template cudaError_t wf_launch_shade_t<28>(const DevScene &, const WfState &, const WfLaunchConfig &, int, cudaStream_t);
template int wf_shade_occupancy_t<28>(int, bool);
template cudaError_t wf_launch_shade_t<29>(const DevScene &, const WfState &, const WfLaunchConfig &, int, cudaStream_t);
template int wf_shade_occupancy_t<29>(int, bool);
}  // namespace hk
