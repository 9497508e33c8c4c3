// Wavefront shade kernels: queues 30 (run-time dispatch: deep stacks, twoSided, maps over smooth types).
#include "hk_wf_kernels.cuh"

namespace hk {
template cudaError_t wf_launch_shade_t<30>(const DevScene &, const WfState &, const WfLaunchConfig &, int, cudaStream_t);
template int wf_shade_occupancy_t<30>(int, bool);
}  // namespace hk
