// Wavefront shade kernels: queues 37 (run-time dispatch: deep stacks, twoSided, maps over them).
#include "hk_wf_kernels.cuh"

namespace hk {
template cudaError_t wf_launch_shade_t<37>(const DevScene &, const WfState &, const WfLaunchConfig &, int, cudaStream_t);
template int wf_shade_occupancy_t<37>(int, bool);
}  // namespace hk
