// kernels_sweep_f32.cu -- F32 instantiations of the sweeps over subtree tasks (kernels_sweep.cuh).
#include "kernels_sweep.cuh"

namespace cupf_b200 {
template void launch_sweep_stage<float>(int, const SweepTaskStage&, const SweepTaskArgs<float>&, int, const int*,
                                      const int*, int, cudaStream_t);
}  // namespace cupf_b200
