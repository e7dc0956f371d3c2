// kernels_task_f32.cu -- F32 instantiations of the subtree-task kernels (kernels_task.cuh).
#include "kernels_task.cuh"

namespace cupf_b200 {
template void launch_factor_stage<float>(const TaskStage&, const FactorArgs<float, float>&, const int*, const int*, int,
                                       cudaStream_t);
}  // namespace cupf_b200
