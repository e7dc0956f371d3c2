// kernels_task_f64.cu -- F64 instantiations of the subtree-task kernels (kernels_task.cuh).
#include "kernels_task.cuh"

namespace cupf_b200 {
template void launch_factor_stage<double>(const TaskStage&, const FactorArgs<double, double>&, const int*, const int*, int,
                                       cudaStream_t);
}  // namespace cupf_b200
