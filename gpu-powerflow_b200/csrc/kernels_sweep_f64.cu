// kernels_sweep_f64.cu -- F64 instantiations of the sweeps over subtree tasks (kernels_sweep.cuh).
#include "kernels_sweep.cuh"

namespace cupf_b200 {
template void launch_sweep_stage<double>(int, const SweepTaskStage&, const SweepTaskArgs<double>&, int, const int*,
                                      const int*, int, cudaStream_t);
}  // namespace cupf_b200
