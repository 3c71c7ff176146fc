// spond_inst_f64_256.cu -- the FP64 run of spond.cuh with 256 threads per CTA.
#include "spond.cuh"

namespace espec {
namespace nd {
cudaError_t nd_launch_f64_256(const NdArgs<double>& a, int grid, size_t smem, cudaStream_t st) {
  return nd_kernel_launch<double, 256, 9>(a, grid, smem, st);
}
}  // namespace nd
}  // namespace espec
