// spond_inst_f32_256.cu -- the FP32 run of spond.cuh with 256 threads per CTA.
#include "spond.cuh"

namespace espec {
namespace nd {
cudaError_t nd_launch_f32_256(const NdArgs<float>& a, int grid, size_t smem, cudaStream_t st) {
  return nd_kernel_launch<float, 256, 9>(a, grid, smem, st);
}
}  // namespace nd
}  // namespace espec
