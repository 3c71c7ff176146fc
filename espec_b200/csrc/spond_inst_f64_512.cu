// spond_inst_f64_512.cu -- the FP64 run of spond.cuh with 512 threads per CTA.
#include "spond.cuh"

namespace espec {
namespace nd {
cudaError_t nd_launch_f64_512(const NdArgs<double>& a, int grid, size_t smem, cudaStream_t st) {
  return nd_kernel_launch<double, 512, kMaxLn512<double>>(a, grid, smem, st);
}
}  // namespace nd
}  // namespace espec
