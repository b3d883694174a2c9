// Persistent run kernels with the FP32-bulk policy, and the per-precision
// dispatch.
#include "fv_persist.cuh"

namespace fvgpu {
namespace tile {
void run_kernels_exact(const FusedParams& FP, RunKernel* k);
void run_kernels_f64(const FusedParams& FP, RunKernel* k);
void run_kernels(int precision, const FusedParams& FP, RunKernel* k) {
    if (precision == 0) run_kernels_exact(FP, k);
    else if (precision == 1) run_kernels_f64(FP, k);
    else RunLaunch<MF32>::kernels(FP, k);
}
}  // namespace tile
}  // namespace fvgpu
