// Persistent run kernels with the FP64 fast policy.
#include "fv_persist.cuh"

namespace fvgpu {
namespace tile {
void run_kernels_f64(const FusedParams& FP, RunKernel* k) { RunLaunch<MF64>::kernels(FP, k); }
}  // namespace tile
}  // namespace fvgpu
