// Persistent run kernels with the exact (reference evaluation order) FP64
// policy.  Compiled with -fmad=false so that no multiply-add is contracted.
#include "fv_persist.cuh"

namespace fvgpu {
namespace tile {
void run_kernels_exact(const FusedParams& FP, RunKernel* k) { RunLaunch<MExact>::kernels(FP, k); }
}  // namespace tile
}  // namespace fvgpu
