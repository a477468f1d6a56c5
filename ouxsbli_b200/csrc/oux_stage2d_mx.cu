// Fused 2D stages, mixed form: FP32 fields and face fluxes, FP64 decode and combination.
#include "oux_dispatch.h"
#include "oux_stage2d.cuh"

namespace oux {
int launch_stage2d_mx(int order, const StepArgs<float>& A, const void* src, void* dst, double* keep, cudaStream_t s) {
  return launch_stage2d_any<float>(order, A, src, dst, keep, s);
}
}  // namespace oux
