// Fused 2D stages, FP64 form, compiled without FMA contraction.
#include "oux_dispatch.h"
#include "oux_stage2d.cuh"

namespace oux {
int launch_stage2d_fp64(int order, const StepArgs<double>& A, const void* src, void* dst, double* keep, cudaStream_t s) {
  return launch_stage2d_any<double>(order, A, src, dst, keep, s);
}
}  // namespace oux
