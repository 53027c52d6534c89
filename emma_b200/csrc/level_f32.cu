// level_f32.cu -- mixed-path instantiation of the level kernel: FP32
// reconstruction, wave speeds and fluxes; FP64 compensated update.
#include "level_kernel.cuh"
#include "column_kernel.cuh"
#include "step_kernel.cuh"

namespace emma {

// shapes: bit i = kShapes[i] used by a level of the work list, plus kLaunchGrav
// for the gravity-coupled variant; occupancy (optional) receives the CTAs per SM
// the kernel fits.
cudaError_t launch_level_f32(const BatchArgs &a, unsigned shapes, int nsm, int ctas_per_sm, cudaStream_t s,
                             int *occupancy) {
  return launch_level_any<MathF32>(a, shapes, nsm, ctas_per_sm, s, occupancy);
}

// One fused coarse step of a subcycled tree (step_kernel.cuh).
cudaError_t launch_step_f32(const StepArgs &a, unsigned variant, int groups, int nsm, cudaStream_t s, int *grid,
                            int *threads) {
  return launch_step_any<MathF32>(a, variant, groups, nsm, s, grid, threads);
}

int step_groups_f32(unsigned variant, int groups) { return step_groups_any<MathF32>(variant, groups); }

// Column kernel of a complete level without split cells (launch flags `variant`: 0
// plain, or one of kLaunchGrav, kLaunchDual, kLaunchTracer); the plain variant with
// the shared-memory or the warp-shuffle x sweep (ColumnArgs::xshfl).
cudaError_t launch_column_f32(const ColumnArgs &a, unsigned variant, cudaStream_t s) {
  switch (variant) {
    case 0u: return a.xshfl ? launch_column32<true, false, false, 0>(a, s) : launch_column32<false, false, false, 0>(a, s);
    case kLaunchGrav: return launch_column32<false, true, false, 0>(a, s);
    case kLaunchDual: return launch_column32<false, false, true, 0>(a, s);
    case kLaunchTracer: return launch_column32<false, false, false, 1>(a, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace emma
