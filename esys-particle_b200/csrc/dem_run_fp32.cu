// FP32-force instances of the multi-step kernel (dem_run.cuh; built with FMA contraction like
// the single-step FP32 form).
#include "dem_kernels.h"
#include "dem_run.cuh"

namespace dem {

cudaError_t launch_run_fp32(const StepArgs& a, bool rot, const RunArgs& ra, cudaStream_t s) {
  bool el = false, fr = false;
  for (int d = 0; d < a.ndyn; ++d) (a.dyn[d].kind == 0 ? el : fr) = true;
  if (!rot) return launch_run_any<false, F_ELASTIC, true>(a, ra, s);
  if (!fr) return launch_run_any<true, F_ELASTIC, true>(a, ra, s);
  if (!el) return launch_run_any<true, F_FRIC, true>(a, ra, s);
  return launch_run_any<true, F_ELASTIC | F_FRIC, true>(a, ra, s);
}

}  // namespace dem
