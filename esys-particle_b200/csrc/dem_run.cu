// FP64 instances of the multi-step kernel (dem_run.cuh; built with --fmad=false like the
// single-step FP64 form).
#include "dem_kernels.h"
#include "dem_run.cuh"

namespace dem {

cudaError_t launch_run(const StepArgs& a, bool rot, const RunArgs& ra, cudaStream_t s) {
  bool el = false, fr = false, widened = false;
  for (int d = 0; d < a.ndyn; ++d) {
    if (a.dyn[d].kind >= 2) widened = true;
    (a.dyn[d].kind == 0 ? el : fr) = true;
  }
  if (widened && rot) return launch_run_any<true, F_ELASTIC | F_FRIC | F_NFRIC, false>(a, ra, s);
  if (widened) return launch_run_any<false, F_ELASTIC | F_NFRIC, false>(a, ra, s);
  if (!rot) return launch_run_any<false, F_ELASTIC, false>(a, ra, s);
  if (!fr) return launch_run_any<true, F_ELASTIC, false>(a, ra, s);
  if (!el) return launch_run_any<true, F_FRIC, false>(a, ra, s);
  return launch_run_any<true, F_ELASTIC | F_FRIC, false>(a, ra, s);
}

}  // namespace dem
