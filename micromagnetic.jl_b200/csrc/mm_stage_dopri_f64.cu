// mm_stage_dopri_f64.cu -- adaptive stage kernels of the compiled term sets, FP64 form.
#include "mm_stage.cuh"

namespace mm {

template <>
bool launch_dopri_fix<double>(const FieldArgs<double>& fa, const double* y, const StageArgs<double>& sa, const StageGrid& g,
                          cudaStream_t st) {
  switch (fa.mask) {
#define CASE(M)                                                                          \
  case (M):                                                                              \
    launch_pdl(k_stage<double, SM_DOPRI, false, (M)>, g.grid, g.block, 0, st, fa, y, sa);     \
    return true;
    MM_FIX_SETS(CASE)
#undef CASE
    default: return false;
  }
}

}  // namespace mm
