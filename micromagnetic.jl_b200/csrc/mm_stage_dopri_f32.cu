// mm_stage_dopri_f32.cu -- adaptive stage kernels of the compiled term sets, FP32 form.
#include "mm_stage.cuh"

namespace mm {

template <>
bool launch_dopri_fix<float>(const FieldArgs<float>& fa, const float* y, const StageArgs<float>& sa, const StageGrid& g,
                          cudaStream_t st) {
  switch (fa.mask) {
#define CASE(M)                                                                          \
  case (M):                                                                              \
    launch_pdl(k_stage<float, SM_DOPRI, false, (M)>, g.grid, g.block, 0, st, fa, y, sa);     \
    return true;
    MM_FIX_SETS(CASE)
#undef CASE
    default: return false;
  }
}

}  // namespace mm
