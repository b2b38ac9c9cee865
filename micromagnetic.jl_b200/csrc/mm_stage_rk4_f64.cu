// mm_stage_rk4_f64.cu -- fixed-step stage kernels of the compiled term sets, FP64 form.
#include "mm_stage.cuh"

namespace mm {

template <>
bool launch_rk4_fix<double>(const FieldArgs<double>& fa, const double* y, const StageArgs<double>& sa, const StageGrid& g, cudaStream_t st) {
  switch (fa.mask) {
#define CASE(M)                                                                                                    \
  case (M):                                                                                                        \
    launch_k<StagePlain<double, (M)>>(g.grid, 0, st,                                                                  \
                                   {fa, y, sa, static_cast<int>(g.block.x), static_cast<int>(g.block.y), dim3()}); \
    return true;
    MM_FIX_SETS(CASE)
#undef CASE
    default: return false;
  }
}

}  // namespace mm
