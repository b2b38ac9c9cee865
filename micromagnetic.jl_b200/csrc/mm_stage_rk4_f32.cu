// mm_stage_rk4_f32.cu -- fixed-step stage kernels of the compiled term sets, FP32 form.
#include "mm_stage.cuh"

namespace mm {

template <>
bool launch_rk4_fix<float>(const FieldArgs<float>& fa, const float* y, const StageArgs<float>& sa, const StageGrid& g, cudaStream_t st) {
  // two cells a thread where rows start on 8 bytes (nx even) and the pairs fill
  // every SM (1024 x 1024 x 16: 0.323 -> 0.294 ms a stage; 256 x 256 x 64 with
  // bulk DMI and anisotropy 0.079 -> 0.068; below ~200 000 cells half the threads
  // only lengthen each one's chain)
  const bool pair = !(fa.nx & 1) && fa.nx >= 32 && fa.N >= (1 << 18);
  int bx = 128, by = 1;
  while (by < 8 && by < fa.ny) by *= 2, bx /= 2;
  const dim3 pg((fa.nx / 2 + bx - 1) / bx, (fa.ny + by - 1) / by, fa.nz);
  switch (fa.mask) {
#define CASE(M)                                                                                                    \
  case (M):                                                                                                        \
    if (pair) launch_k<StagePair<(M)>>(pg, 0, st, {fa, y, sa, bx, by, dim3()});                                      \
    else                                                                                                           \
      launch_k<StagePlain<float, (M)>>(g.grid, 0, st,                                                              \
                                       {fa, y, sa, static_cast<int>(g.block.x), static_cast<int>(g.block.y), dim3()}); \
    return true;
    MM_FIX_SETS(CASE)
#undef CASE
    default: return false;
  }
}

}  // namespace mm
