// mm_rf_yi_f32.cu -- compile-time-length inverse y passes of 3-D meshes, FP32 form.
#include "mm_rf.cuh"
#include "mm_rfpass.cuh"

namespace mm {
namespace rf {

template <>
void inv_y<float>(int L, const cplx_t<float>* in, cplx_t<float>* out, Tw<float> t, const int* gate, int ny, int nz, int Hx,
               cudaStream_t st) {
  const int ncol = 3 * nz * Hx;
  switch (L) {
#define CASE(N)                                                                                                      \
  case N:                                                                                                            \
    launch_rf<YLine<float, N, true>>((ncol + YPass<float, N>::W - 1) / YPass<float, N>::W, st,                                \
                                  {in, out, t.tw2, t.tw3, gate, ny, Hx, ncol});                                    \
    break;
    MM_RF_XY(CASE)
#undef CASE
  }
}

}  // namespace rf
}  // namespace mm
