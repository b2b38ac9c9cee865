// mm_rf_fx_f32.cu -- compile-time-length forward x passes, FP32 form.
#include "mm_rf.cuh"
#include "mm_rfpass.cuh"

namespace mm {
namespace rf {

template <>
void fwd_x<float>(int L, const float* m, const float* Ms, cplx_t<float>* X, Tw<float> t, const cplx_t<float>* twx, const int* gate, int nx,
               int rows, int cols, cudaStream_t st) {
  switch (L) {
#define CASE(N)                                                                                                      \
  case N:                                                                                                            \
    launch_rf<FwdX<float, N>>((3 * rows + FwdX<float, N>::G - 1) / FwdX<float, N>::G, st,                                       \
                           {m, Ms, X, t.tw2, t.tw3, twx, gate, nx, rows, cols});                                     \
    break;
    MM_RF_XY(CASE)
#undef CASE
  }
}

}  // namespace rf
}  // namespace mm
