// mm_rf_ix_f32.cu -- compile-time-length inverse x passes, FP32 form.
#include "mm_rf.cuh"
#include "mm_rfpass.cuh"

namespace mm {
namespace rf {

template <>
void inv_x<float>(int L, const cplx_t<float>* X, float* H, Tw<float> t, const cplx_t<float>* twx, const int* gate, int nx, int rows,
               int cols, cudaStream_t st) {
  switch (L) {
#define CASE(N)                                                                                                      \
  case N:                                                                                                            \
    launch_rf<InvX<float, N>>((3 * rows + InvX<float, N>::G - 1) / InvX<float, N>::G, st,                                       \
                           {X, H, t.tw2, t.tw3, twx, gate, nx, rows, cols});                                         \
    break;
    MM_RF_XY(CASE)
#undef CASE
  }
}

}  // namespace rf
}  // namespace mm
