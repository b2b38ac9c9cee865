// mm_rf_ix_f64.cu -- compile-time-length inverse x passes, FP64 form.
#include "mm_rf.cuh"
#include "mm_rfpass.cuh"

namespace mm {
namespace rf {

template <>
void inv_x<double>(int L, const cplx_t<double>* X, double* H, Tw<double> t, const cplx_t<double>* twx, const int* gate, int nx, int rows,
               int cols, cudaStream_t st) {
  switch (L) {
#define CASE(N)                                                                                                      \
  case N:                                                                                                            \
    launch_rf<InvX<double, N>>((3 * rows + InvX<double, N>::G - 1) / InvX<double, N>::G, st,                                       \
                           {X, H, t.tw2, t.tw3, twx, gate, nx, rows, cols});                                         \
    break;
    MM_RF_XY(CASE)
#undef CASE
  }
}

}  // namespace rf
}  // namespace mm
