// mm_rf_fx_f64.cu -- compile-time-length forward x passes, FP64 form.
#include "mm_rf.cuh"
#include "mm_rfpass.cuh"

namespace mm {
namespace rf {

template <>
void fwd_x<double>(int L, const double* m, const double* Ms, cplx_t<double>* X, Tw<double> t, const cplx_t<double>* twx, const int* gate, int nx,
               int rows, int cols, cudaStream_t st) {
  switch (L) {
#define CASE(N)                                                                                                      \
  case N:                                                                                                            \
    launch_rf<FwdX<double, N>>((3 * rows + FwdX<double, N>::G - 1) / FwdX<double, N>::G, st,                                       \
                           {m, Ms, X, t.tw2, t.tw3, twx, gate, nx, rows, cols});                                     \
    break;
    MM_RF_XY(CASE)
#undef CASE
  }
}

}  // namespace rf
}  // namespace mm
