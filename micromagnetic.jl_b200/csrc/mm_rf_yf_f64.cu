// mm_rf_yf_f64.cu -- compile-time-length forward y passes of 3-D meshes, FP64 form.
#include "mm_rf.cuh"
#include "mm_rfpass.cuh"

namespace mm {
namespace rf {

template <>
void fwd_y<double>(int L, const cplx_t<double>* in, cplx_t<double>* out, Tw<double> t, const int* gate, int ny, int nz, int Hx,
               cudaStream_t st) {
  const int ncol = 3 * nz * Hx;
  switch (L) {
#define CASE(N)                                                                                                      \
  case N:                                                                                                            \
    launch_rf<YLine<double, N, false>>((ncol + YPass<double, N>::W - 1) / YPass<double, N>::W, st,                                \
                                  {in, out, t.tw2, t.tw3, gate, ny, Hx, ncol});                                    \
    break;
    MM_RF_XY(CASE)
#undef CASE
  }
}

}  // namespace rf
}  // namespace mm
