// mm_rf_z_f64.cu -- compile-time-length z convolutions, FP64 form.
#include "mm_rf.cuh"
#include "mm_rfpass.cuh"

namespace mm {
namespace rf {

template <>
void conv_z<double>(int L, cplx_t<double>* Y, const double* Nhat, Tw<double> t, const int* gate, int nz, int Hx, int Py,
                cudaStream_t st) {
  const int64_t n = static_cast<int64_t>(Py) * Hx;
  switch (L) {
#define CASE(N)                                                                                                      \
  case N:                                                                                                            \
    if constexpr (z_has<double>(N)) {                                                                                    \
      const int tiles = static_cast<int>((n + ZConv<double, N>::W - 1) / ZConv<double, N>::W);                               \
      launch_rf<ZConv<double, N>>(tiles, st, {Y, Nhat, t.tw2, t.tw3, gate, nz, Hx, Py, tiles});                          \
    }                                                                                                                \
    break;
    MM_RF_LENGTHS_A(CASE) MM_RF_LENGTHS_B(CASE)
#undef CASE
  }
}

}  // namespace rf
}  // namespace mm
