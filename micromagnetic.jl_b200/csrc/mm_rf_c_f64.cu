// mm_rf_c_f64.cu -- compile-time-length fused film columns, FP64 form.
#include "mm_rf.cuh"
#include "mm_rfpass.cuh"

namespace mm {
namespace rf {

template <int L> static void film_case(cplx_t<double>* X, const double* Nhat, Tw<double> t, const int* gate, int ny, int Hx, cudaStream_t st) {
  if constexpr (film_has<double>(L)) {
    using K = FilmConv<double, L>;
    launch_rf<K>((Hx + K::G - 1) / K::G, st, {X, Nhat, t.tw2, t.tw3, gate, ny, Hx});
  }
}

template <>
void conv_film<double>(int L, cplx_t<double>* X, const double* Nhat, Tw<double> t, const int* gate, int ny, int Hx, cudaStream_t st) {
  switch (L) {
#define CASE(N) \
  case N: film_case<N>(X, Nhat, t, gate, ny, Hx, st); break;
    MM_RF_XY(CASE) MM_RF_LENGTHS_G(CASE)
#undef CASE
  }
}

}  // namespace rf
}  // namespace mm
