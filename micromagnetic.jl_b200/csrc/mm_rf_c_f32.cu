// mm_rf_c_f32.cu -- compile-time-length fused film columns, FP32 form.
#include "mm_rf.cuh"
#include "mm_rfpass.cuh"

namespace mm {
namespace rf {

template <int L> static void film_case(cplx_t<float>* X, const float* Nhat, Tw<float> t, const int* gate, int ny, int Hx, cudaStream_t st) {
  if constexpr (film_has<float>(L)) {
    using K = FilmConv<float, L>;
    launch_rf<K>((Hx + K::G - 1) / K::G, st, {X, Nhat, t.tw2, t.tw3, gate, ny, Hx});
  }
}

template <>
void conv_film<float>(int L, cplx_t<float>* X, const float* Nhat, Tw<float> t, const int* gate, int ny, int Hx, cudaStream_t st) {
  switch (L) {
#define CASE(N) \
  case N: film_case<N>(X, Nhat, t, gate, ny, Hx, st); break;
    MM_RF_XY(CASE) MM_RF_LENGTHS_G(CASE)
#undef CASE
  }
}

}  // namespace rf
}  // namespace mm
