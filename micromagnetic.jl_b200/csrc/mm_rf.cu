// mm_rf.cu -- host-side length rules of the compile-time FFT passes.
#include <algorithm>

#include "mm_rf.cuh"
#include "mm_rfpass.cuh"

namespace mm {
namespace rf {

namespace {
template <typename R, int L> constexpr int width(Kind k) {
  switch (k) {
    case KX: return XPass<R, L>::G;
    case KY: return YPass<R, L>::W;
    case KZ:
      if constexpr (z_has<R>(L)) return ZConv<R, L>::W;
      return 0;
    default:
      if constexpr (film_has<R>(L)) return FilmConv<R, L>::G;
      return 0;
  }
}

struct Entry {
  int L;
  int w[2][4];  // [FP64][kind]: block width, 0 where there is no kernel
};
template <int L> constexpr Entry entry() {
  Entry e{};
  e.L = L;
  for (int k = 0; k < 4; ++k) {
    const bool xy = L <= 4096;
    if (k == KX || k == KY) {
      if constexpr (L <= 4096) {
        e.w[0][k] = xy ? width<float, L>(static_cast<Kind>(k)) : 0;
        e.w[1][k] = xy ? width<double, L>(static_cast<Kind>(k)) : 0;
      }
    } else {
      e.w[0][k] = k == KZ ? (z_has<float>(L) ? width<float, L>(KZ) : 0) : (film_has<float>(L) ? width<float, L>(KC) : 0);
      e.w[1][k] = k == KZ ? (z_has<double>(L) ? width<double, L>(KZ) : 0) : (film_has<double>(L) ? width<double, L>(KC) : 0);
    }
  }
  return e;
}
#define E(L) entry<L>(),
constexpr Entry kEntries[] = {MM_RF_LENGTHS_A(E) MM_RF_LENGTHS_B(E) MM_RF_LENGTHS_C(E) MM_RF_LENGTHS_D(E)
                                  MM_RF_LENGTHS_E(E) MM_RF_LENGTHS_F(E) MM_RF_LENGTHS_G(E)};
#undef E

// largest padding of the next length over a request between lo and hi, in 1/1000
constexpr int worst_padding(Kind k, bool f64, int lo, int hi) {
  int worst = 0, prev = 0;
  for (const Entry& e : kEntries) {
    if (!e.w[f64][k]) continue;
    if (prev >= lo && e.L <= hi) worst = std::max(worst, (1000 * e.L + prev) / (prev + 1) - 1000);
    prev = e.L;
  }
  return worst;
}
constexpr bool padding_bounded() {
  for (Kind k : {KX, KY, KZ, KC})
    for (bool f64 : {false, true})
      if (worst_padding(k, f64, 100, 4096) > 125 || worst_padding(k, f64, 12, 100) > 231) return false;
  return true;
}
static_assert(padding_bounded(), "the lengths leave gaps above 12.5 % (23 % below 100 points)");
}  // namespace

int next_length(Kind k, bool f64, int n) {
  for (const Entry& e : kEntries)
    if (e.L >= n && e.w[f64][k]) return e.L;
  return 0;
}

Radices plan_of(Kind k, bool f64, int L) { return radices(L, k == KZ || k == KC ? cap3(f64, L) : 20); }

int tile_width(Kind k, bool f64, int L) {
  for (const Entry& e : kEntries)
    if (e.L == L) return e.w[f64][k];
  return 0;
}

}  // namespace rf
}  // namespace mm
