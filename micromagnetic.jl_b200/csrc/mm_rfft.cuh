// mm_rfft.cuh -- 1-D complex transforms of compile-time length, one radix
// butterfly a thread at a time, exchanged through one shared buffer in place
// (internal).
//
// A length L = R1 * R2 * R3 (R1 even; R2 = 1 for two-stage lengths) runs as
//   S1  over n = i1 + a R2 R3 (a < R1; i1 = r R3 + q)       -> (r, q, k)
//   S2  over r, twiddle w_{R1 R2}^(r k)                      -> (r', q, k)
//   S3  over q, twiddle w_L^(q i3), i3 = r' R1 + k           -> frequency i3 + j R1 R2
// and the inverse walks the same three stages backwards with the conjugate
// twiddles.  Element (r, q, k) lives at r PB + q PA + k of a line's shared
// buffer; a butterfly of S2 or S3 writes back to the addresses it read, so a
// stage needs one barrier and a line one buffer (the run-time engine of
// mm_lines.cuh ping-pongs between two).  All strides, twiddle strides and
// trip counts are constants of the instantiation: on a 2000-point film column
// the run-time engine spends ~200 instructions a value and stage set, most of
// them index arithmetic, this one ~60.
//
// The transforms are those of zero-padded lines (data in the first half,
// results kept in the first half): S1 of the forward transform takes only the
// R1/2 inputs that can be non-zero and S1 of the inverse forms only the R1/2
// outputs that are kept, each as two transforms of length R1/2 (even and odd
// frequencies), so the padded half is neither loaded nor multiplied.
//
// Twiddles: two tables in the order the lanes read them, tw2[(r-1) R1 + k] and
// tw3[(q-1) R1 R2 + i3] (rfft_fill_twiddles), FP64-accurate.
#pragma once
#include "mm_fft.cuh"

namespace mm {
namespace rf {

// ------------------------------------------------ compile-time constants ---
// cos / sin of 2 pi k / n by their Taylor series on [0, pi/4], evaluated by
// the compiler
struct CS {
  double c, s;
};
constexpr CS cs_series(double x) {
  double c = 0, s = 0, tc = 1, ts = x;
  for (int i = 0; i < 14; ++i) {
    c += tc;
    s += ts;
    tc *= -x * x / ((2.0 * i + 1) * (2.0 * i + 2));
    ts *= -x * x / ((2.0 * i + 2) * (2.0 * i + 3));
  }
  return {c, s};
}
constexpr CS cs_turn(int k, int n) {  // angle 2 pi k / n, 0 <= k < n
  const int o = 8 * k / n;            // octant
  const int num = 8 * k - o * n;      // angle = (o + num / n) pi / 4
  const double pi4 = 0.785398163397448309615660845819875721;
  const bool rev = o & 1;
  const CS b = cs_series(pi4 * (rev ? n - num : num) / n);
  // in the octant: (cos, sin) of the reduced angle, mirrored in odd octants
  const double c0 = rev ? b.s : b.c, s0 = rev ? b.c : b.s;
  switch (o >> 1) {
    case 0: return {c0, s0};
    case 1: return {-s0, c0};
    case 2: return {-c0, -s0};
    default: return {s0, -c0};
  }
}
template <int N> struct CsTab {
  double v[N][2];
};
template <int N> constexpr CsTab<N> make_cs_tab() {
  CsTab<N> t{};
  for (int k = 0; k < N; ++k) {
    const CS a = cs_turn(k, N);
    t.v[k][0] = a.c;
    t.v[k][1] = a.s;
  }
  return t;
}
template <int N> __host__ __device__ constexpr double cs_const(int k, int sin_part) {
  constexpr CsTab<N> t = make_cs_tab<N>();
  return t.v[k][sin_part];
}
// exp(-+ 2 pi i k / N) (minus: forward), 0 <= k < N
template <int N, bool INV, typename C> __device__ __forceinline__ C wconst(int k) {
  using R = decltype(C::x);
  const R c = static_cast<R>(cs_const<N>(k, 0)), s = static_cast<R>(cs_const<N>(k, 1));
  return cmk<C>(c, INV ? s : -s);
}

// ------------------------------------------------------------ butterflies ---
template <int R, bool INV, typename C> __device__ __forceinline__ void dft(C* v);

// N1 * N2 with coprime factors (Good's prime-factor map: no twiddles)
template <int N1, int N2, bool INV, typename C> __device__ __forceinline__ void dft_pfa(C* v) {
  constexpr int N = N1 * N2;
  C t[N1][N2];
#pragma unroll
  for (int a = 0; a < N1; ++a) {
#pragma unroll
    for (int b = 0; b < N2; ++b) t[a][b] = v[(N2 * a + N1 * b) % N];
    dft<N2, INV>(t[a]);
  }
#pragma unroll
  for (int b = 0; b < N2; ++b) {
    C u[N1];
#pragma unroll
    for (int a = 0; a < N1; ++a) u[a] = t[a][b];
    dft<N1, INV>(u);
#pragma unroll
    for (int a = 0; a < N1; ++a) {
      // the k < N with k = a mod N1 and k = b mod N2
      int k = b;
#pragma unroll
      for (int s = 0; s < N1; ++s)
        if ((b + s * N2) % N1 == a) k = b + s * N2;
      v[k] = u[a];
    }
  }
}

template <bool INV, typename C> __device__ __forceinline__ void dft9(C* v) {
  C t[3][3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
#pragma unroll
    for (int b = 0; b < 3; ++b) t[a][b] = v[a + 3 * b];
    dft3<INV>(t[a]);
  }
  t[1][1] = cmul(t[1][1], wconst<9, INV, C>(1));
  t[1][2] = cmul(t[1][2], wconst<9, INV, C>(2));
  t[2][1] = cmul(t[2][1], wconst<9, INV, C>(2));
  t[2][2] = cmul(t[2][2], wconst<9, INV, C>(4));
#pragma unroll
  for (int b = 0; b < 3; ++b) {
    C u[3] = {t[0][b], t[1][b], t[2][b]};
    dft3<INV>(u);
    v[b] = u[0];
    v[b + 3] = u[1];
    v[b + 6] = u[2];
  }
}

template <int R, bool INV, typename C> __device__ __forceinline__ void dft(C* v) {
  if constexpr (R == 1) return;
  else if constexpr (R == 2) dft2<INV>(v);
  else if constexpr (R == 3) dft3<INV>(v);
  else if constexpr (R == 4) dft4<INV>(v);
  else if constexpr (R == 5) dft5<INV>(v);
  else if constexpr (R == 6) dft_pfa<2, 3, INV>(v);
  else if constexpr (R == 8) dft8<INV>(v);
  else if constexpr (R == 9) dft9<INV>(v);
  else if constexpr (R == 10) dft_pfa<2, 5, INV>(v);
  else if constexpr (R == 12) dft_pfa<4, 3, INV>(v);
  else if constexpr (R == 15) dft_pfa<3, 5, INV>(v);
  else if constexpr (R == 16) dft16<INV>(v);
  else {
    static_assert(R == 20, "no butterfly of this radix");
    dft_pfa<4, 5, INV>(v);
  }
}

// Forward radix R (even) of inputs v[0 .. R/2), the others zero: even and odd
// frequencies are transforms of length R/2.
template <int R, typename C> __device__ __forceinline__ void dft_half_in(C* v) {
  constexpr int H = R / 2;
  C o[H], e[H];
#pragma unroll
  for (int n = 0; n < H; ++n) {
    e[n] = v[n];
    o[n] = n == 0 ? v[0] : cmul(v[n], wconst<R, false, C>(n));
  }
  dft<H, false>(e);
  dft<H, false>(o);
#pragma unroll
  for (int k = 0; k < H; ++k) {
    v[2 * k] = e[k];
    v[2 * k + 1] = o[k];
  }
}

// Inverse radix R (even), outputs v[0 .. R/2) only
template <int R, typename C> __device__ __forceinline__ void dft_half_out(C* v) {
  constexpr int H = R / 2;
  C o[H], e[H];
#pragma unroll
  for (int k = 0; k < H; ++k) {
    e[k] = v[2 * k];
    o[k] = v[2 * k + 1];
  }
  dft<H, true>(e);
  dft<H, true>(o);
#pragma unroll
  for (int n = 0; n < H; ++n) v[n] = n == 0 ? cadd(e[0], o[0]) : cadd(e[n], cmul(o[n], wconst<R, true, C>(n)));
}

// ------------------------------------------------------------------ plans ---
struct Radices {
  int r1, r2, r3;  // r1 = 0: no plan
};
// Factors of L into at most three radices, the fewest stages first, then the
// smallest largest radix, then the smallest last radix.  cap bounds the last
// radix: the three-component kernels hold 3 r3 values a thread (FP64: 12 r3
// registers), so they take r3 <= 10 in FP64 and 16 in FP32 where single lines
// take 20.
constexpr bool is_radix(int r) {
  for (int q : {2, 3, 4, 5, 6, 8, 9, 10, 12, 15, 16, 20})
    if (r == q) return true;
  return false;
}
constexpr bool is_first(int r) { return r % 2 == 0 && r >= 4 && is_radix(r); }
constexpr Radices radices(int L, int cap = 20) {
  Radices best{0, 0, 0};
  int cost = 1 << 30;
  for (int a = 4; a <= 20; a += 2) {
    if (!is_first(a) || L % a) continue;
    const int m = L / a;
    if (is_radix(m) && m <= cap) {
      const int mx = a > m ? a : m;
      const int c = mx * 100 + m;
      if (c < cost) {
        cost = c;
        best = {a, 1, m};
      }
    }
  }
  if (best.r1) return best;
  for (int a = 4; a <= 20; a += 2) {
    if (!is_first(a) || L % a) continue;
    for (int b = 2; b <= 20; ++b) {
      if (!is_radix(b) || (L / a) % b) continue;
      const int m = L / a / b;
      if (!is_radix(m) || m > cap) continue;
      const int mx = a > b ? (a > m ? a : m) : (b > m ? b : m);
      // single lines: the smallest sum of the radices; three components: the
      // smallest last radix (the most threads a column)
      const int c = mx * 10000 + (cap == 20 ? (a + b + m) * 100 + m : m * 100 + (a > b ? a - b : b - a));
      if (c < cost) {
        cost = c;
        best = {a, b, m};
      }
    }
  }
  return best;
}

// last radix of the three-component kernels (8000 = 20^3 has no smaller one)
constexpr int cap3(bool f64, int L) { return f64 ? 10 : (radices(L, 16).r1 ? 16 : 20); }

template <typename R_, int L_, int CAP = 20> struct Plan {
  using R = R_;
  using C = cplx_t<R>;
  static constexpr Radices f = radices(L_, CAP);
  static constexpr int L = L_, R1 = f.r1, R2 = f.r2, R3 = f.r3;
  static_assert(R1 * R2 * R3 == L, "length without a plan");
  static constexpr int H1 = R1 / 2;
  static constexpr int M = R1 * R2;  // butterflies of S3
  static constexpr int NB1 = R2 * R3, NB2 = R1 * R3, NB3 = M;
  static constexpr int RMAX = R1 > R2 ? (R1 > R3 ? R1 : R3) : (R2 > R3 ? R2 : R3);
  // entries of the twiddle tables
  static constexpr int NTW2 = (R2 - 1) * R1, NTW3 = (R3 - 1) * M;
  // shared addresses: odd q stride, and an r stride that continues the k run
  // of the next r in the banks (B values of 128 bytes)
  static constexpr int B = 128 / static_cast<int>(sizeof(C));
  static constexpr int PA = R1 | 1;
  static constexpr int PB = R3 * PA + (((R1 - R3 * PA) % B) + B) % B;
  static constexpr int SIZE = R2 > 1 ? R2 * PB : R3 * PA;  // values of one line
};

// ----------------------------------------------------------------- stages ---
// LF (line fastest): NL lines interleaved, element a of line l at a * NL + l,
// butterfly tasks t = i * NL + l; else line l at l * LS + a, t = l * NB + i.
template <class P, int NL, int NT, bool LF> struct Lines {
  using C = typename P::C;
  // interleaved lines fill the banks by themselves: no r padding
  static constexpr int PB = LF ? P::R3 * P::PA : P::PB;
  static constexpr int SIZE = LF ? P::R2 * PB : P::SIZE;
  static constexpr int LS = SIZE + ((P::M - SIZE) % P::B + P::B) % P::B;  // line stride (position fastest)
  static constexpr int kValues = LF ? SIZE * NL : LS * NL;               // shared values of a block
  static __device__ __forceinline__ int at(int line, int a) { return LF ? a * NL + line : line * LS + a; }
  static constexpr int st = LF ? NL : 1;  // stride of an address step

  template <int NB> static __device__ __forceinline__ void split(int t, int& line, int& i) {
    if (LF) {
      line = t % NL;
      i = t / NL;
    } else {
      line = t / NB;
      i = t - line * NB;
    }
  }

  // S1: ld(line, i1, v) gives the R1/2 inputs x[i1 + a NB1] of a line
  template <class LD> static __device__ __forceinline__ void s1(C* sm, const LD& ld) {
#pragma unroll 2
    for (int t = threadIdx.x; t < NL * P::NB1; t += NT) {
      int line, i;
      split<P::NB1>(t, line, i);
      C v[P::R1];
      ld(line, i, v);
      dft_half_in<P::R1>(v);
      const int r = i / P::R3, q = i - r * P::R3;
      C* d = sm + at(line, r * PB + q * P::PA);
#pragma unroll
      for (int k = 0; k < P::R1; ++k) d[k * st] = v[k];
    }
  }
  // S1 of the inverse: sto(line, i1, v) takes the R1/2 outputs y[i1 + a NB1]
  template <class ST> static __device__ __forceinline__ void s1_inv(const C* sm, const ST& sto) {
#pragma unroll 2
    for (int t = threadIdx.x; t < NL * P::NB1; t += NT) {
      int line, i;
      split<P::NB1>(t, line, i);
      const int r = i / P::R3, q = i - r * P::R3;
      const C* d = sm + at(line, r * PB + q * P::PA);
      C v[P::R1];
#pragma unroll
      for (int k = 0; k < P::R1; ++k) v[k] = d[k * st];
      dft_half_out<P::R1>(v);
      sto(line, i, v);
    }
  }
  // S2, in place (with the barrier that follows it)
  template <bool INV> static __device__ __forceinline__ void s2(C* sm, const C* __restrict__ tw2) {
    if constexpr (P::R2 > 1) {
#pragma unroll 2
      for (int t = threadIdx.x; t < NL * P::NB2; t += NT) {
        int line, i;
        split<P::NB2>(t, line, i);
        const int q = i / P::R1, k = i - q * P::R1;
        C* d = sm + at(line, q * P::PA + k);
        C v[P::R2];
#pragma unroll
        for (int r = 0; r < P::R2; ++r) v[r] = d[r * PB * st];
        if (INV) dft<P::R2, true>(v);
#pragma unroll
        for (int r = 1; r < P::R2; ++r) {
          const C w = __ldg(tw2 + (r - 1) * P::R1 + k);
          v[r] = cmul(v[r], INV ? cconj(w) : w);
        }
        if (!INV) dft<P::R2, false>(v);
#pragma unroll
        for (int r = 0; r < P::R2; ++r) d[r * PB * st] = v[r];
      }
      __syncthreads();
    }
  }
  // the shared values of S3 butterfly i3 of a line: base address, q stride PA
  static __device__ __forceinline__ C* s3_base(C* sm, int line, int i3) {
    const int r = i3 / P::R1, k = i3 - r * P::R1;
    return sm + at(line, r * PB + k);
  }
  static __device__ __forceinline__ void s3(const C* d, int i3, const C* __restrict__ tw3, C* v) {
#pragma unroll
    for (int q = 0; q < P::R3; ++q) v[q] = d[q * P::PA * st];
#pragma unroll
    for (int q = 1; q < P::R3; ++q) v[q] = cmul(v[q], __ldg(tw3 + (q - 1) * P::M + i3));
    dft<P::R3, false>(v);
  }
  static __device__ __forceinline__ void s3_inv(C* d, int i3, const C* __restrict__ tw3, C* v) {
    dft<P::R3, true>(v);
#pragma unroll
    for (int q = 1; q < P::R3; ++q) v[q] = cmul(v[q], cconj(__ldg(tw3 + (q - 1) * P::M + i3)));
#pragma unroll
    for (int q = 0; q < P::R3; ++q) d[q * P::PA * st] = v[q];
  }
};

// registers a thread of a kernel is given: blocks an SM so that they fit
constexpr int blocks_for(int nt, int regs, size_t smem) {
  int b = 65536 / (((nt + 31) / 32 * 32) * regs);
  const int s = smem > 0 ? static_cast<int>(227 * 1024 / (smem + 1024)) : 32;
  b = b < s ? b : s;
  const int w = 2048 / ((nt + 31) / 32 * 32);
  b = b < w ? b : w;
  return b < 1 ? 1 : (b > 16 ? 16 : b);
}
template <typename R> constexpr int regs_for(int values) {  // values: complex values held at once
  const int w = sizeof(R) == 4 ? 1 : 2;
  const int r = 36 + 2 * w * values + (w == 2 ? 16 : 0);
  return r > 240 ? 240 : (r < 48 ? 48 : r);
}

}  // namespace rf

// lengths with an instantiation, ascending: even 5-smooth lengths the radices
// reach, so close that from 100 to 4096 points padding a line to the next one
// costs at most 12.5 % (3 % on average; mm_rf.cu checks the bound), below 100
// points up to 23 %, beyond 4096 (FP32 film columns) up to 25 %
#define MM_RF_LENGTHS_A(X) X(12) X(16) X(20) X(24) X(30) X(32) X(36) X(40) X(48) X(50) X(60) X(64) X(72) X(80) X(90) X(96) X(100)
#define MM_RF_LENGTHS_B(X) X(108) X(120) X(128) X(144) X(150) X(160) X(180) X(192) X(200) X(216) X(240) X(250) X(256)
#define MM_RF_LENGTHS_C(X) X(288) X(300) X(320) X(360) X(384) X(400) X(432) X(450) X(480) X(500) X(512) X(540) X(576) X(600)
#define MM_RF_LENGTHS_D(X) X(640) X(720) X(768) X(800) X(864) X(900) X(960) X(1000) X(1024) X(1080) X(1152) X(1200)
#define MM_RF_LENGTHS_E(X) X(1280) X(1350) X(1440) X(1536) X(1600) X(1728) X(1800) X(1920) X(2000) X(2048)
#define MM_RF_LENGTHS_F(X) X(2160) X(2304) X(2400) X(2560) X(2700) X(2880) X(3072) X(3200) X(3600) X(3840) X(4000) X(4096)
#define MM_RF_XY(X)                                                                                           \
  MM_RF_LENGTHS_A(X) MM_RF_LENGTHS_B(X) MM_RF_LENGTHS_C(X) MM_RF_LENGTHS_D(X) MM_RF_LENGTHS_E(X) MM_RF_LENGTHS_F(X)
// film columns beyond 4096
#define MM_RF_LENGTHS_G(X) X(4800) X(5120) X(6000) X(6400) X(8000)

}  // namespace mm
