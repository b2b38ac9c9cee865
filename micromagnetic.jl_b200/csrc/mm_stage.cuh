// mm_stage.cuh -- the per-cell stage kernel (field, right-hand side, energies,
// fixed and adaptive Runge-Kutta stages) and its compiled term sets (internal).
#pragma once
#include <cmath>

#include "mm_cell.cuh"
#include "mm_field.cuh"
#include "mm_launch.cuh"

namespace mm {

// Butcher tables of the adaptive methods (src/integrator/adaptive_rk_steps.jl:
// bs23 11-47, dopri54 49-107, cashkarp54 110-168, fehlberg54 171-229), laid
// out as RkTableau: rows a[s-1] give the input of stage s+1; row sol-1 is the
// solution; w are the error weights.
#define MM_RK_TABLES                                                                                          \
  {                                                                                                           \
    {7, 6, 7, 0, 5, 4,                                                                                        \
     {{1.0 / 5},                                                                                              \
      {3.0 / 40, 9.0 / 40},                                                                                   \
      {44.0 / 45, -56.0 / 15, 32.0 / 9},                                                                      \
      {19372.0 / 6561, -25360.0 / 2187, 64448.0 / 6561, -212.0 / 729},                                        \
      {9017.0 / 3168, -355.0 / 33, 46732.0 / 5247, 49.0 / 176, -5103.0 / 18656},                              \
      {35.0 / 384, 0, 500.0 / 1113, 125.0 / 192, -2187.0 / 6784, 11.0 / 84}},                                 \
     {71.0 / 57600, 0, -71.0 / 16695, 71.0 / 1920, -17253.0 / 339200, 22.0 / 525, -1.0 / 40}},               \
    {4, 3, 4, 1, 3, 2,                                                                                        \
     {{0.5}, {0, 0.75}, {2.0 / 9, 1.0 / 3, 4.0 / 9}},                                                         \
     {-5.0 / 72, 1.0 / 12, 1.0 / 9, -1.0 / 8}},                                                               \
    {6, 6, 6, 0, 5, 4,                                                                                        \
     {{1.0 / 5},                                                                                              \
      {3.0 / 40, 9.0 / 40},                                                                                   \
      {3.0 / 10, -9.0 / 10, 6.0 / 5},                                                                         \
      {-11.0 / 54, 5.0 / 2, -70.0 / 27, 35.0 / 27},                                                           \
      {1631.0 / 55296, 175.0 / 512, 575.0 / 13824, 44275.0 / 110592, 253.0 / 4096},                           \
      {37.0 / 378, 0, 250.0 / 621, 125.0 / 594, 0, 512.0 / 1771}},                                            \
     {-277.0 / 64512, 0, 6925.0 / 370944, -6925.0 / 202752, -277.0 / 14336, 277.0 / 7084}},                  \
    {6, 6, 6, 0, 5, 4,                                                                                        \
     {{1.0 / 4},                                                                                              \
      {3.0 / 32, 9.0 / 32},                                                                                   \
      {1932.0 / 2197, -7200.0 / 2197, 7296.0 / 2197},                                                         \
      {439.0 / 216, -8.0, 3680.0 / 513, -845.0 / 4104},                                                       \
      {-8.0 / 27, 2.0, -3544.0 / 2565, 1859.0 / 4104, -11.0 / 40},                                            \
      {16.0 / 135, 0, 6656.0 / 12825, 28561.0 / 56430, -9.0 / 50, 2.0 / 55}},                                 \
     {-1.0 / 360, 0, 128.0 / 4275, 2197.0 / 75240, -1.0 / 50, -2.0 / 55}},                                    \
  }

static __constant__ RkTableau c_rk[RK_NMETHODS] = MM_RK_TABLES;

template <typename R, int MODE, bool EXTRA, unsigned FIX = 0>
__global__ void __launch_bounds__(kStageThreads, sizeof(R) == 4 ? 3 : 2) k_stage(FieldArgs<R> a, const R* __restrict__ y, StageArgs<R> s) {
  constexpr bool kF32 = sizeof(R) == 4;
  pdl_enter();
  if (MODE == SM_DOPRI && !s.ctrl->active) return;
  if (MODE == SM_FIELD && s.gate && !*s.gate) return;
  const int64_t N = a.N;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int k = blockIdx.z;
  const bool live = i < a.nx && j < a.ny;
  const int I = (k * a.ny + j) * a.nx + i;
  const int tid = threadIdx.y * blockDim.x + threadIdx.x;
  const int blin = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
  double e[kNTerms];
  R m[3], h[3];
  double red = 0.0;  // SM_DOPRI stage 7: error max
  // RK4 operands of this cell, loaded together with the field inputs
  R mN[3], mL[3], av[3];
  if (MODE == SM_RK4 && live) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      mN[c] = s.m[c * N + I];
      mL[c] = kF32 ? s.m_lo[c * N + I] : R(0);
      av[c] = s.stage > 1 ? s.acc[c * N + I] : R(0);
    }
  }
  // FSAL: stage 1 takes k1 from the last stage of the accepted attempt
  const bool reuse = MODE == SM_DOPRI && s.stage == 1 && !s.ctrl->eval1;
  // SM_DOPRI operands of this cell: the start state, and the earlier slopes
  // with a non-zero coefficient in this stage's sums.  Loaded together with
  // the field inputs (walking the tableau row after the field, one dependent
  // load a term, took 0.270 ms a stage on 256x256x64 FP32 against 0.07 ms of
  // traffic).
  R kv[6][3];
  R co[6];  // a[st-1][j] h (zero: not part of the sum)
  if constexpr (MODE == SM_DOPRI) {
    const RkTableau& tb = c_rk[s.method];
    const int st = s.stage;
    const double hstep = s.ctrl->step;
    const bool sum = st <= tb.sol, err = st == tb.err;
#pragma unroll
    for (int j = 0; j < 6; ++j) co[j] = static_cast<R>(sum && j < st ? tb.a[st - 1][j] * hstep : 0.0);
    if (live) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        mN[c] = sum ? s.m[c * N + I] : R(0);
        mL[c] = kF32 && sum ? s.m_lo[c * N + I] : R(0);
      }
#pragma unroll
      for (int j = 0; j < 6; ++j) {
        const bool need = j < st - 1 && (co[j] != R(0) || (err && tb.w[j] != 0.0));
#pragma unroll
        for (int c = 0; c < 3; ++c) kv[j][c] = need ? s.k[j][c * N + I] : R(0);
      }
    }
  }
  if (live) {
    if (!reuse) cell_heff<R, MODE == SM_ENERGY || MODE == SM_FIELD, EXTRA, false, FIX>(a, y, I, i, j, k, m, h, e);
    if (MODE == SM_FIELD) {
      s.out[I] = h[0];
      s.out[N + I] = h[1];
      s.out[2 * N + I] = h[2];
      if (s.ecell) {
        double et = 0.0;
#pragma unroll
        for (int t = 0; t < kNTerms; ++t) et += e[t];
        s.ecell[I] = static_cast<R>(et);
      }
    } else if (MODE == SM_RHS) {
      R f[3];
      llg_rhs(a, I, m, h, f);
      s.out[I] = f[0];
      s.out[N + I] = f[1];
      s.out[2 * N + I] = f[2];
    } else if (MODE == SM_RK4) {
      rk4_update(a, s, I, m, h, mN, mL, av);
    } else if (MODE == SM_DOPRI) {
      // rk_step_bs23! / rk_step_dopri54! / rk_step_cashkarp54! /
      // rk_step_fehlberg54!  src/integrator/adaptive_rk_steps.jl:11-229
      const RkTableau& tb = c_rk[s.method];
      const int st = s.stage;
      R f[3];
      if (reuse) {
#pragma unroll
        for (int c = 0; c < 3; ++c) f[c] = s.k[tb.nstage - 1][c * N + I];
      } else {
        llg_rhs(a, I, m, h, f);
      }
      if (st < tb.err || (tb.fsal && st == tb.nstage)) {
#pragma unroll
        for (int c = 0; c < 3; ++c) s.k[st - 1][c * N + I] = f[c];
      }
      R yabs[3];  // y_next of the error norm
      if (st <= tb.sol) {
        R v[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          R acc = kF32 ? R(0) : mN[c];
#pragma unroll
          for (int j = 0; j < 6; ++j) {
            if (co[j] == R(0)) continue;
            const R kj = j == st - 1 ? f[c] : kv[j][c];
            acc = acc + co[j] * kj;
          }
          v[c] = acc;
        }
        if (st < tb.sol) {
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            if constexpr (kF32) v[c] = mN[c] + (mL[c] + v[c]);
            s.ynext[c * N + I] = v[c];
          }
        } else {
          // the solution is normalised before it is used (adaptive_rk_steps.jl:35,96,156,217)
          if constexpr (kF32) {
            float hi[3], lo[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
              hi[c] = mN[c];
              lo[c] = mL[c];
              df_add(hi[c], lo[c], v[c]);
            }
            df_normalise(hi, lo);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
              s.ynext[c * N + I] = hi[c];
              s.ynext_lo[c * N + I] = lo[c];
              yabs[c] = hi[c];
            }
          } else {
            plain_normalise(v);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
              s.ynext[c * N + I] = v[c];
              yabs[c] = v[c];
            }
          }
        }
      } else {
#pragma unroll
        for (int c = 0; c < 3; ++c) yabs[c] = m[c];
      }
      if (st == tb.err) {
        // error estimate: max |sum_j w_j k_j| / (1 + |y_next|)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          double et = 0.0;
#pragma unroll
          for (int j = 0; j < 7; ++j) {
            if (j >= st || tb.w[j] == 0.0) continue;
            const double kj = j == st - 1 || j == 6 ? double(f[c]) : double(kv[j < 6 ? j : 0][c]);
            et += tb.w[j] * kj;
          }
          const double v = fabs(et / (1.0 + fabs(double(yabs[c]))));
          red = (v > red || isnan(v)) ? v : red;
        }
      }
    }
  }
  if (MODE == SM_ENERGY || (MODE == SM_DOPRI && s.stage == c_rk[s.method].err)) {
    // deterministic block reduction in FP64
    __shared__ double sh[kStageThreads / 32][kNTerms];
    const int lane = tid & 31, warp = tid >> 5;
    constexpr int W = MODE == SM_ENERGY ? kNTerms : 1;
    double v[W];
#pragma unroll
    for (int t = 0; t < W; ++t) v[t] = live ? (MODE == SM_ENERGY ? e[t] : red) : 0.0;
#pragma unroll
    for (int t = 0; t < W; ++t) {
      for (int o = 16; o > 0; o >>= 1) {
        const double u = __shfl_down_sync(0xffffffffu, v[t], o);
        if (MODE == SM_ENERGY) v[t] += u;
        else v[t] = (u > v[t] || isnan(u)) ? u : v[t];
      }
      if (lane == 0) sh[warp][t] = v[t];
    }
    __syncthreads();
    if (tid < W) {
      double acc = 0.0;
      for (int w = 0; w < kStageThreads / 32; ++w) {
        const double u = sh[w][tid];
        if (MODE == SM_ENERGY) acc += u;
        else acc = (u > acc || isnan(u)) ? u : acc;
      }
      s.partials[blin * W + tid] = acc;
    }
  }
}

// Field of one cell of a compiled term set from values in registers (the
// expressions of cell_heff, in its order).
template <typename R, unsigned FIX>
__device__ __forceinline__ void fix_heff(const FieldArgs<R>& a, const R m[3], const R mn[6][3], R Ms, unsigned nbm,
                                         const R hd[3], R h[3]) {
  h[0] = h[1] = h[2] = R(0);
  if (Ms != R(0)) {
    const R Ms_inv = R(1) / Ms;
    {
      R fx = 0, fy = 0, fz = 0;
      const R coef[6] = {a.ex_x, a.ex_x, a.ex_y, a.ex_y, a.ex_z, a.ex_z};
#pragma unroll
      for (int d = 0; d < 6; ++d) {
        if ((nbm >> d) & 1u) {
          const R c = coef[d];
          fx += c * (mn[d][0] - m[0]);
          fy += c * (mn[d][1] - m[1]);
          fz += c * (mn[d][2] - m[2]);
        }
      }
      h[0] += fx * Ms_inv;
      h[1] += fy * Ms_inv;
      h[2] += fz * Ms_inv;
    }
    if (FIX & TB_DMI_BULK) {
      R fx = 0, fy = 0, fz = 0;
      if (nbm & 1u) { fy += a.bd_x * (-mn[0][2]); fz += a.bd_x * mn[0][1]; }
      if (nbm & 2u) { fy += a.bd_x * mn[1][2]; fz += a.bd_x * (-mn[1][1]); }
      if (nbm & 4u) { fx += a.bd_y * mn[2][2]; fz += a.bd_y * (-mn[2][0]); }
      if (nbm & 8u) { fx += a.bd_y * (-mn[3][2]); fz += a.bd_y * mn[3][0]; }
      if (nbm & 16u) { fx += a.bd_z * (-mn[4][1]); fy += a.bd_z * mn[4][0]; }
      if (nbm & 32u) { fx += a.bd_z * mn[5][1]; fy += a.bd_z * (-mn[5][0]); }
      h[0] += fx * Ms_inv;
      h[1] += fy * Ms_inv;
      h[2] += fz * Ms_inv;
    }
    if ((FIX & TB_DMI_INTERFACIAL) && a.D_uni != R(0)) {
      R fx = 0, fy = 0, fz = 0;
      const R cx = a.D_uni * a.id_x, cy = a.D_uni * a.id_y;
      if (nbm & 1u) { fx += cx * mn[0][2]; fz += cx * (-mn[0][0]); }
      if (nbm & 2u) { fx += cx * (-mn[1][2]); fz += cx * mn[1][0]; }
      if (nbm & 4u) { fy += cy * mn[2][2]; fz += cy * (-mn[2][1]); }
      if (nbm & 8u) { fy += cy * (-mn[3][2]); fz += cy * mn[3][1]; }
      h[0] += fx * Ms_inv;
      h[1] += fy * Ms_inv;
      h[2] += fz * Ms_inv;
    }
    if (FIX & TB_ANIS) {
      const R inv2 = R(2) / Ms;
      const R sa = m[0] * a.ux + m[1] * a.uy + m[2] * a.uz;
      h[0] += a.Ku_uni * sa * a.ux * inv2;
      h[1] += a.Ku_uni * sa * a.uy * inv2;
      h[2] += a.Ku_uni * sa * a.uz * inv2;
    }
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) h[c] += hd[c];
  if (FIX & TB_ZEEMAN) {
    h[0] += a.hz_x;
    h[1] += a.hz_y;
    h[2] += a.hz_z;
  }
}

// RK4 / Heun stage of the compiled term sets, two x-neighbouring cells a thread
// (FP32, nx even: every row of every array starts on 8 bytes): all arrays but
// the two outer x neighbours move as 8-byte values, and the cells share their
// index arithmetic.
struct PairOut {  // the written values of one cell, to leave with its neighbour's
  float k[3], a[3], y[3], n[3], l[3];
  __device__ __forceinline__ void slope(int c, float v) { k[c] = v; }
  __device__ __forceinline__ void acc(int c, float v) { a[c] = v; }
  __device__ __forceinline__ void ynext(int c, float v) { y[c] = v; }
  __device__ __forceinline__ void m(int c, float v) { n[c] = v; }
  __device__ __forceinline__ void m_lo(int c, float v) { l[c] = v; }
};
template <unsigned FIX>
struct StagePair {
  static constexpr int kNT = 128, kMinB = 5;
  using Args = typename StagePlain<float, FIX>::Args;  // bx counts pairs
  static __device__ __forceinline__ void body(const Args& args, uint3 blockIdx) {
    const FieldArgs<float>& a = args.a;
    const StageArgs<float>& s = args.s;
    const float* __restrict__ y = args.y;
    const int N = static_cast<int>(a.N), nx = a.nx, ny = a.ny, nz = a.nz, nxy = nx * ny;
    const int tid = threadIdx.x, bx = args.bx;  // a power of two
    const int i = 2 * (blockIdx.x * bx + (tid & (bx - 1)));
    const int j = blockIdx.y * args.by + (tid >> (__ffs(bx) - 1));
    const int k = blockIdx.z;
    if (i >= nx || j >= ny) return;
    const int I = (k * ny + j) * nx + i;
    const bool px = a.pbc & 1, py = a.pbc & 2, pz = a.pbc & 4;
    const int il = i > 0 ? I - 1 : (px ? I + nx - 1 : I);
    const int ir = i + 2 < nx ? I + 2 : (px ? I + 2 - nx : I);
    const int nb[4] = {j > 0 ? I - nx : (py ? I + (ny - 1) * nx : I), j < ny - 1 ? I + nx : (py ? I - (ny - 1) * nx : I),
                       k > 0 ? I - nxy : (pz ? I + (nz - 1) * nxy : I),
                       k < nz - 1 ? I + nxy : (pz ? I - (nz - 1) * nxy : I)};
    auto ld = [](const float* p, int64_t o) { return *reinterpret_cast<const float2*>(p + o); };
    float2 c0[3], nn[4][3], mN[3], mL[3], av[3], hd[3];
    float xl[3], xr[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int64_t o = static_cast<int64_t>(c) * N;
      c0[c] = __ldg(reinterpret_cast<const float2*>(y + o + I));
      xl[c] = __ldg(y + o + il);
      xr[c] = __ldg(y + o + ir);
#pragma unroll
      for (int d = 0; d < 4; ++d) nn[d][c] = __ldg(reinterpret_cast<const float2*>(y + o + nb[d]));
      mN[c] = ld(s.m, o + I);
      mL[c] = ld(s.m_lo, o + I);
      av[c] = s.stage > 1 ? ld(s.acc, o + I) : make_float2(0.f, 0.f);
      hd[c] = ld(a.Hd, o + I);
    }
    const float2 Ms = __ldg(reinterpret_cast<const float2*>(a.Ms + I));
    const uchar2 nm = __ldg(reinterpret_cast<const uchar2*>(a.nbm + I));
    PairOut out[2];
#pragma unroll
    for (int w = 0; w < 2; ++w) {
      auto at = [w](float2 v) { return w ? v.y : v.x; };
      float m[3], mn[6][3], h[3], d3[3], n3[3], l3[3], a3[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        m[c] = at(c0[c]);
        mn[0][c] = w ? c0[c].x : xl[c];
        mn[1][c] = w ? xr[c] : c0[c].y;
#pragma unroll
        for (int d = 0; d < 4; ++d) mn[2 + d][c] = at(nn[d][c]);
        d3[c] = at(hd[c]);
        n3[c] = at(mN[c]);
        l3[c] = at(mL[c]);
        a3[c] = at(av[c]);
      }
      fix_heff<float, FIX>(a, m, mn, at(Ms), w ? nm.y : nm.x, d3, h);
      rk4_update_to(a, s, I + w, m, h, n3, l3, a3, out[w]);
    }
    float* const kout = s.scheme == 1 ? nullptr : s.k[s.stage - 1];
    const bool last = s.stage == (s.scheme == 1 ? 2 : 4);
    auto sto = [](float* p, int64_t o, float u, float v) { *reinterpret_cast<float2*>(p + o) = make_float2(u, v); };
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int64_t o = static_cast<int64_t>(c) * N + I;
      if (kout) sto(kout, o, out[0].k[c], out[1].k[c]);
      if (last) {
        sto(s.m, o, out[0].n[c], out[1].n[c]);
        sto(s.m_lo, o, out[0].l[c], out[1].l[c]);
      } else {
        sto(s.acc, o, out[0].a[c], out[1].a[c]);
        sto(s.ynext, o, out[0].y[c], out[1].y[c]);
      }
    }
  }
};

// Term sets with compiled stage kernels: exchange + demag with at most one DMI
// and any of anisotropy and Zeeman, all parameters uniform -- what films and
// boxes are built from.  The general kernel reads the mask and tests every
// per-cell array a term may have.
constexpr unsigned kFixBase = TB_EXCH | TB_DEMAG;
#define MM_FIX_SETS(X)                                                                                                \
  X(kFixBase) X(kFixBase | TB_ANIS) X(kFixBase | TB_ZEEMAN) X(kFixBase | TB_ANIS | TB_ZEEMAN)                         \
  X(kFixBase | TB_DMI_BULK) X(kFixBase | TB_DMI_BULK | TB_ANIS) X(kFixBase | TB_DMI_BULK | TB_ZEEMAN)                 \
  X(kFixBase | TB_DMI_BULK | TB_ANIS | TB_ZEEMAN) X(kFixBase | TB_DMI_INTERFACIAL)                                    \
  X(kFixBase | TB_DMI_INTERFACIAL | TB_ANIS) X(kFixBase | TB_DMI_INTERFACIAL | TB_ZEEMAN)                             \
  X(kFixBase | TB_DMI_INTERFACIAL | TB_ANIS | TB_ZEEMAN)

// Launches the compiled kernel of fa's term set; false when it has none.
template <typename R>
bool launch_rk4_fix(const FieldArgs<R>& fa, const R* y, const StageArgs<R>& sa, const StageGrid& g, cudaStream_t st);
template <typename R>
bool launch_dopri_fix(const FieldArgs<R>& fa, const R* y, const StageArgs<R>& sa, const StageGrid& g, cudaStream_t st);

}  // namespace mm
