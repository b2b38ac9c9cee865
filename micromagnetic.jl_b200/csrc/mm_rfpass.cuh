// mm_rfpass.cuh -- the demag FFT passes on compile-time line lengths
// (mm_rfft.cuh) as launch descriptors: forward / inverse x, forward / inverse
// y of 3-D meshes, the z convolution and the fused film column (internal).
//
// Measured against the run-time-length passes (mm_passes.cuh) they replace for
// meshes of 8192 cells and more, per launch (cold caches, FP32 unless noted):
// film column of 1000 x 1000 (2000 points) 105 -> 40 us, its x passes 44 / 45 ->
// 24 / 19; 300 x 200 x 20: z convolution (40 points) 165 -> 55, y passes 43 ->
// 23, x passes 50 / 44 -> 28 / 16; 150 x 126 x 37 FP64: z (80 points) 166 -> 68,
// y 56 -> 22, x 39 / 34 -> 35 / 28; 4000 x 4000 film columns (8000 points) 7 global
// round trips and a product, 2.7 ms, -> one pass, 0.73 ms.  What bounds them
// now: instruction issue (57 % active in the 2000-point columns, 71 % in the
// 40-point z convolution), latency at one block an SM for the 8000-point columns
// (19 warps), HBM and issue together for the y passes of meshes beyond L2 (0.6 of
// the measured bandwidth).
//
// One kernel serves a mesh launched alone and several meshes of a batch in one
// launch (k_rf): its few arguments are copied to registers, from the
// parameters or from the batch's table.
#pragma once
#include "mm_demag.cuh"
#include "mm_launch.cuh"
#include "mm_rfft.cuh"

namespace mm {
namespace rf {

template <class K>
__global__ void __launch_bounds__(K::kNT, K::kMinB) k_rf(const typename K::Args inl, const typename K::Args* __restrict__ arr,
                                                         const int* __restrict__ begins, int n) {
  pdl_enter();
  int b = static_cast<int>(blockIdx.x);
  if (n == 0) {
    K::body(inl, b);
    return;
  }
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (begins[mid] <= b) lo = mid;
    else hi = mid - 1;
  }
  const typename K::Args a = arr[lo];
  K::body(a, b - begins[lo]);
}

template <class K>
cudaError_t launch_many_rf(const void* args_dev, const int* begins_dev, int n, int blocks, size_t smem, cudaStream_t st) {
  if (smem > 48 * 1024) smem_optin(reinterpret_cast<const void*>(&k_rf<K>));
  k_rf<K><<<blocks, K::kNT, smem, st>>>(typename K::Args{}, static_cast<const typename K::Args*>(args_dev), begins_dev, n);
  return cudaGetLastError();
}

template <class K>
void launch_rf(int blocks, cudaStream_t st, const typename K::Args& a) {
  if (LaunchRecorder* r = launch_recorder()) {
    LaunchRec rec;
    rec.kind = reinterpret_cast<const void*>(&k_rf<K>);
    rec.pkind = -1;
    rec.grid = dim3(blocks);
    rec.many = &launch_many_rf<K>;
    rec.args_size = sizeof(a);
    rec.args.resize(sizeof(a));
    std::memcpy(rec.args.data(), &a, sizeof(a));
    rec.blocks = blocks;
    rec.smem = K::kSmem;
    r->recs.push_back(std::move(rec));
    return;
  }
  if (K::kSmem > 48 * 1024) smem_optin(reinterpret_cast<const void*>(&k_rf<K>));
  launch_pdl(k_rf<K>, dim3(blocks), dim3(K::kNT), K::kSmem, st, a, static_cast<const typename K::Args*>(nullptr),
             static_cast<const int*>(nullptr), 0);
}

template <typename C> __device__ __forceinline__ C* dyn_smem() {
  extern __shared__ __align__(16) unsigned char rf_smem_raw[];
  return reinterpret_cast<C*>(rf_smem_raw);
}

// Threads a line of a single-component kernel: the rounds n of S3 butterflies a
// thread that leave the most warps resident (registers by regs_for; hold: the
// x passes keep n R3 values across a barrier), fewer rounds where that is within
// 10 %.  1024 points FP64, 4 lines: 256 threads (2 blocks an SM) 61 / 52 us
// against 344 threads (1 block) 71 / 65 (1024 x 2048 rows).
template <class P> constexpr int line_threads(int lines, bool hold, size_t smem) {
  int best = 0, warps = 0;
  for (int n = 1; n <= 8; ++n) {
    const int tl = (P::NB3 + n - 1) / n, nt = (tl * lines + 31) / 32 * 32;
    const int v = hold && n * P::R3 > P::RMAX ? n * P::R3 : P::RMAX;
    const int regs = regs_for<typename P::R>(v);
    if (nt > 1024 || nt * regs > 65536) continue;
    const int b = blocks_for(nt, regs, smem);
    const int w = b * nt / 32 - (b == 1 ? 8 : 0);  // a lone block's barriers idle its SM
    if (best == 0 || 10 * w > 11 * warps) {
      best = tl;
      warps = w;
    }
  }
  return best > 0 ? best : (P::NB3 + 7) / 8;
}

// ------------------------------------------------------------- x passes ---
// G lines (rows of one component) a block, line fastest: the lanes of a warp
// cover G rows x 32/G positions, so rows are read in 64-byte runs and a
// column-major X (films) is written in G-row segments (32 bytes for G = 4
// FP32 / 2 FP64).
// More lines a block do not pay: each line is an independent chain, and on small
// meshes (200 x 50: 150 lines) more, shorter blocks finish sooner.
template <typename R> constexpr int x_lines(int L) {
  return L <= 128 ? 8 : (sizeof(R) == 4 || L <= 1024 ? 4 : 2);
}

template <typename R, int L> struct XPass {
  using P = Plan<R, L>;
  using C = typename P::C;
  static constexpr int G = x_lines<R>(L);
  static constexpr size_t kSmem = sizeof(C) * Lines<P, G, 1, true>::kValues;
  static constexpr int TL = line_threads<P>(G, true, kSmem), kNT = G * TL;
  static constexpr int NJ3 = (P::NB3 + TL - 1) / TL;
  using S = Lines<P, G, kNT, true>;
  static constexpr int kMinB = blocks_for(kNT, regs_for<R>(P::RMAX > NJ3 * P::R3 ? P::RMAX : NJ3 * P::R3), kSmem);
};

// real rows m * Ms (zero padded to 2 L) -> half spectrum
template <typename R, int L> struct FwdX : XPass<R, L> {
  using B = XPass<R, L>;
  using P = typename B::P;
  using C = typename B::C;
  using S = typename B::S;
  struct Args {
    const R* m;
    const R* Ms;
    C* X;
    const C *tw2, *tw3, *twx;
    const int* gate;
    int nx, rows, cols;  // cols: X column-major
  };
  static __device__ __forceinline__ void body(const Args& a, int blk) {
    if (a.gate && !*a.gate) return;
    C* sm = dyn_smem<C>();
    const int g = threadIdx.x % B::G;
    const int line = blk * B::G + g;
    const bool live = line < 3 * a.rows;
    const int c = live ? line / a.rows : 0, row = live ? line - c * a.rows : 0;
    const int nx = a.nx;
    const int64_t N = static_cast<int64_t>(a.rows) * nx;
    const R* mr = a.m + c * N + static_cast<int64_t>(row) * nx;
    const R* Mr = a.Ms + static_cast<int64_t>(row) * nx;
    const bool even = !(nx & 1);
    S::s1(sm, [&](int, int i1, C* v) {
      // every load is issued before any product waits for one
      C p[P::H1], s[P::H1];
#pragma unroll
      for (int q = 0; q < P::H1; ++q) {
        const int u = 2 * (i1 + q * P::NB1);
        p[q] = s[q] = cmk<C>(R(0), R(0));
        if (even) {
          if (live && u < nx) {
            p[q] = *reinterpret_cast<const C*>(mr + u);
            s[q] = __ldg(reinterpret_cast<const C*>(Mr + u));
          }
        } else {
          if (live && u < nx) {
            p[q].x = mr[u];
            s[q].x = __ldg(Mr + u);
          }
          if (live && u + 1 < nx) {
            p[q].y = mr[u + 1];
            s[q].y = __ldg(Mr + u + 1);
          }
        }
      }
#pragma unroll
      for (int q = 0; q < P::H1; ++q) v[q] = cmk<C>(p[q].x * s[q].x, p[q].y * s[q].y);
    });
    __syncthreads();
    S::template s2<false>(sm, a.tw2);
    const int tl = threadIdx.x / B::G;
    C v[B::NJ3][P::R3];
#pragma unroll
    for (int j = 0; j < B::NJ3; ++j) {
      const int i3 = tl + j * B::TL;
      if (i3 < P::NB3) {
        C* d = S::s3_base(sm, g, i3);
        S::s3(d, i3, a.tw3, v[j]);
        // Z in place: frequency i3 + q M in the slot of (i3, q)
#pragma unroll
        for (int q = 0; q < P::R3; ++q) d[q * P::PA * S::st] = v[j][q];
      }
    }
    __syncthreads();
    if (!live) return;
    const int64_t ks = a.cols ? a.rows : 1;  // step of X along k
    C* xo = a.cols ? a.X + static_cast<int64_t>(c) * (L + 1) * a.rows + row : a.X + static_cast<int64_t>(line) * (L + 1);
#pragma unroll
    for (int j = 0; j < B::NJ3; ++j) {
      const int i3 = tl + j * B::TL;
      if (i3 >= P::NB3) continue;
      const C* p = S::s3_base(sm, g, i3 == 0 ? 0 : P::M - i3);  // holds the mirrored frequencies
#pragma unroll
      for (int q = 0; q < P::R3; ++q) {
        const int k = i3 + q * P::M;
        const int qm = i3 == 0 ? (P::R3 - q) % P::R3 : P::R3 - 1 - q;
        const C zk = v[j][q], zc = cconj(p[qm * P::PA * S::st]);
        const C ev = cscale(cadd(zk, zc), R(0.5));
        const C od = crot<false>(cscale(csub(zk, zc), R(0.5)));  // (zk - zc)/(2i)
        xo[k * ks] = cadd(ev, cmul(__ldg(a.twx + k), od));
      }
      if (i3 == 0) xo[L * ks] = cmk<C>(v[j][0].x - v[j][0].y, R(0));
    }
  }
};

// half spectrum -> real rows (unnormalised), keeps nx
template <typename R, int L> struct InvX : XPass<R, L> {
  using B = XPass<R, L>;
  using P = typename B::P;
  using C = typename B::C;
  using S = typename B::S;
  struct Args {
    const C* X;
    R* H;
    const C *tw2, *tw3, *twx;
    const int* gate;
    int nx, rows, cols;
  };
  static __device__ __forceinline__ void body(const Args& a, int blk) {
    if (a.gate && !*a.gate) return;
    C* sm = dyn_smem<C>();
    const int g = threadIdx.x % B::G, tl = threadIdx.x / B::G;
    const int line = blk * B::G + g;
    const bool live = line < 3 * a.rows;
    const int c = live ? line / a.rows : 0, row = live ? line - c * a.rows : 0;
    const int64_t ks = a.cols ? a.rows : 1;
    const C* xi = a.cols ? a.X + static_cast<int64_t>(c) * (L + 1) * a.rows + row : a.X + static_cast<int64_t>(live ? line : 0) * (L + 1);
#pragma unroll
    for (int j = 0; j < B::NJ3; ++j) {
      const int i3 = tl + j * B::TL;
      if (i3 < P::NB3) {
        C v[P::R3];
#pragma unroll
        for (int q = 0; q < P::R3; ++q) {
          // Z'[k] = (A + B) + i (A - B) conj(W^k), A = X[k], B = conj(X[L - k])
          const int k = i3 + q * P::M;
          const C x = xi[k * ks], y = cconj(xi[(L - k) * ks]);
          v[q] = cadd(cadd(x, y), crot<true>(cmul(csub(x, y), cconj(__ldg(a.twx + k)))));
        }
        S::s3_inv(S::s3_base(sm, g, i3), i3, a.tw3, v);
      }
    }
    __syncthreads();
    S::template s2<true>(sm, a.tw2);
    const int nx = a.nx;
    const int64_t N = static_cast<int64_t>(a.rows) * nx;
    R* out = a.H + c * N + static_cast<int64_t>(row) * nx;
    const bool even = !(nx & 1);
    S::s1_inv(sm, [&](int, int i1, const C* v) {
#pragma unroll
      for (int q = 0; q < P::H1; ++q) {
        const int u = 2 * (i1 + q * P::NB1);
        if (live && u < nx) {
          if (even) {
            *reinterpret_cast<C*>(out + u) = v[q];
          } else {
            out[u] = v[q].x;
            if (u + 1 < nx) out[u + 1] = v[q].y;
          }
        }
      }
    });
  }
};

// ------------------------------------------------- y passes, 3-D meshes ---
// Columns (c, z, kx) of the row-major spectra numbered consecutively, W of
// them a block, column fastest: every row access of a warp is a run of W
// neighbouring values (a block may straddle two planes; no tile is left
// partly empty at the end of a plane).
// 16-column rows up to 800 points, while two blocks an SM fit: 512 points took
// 80 / 74 us (forward / inverse, 256 x 256 x 64) against 103 / 82 with 8 columns.
template <typename R> constexpr int y_cols(int L) {
  const int w = L <= 800 ? 16 : (L <= 1600 ? 8 : 4);
  return sizeof(R) == 4 ? w : w / 2;
}

template <typename R, int L> struct YPass {
  using P = Plan<R, L>;
  using C = typename P::C;
  static constexpr int W = y_cols<R>(L);
  static constexpr size_t kSmem = sizeof(C) * Lines<P, W, 1, true>::kValues;
  static constexpr int TL = line_threads<P>(W, false, kSmem), kNT = W * TL;
  static constexpr int NJ3 = (P::NB3 + TL - 1) / TL;
  using S = Lines<P, W, kNT, true>;
  static constexpr int kMinB = blocks_for(kNT, regs_for<R>(P::RMAX), kSmem);
  struct Args {
    const C* in;
    C* out;
    const C *tw2, *tw3;
    const int* gate;
    int ny, Hx, ncol;  // ncol = 3 nz Hx
  };
};

template <typename R, int L, bool INV> struct YLine : YPass<R, L> {
  using B = YPass<R, L>;
  using P = typename B::P;
  using C = typename B::C;
  using S = typename B::S;
  using Args = typename B::Args;
  static __device__ __forceinline__ void body(const Args& a, int blk) {
    if (a.gate && !*a.gate) return;
    C* sm = dyn_smem<C>();
    const int w = threadIdx.x % B::W, tl = threadIdx.x / B::W;
    const int id = blk * B::W + w;
    const bool live = id < a.ncol;
    const int Hx = a.Hx, ny = a.ny;
    const int cz = live ? id / Hx : 0, kx = live ? id - cz * Hx : 0;
    const int64_t xo = static_cast<int64_t>(cz) * ny * Hx + kx, yo = static_cast<int64_t>(cz) * L * Hx + kx;
    if (!INV) {
      const C* x = a.in + xo;
      S::s1(sm, [&](int, int i1, C* v) {
#pragma unroll
        for (int q = 0; q < P::H1; ++q) {
          const int y = i1 + q * P::NB1;
          v[q] = live && y < ny ? x[static_cast<int64_t>(y) * Hx] : cmk<C>(R(0), R(0));
        }
      });
      __syncthreads();
      S::template s2<false>(sm, a.tw2);
      if (!live) return;
#pragma unroll
      for (int j = 0; j < B::NJ3; ++j) {
        const int i3 = tl + j * B::TL;
        if (i3 >= P::NB3) continue;
        C v[P::R3];
        S::s3(S::s3_base(sm, w, i3), i3, a.tw3, v);
        C* y = a.out + yo + static_cast<int64_t>(i3) * Hx;
#pragma unroll
        for (int q = 0; q < P::R3; ++q) y[static_cast<int64_t>(q * P::M) * Hx] = v[q];
      }
    } else {
#pragma unroll
      for (int j = 0; j < B::NJ3; ++j) {
        const int i3 = tl + j * B::TL;
        if (i3 < P::NB3) {
          C v[P::R3];
          const C* y = a.in + yo + static_cast<int64_t>(i3) * Hx;
#pragma unroll
          for (int q = 0; q < P::R3; ++q) v[q] = y[static_cast<int64_t>(q * P::M) * Hx];
          S::s3_inv(S::s3_base(sm, w, i3), i3, a.tw3, v);
        }
      }
      __syncthreads();
      S::template s2<true>(sm, a.tw2);
      C* x = a.out + xo;
      S::s1_inv(sm, [&](int, int i1, const C* v) {
#pragma unroll
        for (int q = 0; q < P::H1; ++q) {
          const int y = i1 + q * P::NB1;
          if (live && y < ny) x[static_cast<int64_t>(y) * Hx] = v[q];
        }
      });
    }
  }
};

// product of the three components with one tensor entry
template <typename R, typename C>
__device__ __forceinline__ void tensor_mul(C& a, C& b, C& c, R xx, R yy, R zz, R xy, R xz, R yz) {
  const C p = a, q = b, r = c;
  a = cmk<C>(xx * p.x + xy * q.x + xz * r.x, xx * p.y + xy * q.y + xz * r.y);
  b = cmk<C>(xy * p.x + yy * q.x + yz * r.x, xy * p.y + yy * q.y + yz * r.y);
  c = cmk<C>(xz * p.x + yz * q.x + zz * r.x, xz * p.y + yz * q.y + zz * r.y);
}

// ---------------------------------------------------------- z convolution ---
// Lines along z of W consecutive (ky, kx) positions (they are consecutive in
// memory), the three components in one block: S1, S2, then per butterfly of S3
// the last forward stage, the tensor product and the first inverse stage in
// registers.  Tiles are taken alternately from both ends, so that the tiles of
// ky and Py - ky, which read the same tensor entries, run close together.
template <typename R, int L> struct ZConv {
  using P = Plan<R, L, cap3(sizeof(R) == 8, L)>;
  using C = typename P::C;
  static constexpr int W = 128 / static_cast<int>(sizeof(C));
  static constexpr int kNT = W * P::M;
  using S = Lines<P, 3 * W, kNT, true>;
  static constexpr size_t kSmem = sizeof(C) * S::kValues;
  static constexpr int kMinB = blocks_for(kNT, regs_for<R>(3 * P::R3 > P::RMAX ? 3 * P::R3 : P::RMAX), kSmem);
  struct Args {
    C* Y;
    const R* Nhat;
    const C *tw2, *tw3;
    const int* gate;
    int nz, Hx, Py, tiles;
  };
  static __device__ __forceinline__ void body(const Args& a, int blk) {
    if (a.gate && !*a.gate) return;
    C* sm = dyn_smem<C>();
    const int tile = (blk & 1) ? a.tiles - 1 - (blk >> 1) : (blk >> 1);
    const int Hx = a.Hx, Py = a.Py, nz = a.nz;
    const int64_t S2d = static_cast<int64_t>(Py) * Hx, id0 = static_cast<int64_t>(tile) * W;
    C* base = a.Y + id0;
    const int nw = static_cast<int>(S2d - id0 < W ? S2d - id0 : W);
    S::s1(sm, [&](int line, int i1, C* v) {
      const int c = line / W, w = line - c * W;
      const C* y = base + static_cast<int64_t>(c * nz + i1) * S2d + w;
#pragma unroll
      for (int q = 0; q < P::H1; ++q)
        v[q] = w < nw && i1 + q * P::NB1 < nz ? y[static_cast<int64_t>(q * P::NB1) * S2d] : cmk<C>(R(0), R(0));
    });
    __syncthreads();
    S::template s2<false>(sm, a.tw2);
    {
      const int w = threadIdx.x % W, i3 = threadIdx.x / W;
      C v[3][P::R3];
#pragma unroll
      for (int c = 0; c < 3; ++c) S::s3(S::s3_base(sm, c * W + w, i3), i3, a.tw3, v[c]);
      if (w < nw) {
        const int64_t id = id0 + w;
        const int ky = static_cast<int>(id / Hx), kx = static_cast<int>(id - static_cast<int64_t>(ky) * Hx);
        const int Tyq = Py / 2 + 1;
        constexpr int Tzq = L / 2 + 1;
        const int64_t Tp = static_cast<int64_t>(Tyq) * Hx, Ts = Tzq * Tp;
        const bool fy = ky > Py / 2;
        const R sy = fy ? R(-1) : R(1);
        const R* nb = a.Nhat + static_cast<int64_t>(fy ? Py - ky : ky) * Hx + kx;
#pragma unroll
        for (int q = 0; q < P::R3; ++q) {
          const int kz = i3 + q * P::M;
          const bool fz = kz > L / 2;
          const R sz = fz ? R(-1) : R(1);
          const R* t = nb + (fz ? L - kz : kz) * Tp;
          tensor_mul<R>(v[0][q], v[1][q], v[2][q], __ldg(t), __ldg(t + Ts), __ldg(t + 2 * Ts), sy * __ldg(t + 3 * Ts),
                        sz * __ldg(t + 4 * Ts), sy * sz * __ldg(t + 5 * Ts));
        }
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) S::s3_inv(S::s3_base(sm, c * W + w, i3), i3, a.tw3, v[c]);
    }
    __syncthreads();
    S::template s2<true>(sm, a.tw2);
    S::s1_inv(sm, [&](int line, int i1, const C* v) {
      const int c = line / W, w = line - c * W;
      C* y = base + static_cast<int64_t>(c * nz + i1) * S2d + w;
#pragma unroll
      for (int q = 0; q < P::H1; ++q)
        if (w < nw && i1 + q * P::NB1 < nz) y[static_cast<int64_t>(q * P::NB1) * S2d] = v[q];
    });
  }
};

template <typename R> constexpr bool z_has(int L) { return L <= 256 && radices(L, cap3(sizeof(R) == 8, L)).r1 != 0; }

// ------------------------------------------------------------ film column ---
// Films (nz = 1, column-major X): forward y, tensor product and inverse y of
// the three components of G columns kx, in place on X.  Position fastest: a
// column is one contiguous run of memory.
// SPLIT (columns beyond 4096, one block an SM): the last stage, the product and
// the first inverse stage as three passes over shared memory instead of 3 R3
// values in registers, so that the block has 3/2 threads a butterfly (8000-point
// columns: 600 instead of 400 threads; 4000 x 4000 film, where 13 warps issued on
// 41 % of the cycles: 868 -> 734 us).
template <typename R, int L> struct FilmConv {
  using P = Plan<R, L, cap3(sizeof(R) == 8, L)>;
  using C = typename P::C;
  static constexpr bool SPLIT = L > 4096;
  static constexpr int G = P::M >= 96 ? 1 : (96 + P::M - 1) / P::M;
  static constexpr int kNT = SPLIT ? 3 * P::M / 2 : G * P::M;
  using S = Lines<P, 3 * G, kNT, false>;
  static constexpr size_t kSmem = sizeof(C) * S::kValues;
  static constexpr int kMinB = blocks_for(kNT, regs_for<R>(!SPLIT && 3 * P::R3 > P::RMAX ? 3 * P::R3 : P::RMAX), kSmem);
  struct Args {
    C* X;
    const R* Nhat;
    const C *tw2, *tw3;
    const int* gate;
    int ny, Hx;
  };
  static __device__ __forceinline__ void body(const Args& a, int blk) {
    if (a.gate && !*a.gate) return;
    C* sm = dyn_smem<C>();
    const int kx0 = blk * G, ny = a.ny, Hx = a.Hx;
    S::s1(sm, [&](int line, int i1, C* v) {
      const int g = line / 3, c = line - 3 * g;
      const C* x = a.X + (static_cast<int64_t>(c) * Hx + kx0 + g) * ny + i1;
      const bool live = kx0 + g < Hx;
#pragma unroll
      for (int q = 0; q < P::H1; ++q)
        v[q] = live && i1 + q * P::NB1 < ny ? x[q * P::NB1] : cmk<C>(R(0), R(0));
    });
    __syncthreads();
    S::template s2<false>(sm, a.tw2);
    constexpr int Tyq = L / 2 + 1;
    const int64_t Ts = static_cast<int64_t>(Hx) * Tyq;
    if constexpr (SPLIT) {
      for (int t = threadIdx.x; t < 3 * P::M; t += kNT) {
        const int c = t / P::M, i3 = t - c * P::M;
        C* d = S::s3_base(sm, c, i3);
        C v[P::R3];
        S::s3(d, i3, a.tw3, v);
#pragma unroll
        for (int q = 0; q < P::R3; ++q) d[q * P::PA] = v[q];  // frequency i3 + q M in slot q
      }
      __syncthreads();
      const R* nb = a.Nhat + static_cast<int64_t>(kx0) * Tyq;
#pragma unroll 4
      for (int ky = threadIdx.x; ky < L; ky += kNT) {
        const int q = ky / P::M, i3 = ky - q * P::M;
        C* d = S::s3_base(sm, 0, i3) + q * P::PA;
        const bool fy = ky > L / 2;
        const R sy = fy ? R(-1) : R(1);
        const R* t = nb + (fy ? L - ky : ky);
        C x = d[0], y = d[S::LS], z = d[2 * S::LS];
        tensor_mul<R>(x, y, z, __ldg(t), __ldg(t + Ts), __ldg(t + 2 * Ts), sy * __ldg(t + 3 * Ts), __ldg(t + 4 * Ts),
                      sy * __ldg(t + 5 * Ts));
        d[0] = x;
        d[S::LS] = y;
        d[2 * S::LS] = z;
      }
      __syncthreads();
      for (int t = threadIdx.x; t < 3 * P::M; t += kNT) {
        const int c = t / P::M, i3 = t - c * P::M;
        C* d = S::s3_base(sm, c, i3);
        C v[P::R3];
#pragma unroll
        for (int q = 0; q < P::R3; ++q) v[q] = d[q * P::PA];
        S::s3_inv(d, i3, a.tw3, v);
      }
    } else {
      const int g = threadIdx.x / P::M, i3 = threadIdx.x - g * P::M;
      C v[3][P::R3];
#pragma unroll
      for (int c = 0; c < 3; ++c) S::s3(S::s3_base(sm, 3 * g + c, i3), i3, a.tw3, v[c]);
      if (kx0 + g < Hx) {
        const R* nb = a.Nhat + static_cast<int64_t>(kx0 + g) * Tyq;
#pragma unroll
        for (int q = 0; q < P::R3; ++q) {
          const int ky = i3 + q * P::M;
          const bool fy = ky > L / 2;
          const R sy = fy ? R(-1) : R(1);
          const R* t = nb + (fy ? L - ky : ky);
          tensor_mul<R>(v[0][q], v[1][q], v[2][q], __ldg(t), __ldg(t + Ts), __ldg(t + 2 * Ts), sy * __ldg(t + 3 * Ts),
                        __ldg(t + 4 * Ts), sy * __ldg(t + 5 * Ts));
        }
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) S::s3_inv(S::s3_base(sm, 3 * g + c, i3), i3, a.tw3, v[c]);
    }
    __syncthreads();
    S::template s2<true>(sm, a.tw2);
    S::s1_inv(sm, [&](int line, int i1, const C* v) {
      const int g = line / 3, c = line - 3 * g;
      C* x = a.X + (static_cast<int64_t>(c) * Hx + kx0 + g) * ny + i1;
      if (kx0 + g >= Hx) return;
#pragma unroll
      for (int q = 0; q < P::H1; ++q)
        if (i1 + q * P::NB1 < ny) x[q * P::NB1] = v[q];
    });
  }
};

// a column's three lines in one block's shared memory
template <typename R> constexpr bool film_has(int L) {
  const Radices f = radices(L, cap3(sizeof(R) == 8, L));
  if (f.r1 == 0 || f.r1 * f.r2 > 512) return false;
  const size_t line = static_cast<size_t>(f.r2) * (f.r3 * (f.r1 | 1) + 16) + 16;
  return 3 * line * sizeof(cplx_t<R>) <= 227 * 1024;
}

}  // namespace rf
}  // namespace mm
