// mm_hotpass.cuh -- launchers of the run-time-length demag passes
// (mm_passes.cuh) and the fused power-of-two z convolution (internal).
#pragma once
#include <algorithm>
#include <cstdlib>
#include <mutex>

#include "mm_passes.cuh"

namespace mm {

inline int floor_pow2(int v) {
  int p = 1;
  while (p * 2 <= v) p *= 2;
  return p;
}
inline int ilog2(int v) {
  int l = 0;
  while ((1 << l) < v) ++l;
  return l;
}

// Shared-memory budget of one strided-pass block; the kx tile W is the
// largest power of two (up to 128 bytes of row segment) that fits.
// Multiprocessors of the current device (cached on first use)
inline int sm_count() {
  static const int v = [] {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 148;
  }();
  return v;
}

// Lines a shared-memory x-pass block transforms: as many as fill its tile
// (cap / Lc), but for a mesh launched alone no more than spread `lines` over
// two blocks an SM -- on small meshes (c1: 150 lines of 200 points) more,
// shorter blocks finish sooner than a few full ones.  A pass recorded for a
// batch keeps full tiles: its launch covers the lines of every mesh.  Each
// line's arithmetic is the same whatever block it lands in.
template <typename R, int NT>
inline int x_lines_per_block(int lines, int Lc) {
  const int full = std::max(1, PassCfg<R, NT>::cap / Lc);
  if (launch_recorder()) return full;
  const int spread = std::max(1, (lines + 2 * sm_count() - 1) / (2 * sm_count()));
  return std::min(full, spread);
}

inline int smem_budget_bytes() {
  static int v = [] {
    const char* e = getenv("MMCUDA_LINES_SMEM_KB");
    const int kb = e ? atoi(e) : 100;
    return (kb > 8 && kb <= 200 ? kb : 100) * 1024;
  }();
  return v;
}


// Largest power-of-two radix of the FP32 shared-memory passes (32 or 16;
// MMCUDA_MAXRADIX=16 selects 16).  A radix-32 butterfly holds 32 complex
// values a thread, a little above the 80-register budget of the
// 3-blocks-per-SM passes (a few spilled words), yet one stage fewer a line:
// c2's 512-point FP32 y passes take 0.076 ms with radix 32 and 0.114 ms with
// radix 16.
inline int fp32_max_radix() {
  static const int v = [] {
    const char* e = getenv("MMCUDA_MAXRADIX");
    return e && atoi(e) == 16 ? 16 : 32;
  }();
  return v;
}

// The register-resident x and y passes (mm_wreg.cu) where they apply, unless
// MMCUDA_WREG=0 keeps the shared-memory kernels
inline bool wreg_enabled() {
  static const bool on = [] {
    const char* e = getenv("MMCUDA_WREG");
    return !(e && e[0] == '0');
  }();
  return on;
}

// The direct-DFT z convolution for Pz <= 9 (ZSmall) unless MMCUDA_ZSMALL=0
inline bool zsmall_enabled() {
  static const bool on = [] {
    const char* e = getenv("MMCUDA_ZSMALL");
    return !(e && e[0] == '0');
  }();
  return on;
}

// The register-resident z convolution (mm_zpair.cu) where it applies, unless
// MMCUDA_ZPAIR=0 keeps the shared-memory kernels
inline bool zpair_enabled() {
  static const bool on = [] {
    const char* e = getenv("MMCUDA_ZPAIR");
    return !(e && e[0] == '0');
  }();
  return on;
}

// 3-D column-major spectra (DemagGeom::yT) unless MMCUDA_COLS3D=0 keeps the
// row-major layout; both run the same arithmetic on every line
inline bool cols3d_enabled() {
  static const bool on = [] {
    const char* e = getenv("MMCUDA_COLS3D");
    return !(e && e[0] == '0');
  }();
  return on;
}

// z convolution for Pz = RA * RB (powers of two): forward radix-RA stage from
// the Y rows into shared memory; then, per butterfly i < RA and in registers,
// the forward radix-RB stage (outputs kz = i + r*RA), the tensor product at
// those kz for the three components, and the inverse radix-RB stage (its
// inputs are the same positions), written back in place after a barrier;
// finally the inverse radix-RA stage straight to the Y rows kz < nz.
// One shared buffer; requires W * RA <= NT (one middle task per thread).
// YT (column-major spectra, DemagGeom::yT): a block takes one kx and a tile of
// W consecutive ky (grid: (Hx, ky tiles), tile q and its mirror Py/W-1-q
// adjacent in launch order); the tile's rows are W contiguous entries of
// Y[((c*Hx + kx)*nz + z)*Py + ky], the tensor Nhat[((c*Tzq + kz)*Hx + kx)*Tyq + ky].
// Row-major: blocks blockIdx.x < nfull take W-wide kx tiles; the columns
// kx >= nfull * W left over (Hx = 16 m + 1 for nx = 2^k) are tiled along ky
// instead, block (nfull + r, q) taking column nfull * W + r and ky in
// [q W, q W + W) (the blocks with q W >= Py return), so that no block
// transforms a tile of mostly absent columns.
template <typename R, int RA, int RB, int NT, bool I32, bool YT = false>
__global__ void __launch_bounds__(NT, (zconv2_minb<R, NT>())) k_zconv2(cplx_t<R>* Y, const R* __restrict__ Nhat, DemagGeom g, int lgW,
                                                  FastDiv fnl, const cplx_t<R>* __restrict__ twz, int nfull) {
  using C = cplx_t<R>;
  using IX = std::conditional_t<I32, int, int64_t>;
  constexpr int L = RA * RB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* a = reinterpret_cast<C*>(smem_raw);
  pdl_enter();
  if (g.gate && !*g.gate) return;
  const int LS = L | 1, Hx = g.Hx, Py = g.Py, nz = g.nz;
  const int W = 1 << lgW;
  const int bq = blockIdx.y;
  int kx0, ky0;  // first column of the tile: (kx0 + w, ky0) or, along ky, (kx0, ky0 + w)
  bool along_ky = YT;
  if (YT) {
    const int nq = gridDim.y;
    kx0 = blockIdx.x;
    ky0 = ((bq & 1) ? nq - 1 - (bq >> 1) : (bq >> 1)) << lgW;
  } else if (static_cast<int>(blockIdx.x) >= nfull) {
    if ((bq << lgW) >= Py) return;
    kx0 = nfull * W + (blockIdx.x - nfull);
    ky0 = bq << lgW;
    along_ky = true;
  } else {
    const int q = (bq + 1) >> 1;
    kx0 = blockIdx.x * W;
    ky0 = bq == 0 ? 0 : ((bq & 1) ? q : Py - q);
  }
  const int nlines = 3 * W;
  // rows of the tile: element (c, z, w) at base + c*cs + z*rs + (t0 + w)*ws, t0 + w < tn
  const IX cs = static_cast<IX>(static_cast<int64_t>(nz) * Py * Hx), rs = static_cast<IX>(YT ? Py : static_cast<int64_t>(Py) * Hx);
  C* base = YT ? Y + static_cast<int64_t>(kx0) * nz * Py : (along_ky ? Y + kx0 : Y + static_cast<int64_t>(ky0) * Hx);
  const int t0 = along_ky ? ky0 : kx0, tn = along_ky ? Py : Hx;
  const IX ws = static_cast<IX>(along_ky && !YT ? Hx : 1);
  RowsInW<C, IX> src{base, cs, rs, ws, lgW, t0, tn, nz};
  RowsOutW<C, IX> dst{base, cs, rs, ws, lgW, t0, tn, nz};
  SmemLines<C> A{a, LS};
  lstage<RA, false, true, NT>(src, A, L, nlines, fnl, 1, twz, 1);
  // fused middle: thread -> (w, i), w fastest
  const int task = threadIdx.x;
  const bool act = task < W * RA;
  const int w = task & (W - 1), i = task >> lgW;
  const int kx = along_ky ? kx0 : kx0 + w;
  const int ky = along_ky ? ky0 + w : ky0;
  C v[3][RB];
  if (act) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
#pragma unroll
      for (int r = 0; r < RB; ++r) v[c][r] = A.load(c * W + w, i + r * RA);
      // forward radix-RB stage, span p = RA, k = i: twiddles w_L^(r*i)
#pragma unroll
      for (int r = 1; r < RB; ++r) v[c][r] = cmul(v[c][r], __ldg(twz + r * i));
      dftR<RB, false>(v[c]);
    }
    if (kx < Hx && ky < Py) {
      const int Tyq = Py / 2 + 1, Tzq = L / 2 + 1;
      const int64_t Ts = static_cast<int64_t>(Tzq) * Tyq * Hx;
      const bool fy = ky > Py / 2;
      const int kyq = fy ? Py - ky : ky;
      const R sy = fy ? R(-1) : R(1);
#pragma unroll
      for (int r = 0; r < RB; ++r) {
        const int kz = i + r * RA;
        const bool fz = kz > L / 2;
        const int kzq = fz ? L - kz : kz;
        const R sz = fz ? R(-1) : R(1);
        const int64_t b = YT ? (static_cast<int64_t>(kzq) * Hx + kx) * Tyq + kyq
                             : (static_cast<int64_t>(kzq) * Tyq + kyq) * Hx + kx;
        const R xx = __ldg(Nhat + b), yy = __ldg(Nhat + Ts + b), zz = __ldg(Nhat + 2 * Ts + b);
        const R xy = sy * __ldg(Nhat + 3 * Ts + b), xz = sz * __ldg(Nhat + 4 * Ts + b),
                yz = sy * sz * __ldg(Nhat + 5 * Ts + b);
        const C p0 = v[0][r], p1 = v[1][r], p2 = v[2][r];
        v[0][r] = cmk<C>(xx * p0.x + xy * p1.x + xz * p2.x, xx * p0.y + xy * p1.y + xz * p2.y);
        v[1][r] = cmk<C>(xy * p0.x + yy * p1.x + yz * p2.x, xy * p0.y + yy * p1.y + yz * p2.y);
        v[2][r] = cmk<C>(xz * p0.x + yz * p1.x + zz * p2.x, xz * p0.y + yz * p1.y + zz * p2.y);
      }
    }
    // inverse radix-RB stage, span 1: outputs at i*RB + r
#pragma unroll
    for (int c = 0; c < 3; ++c) dftR<RB, true>(v[c]);
  }
  __syncthreads();
  if (act) {
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int r = 0; r < RB; ++r) A.store(c * W + w, i * RB + r, v[c][r]);
  }
  __syncthreads();
  lstage<RA, true, true, NT>(A, dst, L, nlines, fnl, RB, twz, 1);
}

template <typename R, int MODE, int NT>
void launch_fwd_x(const DemagGeom& g, const R* m, const R* Ms, const double* Tr, int tsign, cplx_t<R>* X,
                         int ncomp, const cplx_t<R>* twx, cudaStream_t st) {
  using C = cplx_t<R>;
  const int rows = g.ny * g.nz;
  const int lines = ncomp * rows;
  if (g.Px == 1) {
    k_fwd_x1<R, MODE><<<(lines + 255) / 256, 256, 0, st>>>(m, Ms, Tr, X, rows, lines, g.gate);
    return;
  }
  const int nl = x_lines_per_block<R, NT>(lines, g.Lc);
  const int blocks = (lines + nl - 1) / nl;
  const int half = nl * (g.Lc | 1);
  const size_t sm = 2 * sizeof(C) * half;
  launch_k<FwdX<R, MODE, NT>>(dim3(blocks), sm, st, {m, Ms, Tr, tsign, X, g, lines, nl, twx, half, make_fastdiv(nl), dim3()});
}

template <typename R>
void launch_inv_x(const DemagGeom& g, const cplx_t<R>* X, R* Hd, const cplx_t<R>* twx, cudaStream_t st) {
  constexpr int NT = kHotNT;
  const int lines = 3 * g.ny * g.nz;
  const int nl = x_lines_per_block<R, NT>(lines, g.Lc);
  const int half = nl * (g.Lc | 1);
  const size_t sm = 2 * sizeof(cplx_t<R>) * half;
  launch_k<InvX<R, NT>>(dim3((lines + nl - 1) / nl), sm, st, {X, Hd, g, lines, nl, twx, half, make_fastdiv(nl), dim3()});
}

// every element offset of the X and Y spectra (3 * nz * max(Py, ny) * Hx
// complex words) fits in a signed 32-bit int
inline bool offsets_fit_int(const DemagGeom& g) {
  return 3LL * g.nz * std::max(g.Py, g.ny) * g.Hx < (1LL << 31);
}

template <typename R>
inline int lines_tile(int Hx, int L, int lines_per_col, int nbuf) {
  using C = cplx_t<R>;
  int W = 128 / static_cast<int>(sizeof(C));
  const size_t per = static_cast<size_t>(std::max(1, nbuf)) * lines_per_col * (L | 1) * sizeof(C);
  while (W > 1 && W * per > static_cast<size_t>(smem_budget_bytes())) W /= 2;
  while (W > 1 && W / 2 >= Hx) W /= 2;
  return W;
}

// shared memory of one block of a strided pass with tile width W (bytes)
template <typename R>
inline size_t pass_smem(const DemagGeom& g, int which, bool fused2d, int W) {
  using C = cplx_t<R>;
  if (which == 1 || which == 3)
    return static_cast<size_t>(std::max(1, line_fft_buffers(g.ply))) * sizeof(C) * W *
           (g.yT ? padded_line_stride(g.Py) : g.Py | 1);
  if (fused2d) return 2 * sizeof(C) * 3 * W * (g.xT ? padded_line_stride(g.Py) : g.Py | 1);
  const bool zc2 = (g.Pz & (g.Pz - 1)) == 0 && g.Pz >= 4 && (g.Pz <= 128 || (sizeof(R) == 4 && g.Pz == 256));
  return (zc2 ? 1 : 2) * sizeof(C) * 3 * W * (g.Pz | 1);
}

// first radix of the fused-middle z kernel (W * RA threads carry the middle)
inline int zconv2_ra(int Pz) {
  switch (Pz) {
    case 4: return 2;
    case 8: return 4;
    case 16: return 4;
    case 32: return 8;
    case 64: return 8;
    case 128: return 16;
    case 256: return 32;
    default: return 0;
  }
}

template <typename R, int MODE>
void launch_ylines(const DemagGeom& g, const cplx_t<R>* in, cplx_t<R>* out, const R* Nhat,
                          const cplx_t<R>* twy, cudaStream_t st, int Wforce = 0) {
  using C = cplx_t<R>;
  const int ncompc = MODE == YL_CONV2D ? 3 : 1;
  const int nbuf = MODE == YL_CONV2D ? 2 : line_fft_buffers(g.ply);
  const bool xt = MODE == YL_CONV2D ? g.xT != 0 : g.yT != 0;
  const int W = Wforce > 0 ? Wforce : lines_tile<R>(g.Hx, g.Py, ncompc, nbuf);
  const int half = ncompc * W * (xt ? padded_line_stride(g.Py) : g.Py | 1);
  // full tiles; up to W/4 leftover columns (row-major) run as one-column blocks
  const int rem = g.Hx % W;
  const int nfull = !xt && rem > 0 && rem <= W / 4 ? g.Hx / W : (g.Hx + W - 1) / W;
  const int ncols = nfull * W >= g.Hx ? 0 : g.Hx - nfull * W;
  dim3 grid(nfull + ncols, g.nz, 3 / ncompc);
  const size_t sm = static_cast<size_t>(std::max(1, nbuf)) * sizeof(C) * half;
  const FastDiv fnl = make_fastdiv(ncompc * W), fnl1 = make_fastdiv(ncompc);
  if (xt) {
    if (offsets_fit_int(g))
      launch_k<YLines<R, MODE, kHotNT, true, true>>(grid, sm, st, {in, out, Nhat, g, ilog2(W), ncompc, fnl, twy, half, nfull, fnl1, dim3()});
    else
      launch_k<YLines<R, MODE, kHotNT, false, true>>(grid, sm, st, {in, out, Nhat, g, ilog2(W), ncompc, fnl, twy, half, nfull, fnl1, dim3()});
    return;
  }
  if (offsets_fit_int(g))
    launch_k<YLines<R, MODE, kHotNT, true>>(grid, sm, st, {in, out, Nhat, g, ilog2(W), ncompc, fnl, twy, half, nfull, fnl1, dim3()});
  else
    launch_k<YLines<R, MODE, kHotNT, false>>(grid, sm, st, {in, out, Nhat, g, ilog2(W), ncompc, fnl, twy, half, nfull, fnl1, dim3()});
}

template <typename R, int RA, int RB>
void launch_zconv2(const DemagGeom& g, cplx_t<R>* Y, const R* Nhat, const cplx_t<R>* twz, cudaStream_t st,
                          int Wforce) {
  using C = cplx_t<R>;
  constexpr int L = RA * RB;
  constexpr int NTZ = zconv2_nt<R>();
  // tiles of W columns along kx, or along ky for column-major spectra (yT)
  int W = Wforce > 0 ? Wforce : lines_tile<R>(g.yT ? g.Py : g.Hx, L, 3, 1);
  while (W * RA > NTZ) W /= 2;
  const size_t sm = sizeof(C) * 3 * W * (L | 1);
  {
    static std::mutex mu;
    static uint64_t done = 0;
    int dev = 0;
    cudaGetDevice(&dev);
    const bool tracked = dev >= 0 && dev < 64;
    std::lock_guard<std::mutex> lk(mu);
    if (!tracked || !((done >> dev) & 1ull)) {
      const int mx = static_cast<int>(kMaxSmem);
      cudaFuncSetAttribute(k_zconv2<R, RA, RB, NTZ, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx);
      cudaFuncSetAttribute(k_zconv2<R, RA, RB, NTZ, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx);
      cudaFuncSetAttribute(k_zconv2<R, RA, RB, NTZ, true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx);
      cudaFuncSetAttribute(k_zconv2<R, RA, RB, NTZ, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx);
      if (tracked) done |= 1ull << dev;
    }
  }
  const FastDiv fnl = make_fastdiv(3 * W);
  if (g.yT) {
    dim3 grid(g.Hx, (g.Py + W - 1) / W, 1);
    if (offsets_fit_int(g))
      launch_pdl(k_zconv2<R, RA, RB, NTZ, true, true>, grid, dim3(NTZ), sm, st, Y, Nhat, g, ilog2(W), fnl, twz, g.Hx);
    else
      launch_pdl(k_zconv2<R, RA, RB, NTZ, false, true>, grid, dim3(NTZ), sm, st, Y, Nhat, g, ilog2(W), fnl, twz, g.Hx);
    return;
  }
  // full kx tiles; up to W/4 leftover columns run as ky tiles in the same grid
  const int rem = g.Hx % W;
  const int nfull = rem > 0 && rem <= W / 4 && W <= g.Py ? g.Hx / W : (g.Hx + W - 1) / W;
  const int ncols = nfull * W >= g.Hx ? 0 : g.Hx - nfull * W;
  dim3 grid(nfull + ncols, g.Py, 1);
  if (offsets_fit_int(g))
    launch_pdl(k_zconv2<R, RA, RB, NTZ, true>, grid, dim3(NTZ), sm, st, Y, Nhat, g, ilog2(W), fnl, twz, nfull);
  else
    launch_pdl(k_zconv2<R, RA, RB, NTZ, false>, grid, dim3(NTZ), sm, st, Y, Nhat, g, ilog2(W), fnl, twz, nfull);
}

// Power-of-two z lengths with a fused-middle kernel: L = RA * RB
template <typename R>
inline bool try_zconv2(const DemagGeom& g, cplx_t<R>* Y, const R* Nhat, const cplx_t<R>* twz, cudaStream_t st,
                       int Wf) {
  switch (g.Pz) {
    case 4: launch_zconv2<R, 2, 2>(g, Y, Nhat, twz, st, Wf); return true;
    case 8: launch_zconv2<R, 4, 2>(g, Y, Nhat, twz, st, Wf); return true;
    case 16: launch_zconv2<R, 4, 4>(g, Y, Nhat, twz, st, Wf); return true;
    case 32: launch_zconv2<R, 8, 4>(g, Y, Nhat, twz, st, Wf); return true;
    case 64: launch_zconv2<R, 8, 8>(g, Y, Nhat, twz, st, Wf); return true;
    case 128: launch_zconv2<R, 16, 8>(g, Y, Nhat, twz, st, Wf); return true;
    case 256:
      if constexpr (sizeof(R) == 4) {
        launch_zconv2<R, 32, 8>(g, Y, Nhat, twz, st, Wf);
        return true;
      }
      return false;
    default: return false;
  }
}

template <typename R, int PZ>
void launch_zsmall_pz(const DemagGeom& g, cplx_t<R>* Y, const R* Nhat, cudaStream_t st) {
  typename ZSmall<R, PZ>::Args a{};
  a.Y = Y;
  a.Nhat = Nhat;
  a.gate = g.gate;
  a.Hx = g.Hx;
  a.Py = g.Py;
  a.nz = g.nz;
  a.Tyq = g.Tyq;
  a.Tzq = g.Tzq;
  for (int t = 0; t < PZ; ++t) {
    const long double ang = -2.0L * 3.141592653589793238462643383279502884L * t / PZ;
    a.twr[t] = static_cast<R>(static_cast<double>(cosl(ang)));
    a.twi[t] = static_cast<R>(static_cast<double>(sinl(ang)));
  }
  const int64_t lines = static_cast<int64_t>(g.Hx) * g.Py;
  launch_k<ZSmall<R, PZ>>(dim3(static_cast<unsigned>((lines + 255) / 256)), 0, st, a);
}

// the direct-DFT z convolution for Pz = 3, 5, 7, 9 on row-major spectra
template <typename R>
inline bool try_zsmall(const DemagGeom& g, cplx_t<R>* Y, const R* Nhat, cudaStream_t st) {
  if (g.yT || !zsmall_enabled()) return false;
  switch (g.Pz) {
    case 3: launch_zsmall_pz<R, 3>(g, Y, Nhat, st); return true;
    case 5: launch_zsmall_pz<R, 5>(g, Y, Nhat, st); return true;
    case 7: launch_zsmall_pz<R, 7>(g, Y, Nhat, st); return true;
    case 9: launch_zsmall_pz<R, 9>(g, Y, Nhat, st); return true;
    default: return false;
  }
}

template <typename R>
void launch_zconv(const DemagGeom& g, cplx_t<R>* Y, const R* Nhat, const cplx_t<R>* twz, cudaStream_t st,
                         int Wforce, const void* zmap) {
  using C = cplx_t<R>;
  if constexpr (sizeof(R) == 4) {
    if (zpair_enabled() && zpair_applies(g)) {
      launch_zpair_f32(g, Y, Nhat, zmap, st);
      return;
    }
  } else {
    if (zquad_applies(g)) {
      launch_zquad_f64(g, Y, Nhat, st);
      return;
    }
  }
  if (try_zconv2<R>(g, Y, Nhat, twz, st, Wforce)) return;
  if (try_zsmall<R>(g, Y, Nhat, st)) return;
  const int W = Wforce > 0 ? Wforce : lines_tile<R>(g.Hx, g.Pz, 3, 2);
  const int half = 3 * W * (g.Pz | 1);
  dim3 grid((g.Hx + W - 1) / W, g.Py, 1);
  const size_t sm = 2 * sizeof(C) * half;
  if (offsets_fit_int(g))
    launch_k<ZConv<R, kHotNT, true>>(grid, sm, st, {Y, Nhat, g, ilog2(W), make_fastdiv(3 * W), twz, half, dim3()});
  else
    launch_k<ZConv<R, kHotNT, false>>(grid, sm, st, {Y, Nhat, g, ilog2(W), make_fastdiv(3 * W), twz, half, dim3()});
}

// The run-time-length passes are compiled one kind and form a file
// (mm_hot_*.cu); other files only declare them.
#define MM_HOT_X(EXT, R)                                                                                             \
  EXT template void launch_fwd_x<R, XM_MAGN, kHotNT>(const DemagGeom&, const R*, const R*, const double*, int,       \
                                                     cplx_t<R>*, int, const cplx_t<R>*, cudaStream_t);              \
  EXT template void launch_inv_x<R>(const DemagGeom&, const cplx_t<R>*, R*, const cplx_t<R>*, cudaStream_t);
#define MM_HOT_Y(EXT, R)                                                                                             \
  EXT template void launch_ylines<R, YL_FWD>(const DemagGeom&, const cplx_t<R>*, cplx_t<R>*, const R*,               \
                                             const cplx_t<R>*, cudaStream_t, int);                                   \
  EXT template void launch_ylines<R, YL_INV>(const DemagGeom&, const cplx_t<R>*, cplx_t<R>*, const R*,               \
                                             const cplx_t<R>*, cudaStream_t, int);
#define MM_HOT_YC(EXT, R)                                                                                            \
  EXT template void launch_ylines<R, YL_CONV2D>(const DemagGeom&, const cplx_t<R>*, cplx_t<R>*, const R*,            \
                                                const cplx_t<R>*, cudaStream_t, int);
#define MM_HOT_Z(EXT, R)                                                                                             \
  EXT template void launch_zconv<R>(const DemagGeom&, cplx_t<R>*, const R*, const cplx_t<R>*, cudaStream_t, int,     \
                                    const void*);
#ifndef MM_HOT_IMPL
MM_HOT_X(extern, float) MM_HOT_X(extern, double)
MM_HOT_Y(extern, float) MM_HOT_Y(extern, double)
MM_HOT_YC(extern, float) MM_HOT_YC(extern, double)
MM_HOT_Z(extern, float) MM_HOT_Z(extern, double)
#endif

}  // namespace mm
