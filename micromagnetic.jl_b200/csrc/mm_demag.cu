// mm_demag.cu -- demag tensor assembly (FP64) and FFT convolution passes.
#include <algorithm>
#include <tuple>
#include <mutex>
#include <map>
#include <set>
#include <array>
#include <cstdlib>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "mm_dd.cuh"
#include "mm_demag.cuh"
#include "mm_hotpass.cuh"
#include "mm_persist.cuh"
#include "mm_passes.cuh"
#include "mm_fft.cuh"
#include "mm_launch.cuh"
#include "mm_lines.cuh"

namespace mm {

// FP64 tensor quadrant [6][Tzq][Tyq][Hx] to RO, column-major [6][Tzq][Hx][Tys]
// (rows of Tyq values at stride Tys >= Tyq; films: Tzq = 1)
template <typename RO>
__global__ void k_cast_cols(const double* __restrict__ a, RO* __restrict__ b, int Tyq, int Tys, int Hx, int Tzq) {
  const int64_t plane = static_cast<int64_t>(Tyq) * Hx, n = 6LL * Tzq * plane;
  for (int64_t o = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; o < n;
       o += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t c = o / plane, r = o - c * plane;
    const int64_t kx = r / Tyq, ky = r - kx * Tyq;
    b[(c * Hx + kx) * Tys + ky] = static_cast<RO>(a[c * plane + ky * Hx + kx]);
  }
}

template <typename RO>
__global__ void k_cast(const double* __restrict__ a, RO* __restrict__ b, int64_t n) {
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    b[i] = static_cast<RO>(a[i]);
}

// ------------------------------------------------------ Newell tensor -----
// newell_f / newell_g: src/micro/demag.jl:133-192 (Newell, Williams & Dunlop,
// J. Geophys. Res. 98 (1993) 9551); 27-point second differences
// demag_tensor_xx / _xy demag.jl:194-296; dipole far field
// src/atomistic/demag.jl:106-138 beyond R > 60 cells (demag.jl:196-201,
// 247-252); macro-PBC image sums demag.jl:298-386.
//
// The second differences cancel up to R^6 (5e10 at R = 60) of the function
// values, so an FP64 evaluation carries relative errors up to ~1e-6 in the
// tensor entries near the dipole switch (its rounding, and 1-ulp differences
// between libm implementations, show in H_demag at ~1e-9).  Here f and g are
// evaluated in double-double arithmetic at the exact coordinates
// (X + a) * dx (X an integer offset, dx the normalised cell size), the
// differences, image sums and dipole terms are summed in double-double, and
// each entry is rounded to FP64 once: the tensor of the given normalised
// cell is then correct to the last bit or so.  The near field is evaluated
// once per grid point (every point serves up to 27 entries) and stored; f is
// even in each argument, g odd in its first two and even in the third.
using dd::DD;

__device__ DD ddf(DD x, DD y, DD z) {
  const DD x2 = dd::mul(x, x), y2 = dd::mul(y, y), z2 = dd::mul(z, z);
  const DD R = dd::sqrt(dd::add(dd::add(x2, y2), z2));
  if (dd::is_zero(R)) return dd::mk(0.0);
  DD f = dd::div(dd::mul(dd::sub(dd::sub(dd::scale2(x2, 2.0), y2), z2), R), 6.0);
  if (dd::positive(x2))
    f = dd::sub(f, dd::mul(dd::mul(dd::mul(x, y), z), dd::atan(dd::div(dd::mul(y, z), dd::mul(x, R)))));
  const DD xz = dd::add(x2, z2), xy = dd::add(x2, y2);
  if (dd::positive(xz))
    f = dd::add(f, dd::mul(dd::scale2(dd::mul(y, dd::sub(z2, x2)), 0.5), dd::asinh(dd::div(y, dd::sqrt(xz)))));
  if (dd::positive(xy))
    f = dd::add(f, dd::mul(dd::scale2(dd::mul(z, dd::sub(y2, x2)), 0.5), dd::asinh(dd::div(z, dd::sqrt(xy)))));
  return f;
}

__device__ DD ddg(DD x, DD y, DD z) {
  const DD x2 = dd::mul(x, x), y2 = dd::mul(y, y), z2 = dd::mul(z, z);
  const DD R = dd::sqrt(dd::add(dd::add(x2, y2), z2));
  if (dd::is_zero(R)) return dd::mk(0.0);
  DD g = dd::neg(dd::div(dd::mul(dd::mul(x, y), R), 3.0));
  if (dd::positive(z2))
    g = dd::sub(g, dd::div(dd::mul(dd::mul(z2, z), dd::atan(dd::div(dd::mul(x, y), dd::mul(z, R)))), 6.0));
  if (dd::positive(y2))
    g = dd::sub(g, dd::scale2(dd::mul(dd::mul(y2, z), dd::atan(dd::div(dd::mul(x, z), dd::mul(y, R)))), 0.5));
  if (dd::positive(x2))
    g = dd::sub(g, dd::scale2(dd::mul(dd::mul(x2, z), dd::atan(dd::div(dd::mul(y, z), dd::mul(x, R)))), 0.5));
  const DD xy = dd::add(x2, y2), yz = dd::add(y2, z2), xz = dd::add(x2, z2);
  const DD z3 = dd::scale2(z2, 3.0);
  if (dd::positive(xy)) g = dd::add(g, dd::mul(dd::mul(dd::mul(x, y), z), dd::asinh(dd::div(z, dd::sqrt(xy)))));
  if (dd::positive(yz))
    g = dd::add(g, dd::div(dd::mul(dd::mul(y, dd::sub(z3, y2)), dd::asinh(dd::div(x, dd::sqrt(yz)))), 6.0));
  if (dd::positive(xz))
    g = dd::add(g, dd::div(dd::mul(dd::mul(x, dd::sub(z3, x2)), dd::asinh(dd::div(y, dd::sqrt(xz)))), 6.0));
  return g;
}

struct NewellGrid {
  double dx, dy, dz;  // normalised cell (max = 1)
  int ex, ey, ez;     // grid extents: offsets 0..ex etc. are stored
  DD* F;              // [6][ez+1][ey+1][ex+1]
};

// f or g of component c (xx yy zz xy xz yz) at the integer offset (X, Y, Z),
// arguments permuted as demag_tensor_yy / zz / xz / yz do
__device__ DD newell_fn(int c, int64_t X, int64_t Y, int64_t Z, const NewellGrid& G) {
  const DD x = dd::two_prod(static_cast<double>(X), G.dx), y = dd::two_prod(static_cast<double>(Y), G.dy),
           z = dd::two_prod(static_cast<double>(Z), G.dz);
  switch (c) {
    case 0: return ddf(x, y, z);
    case 1: return ddf(y, x, z);
    case 2: return ddf(z, y, x);
    case 3: return ddg(x, y, z);
    case 4: return ddg(x, z, y);
    default: return ddg(y, z, x);
  }
}

__global__ void k_newell_grid(NewellGrid G) {
  const int64_t nxg = G.ex + 1, nyg = G.ey + 1, nzg = G.ez + 1;
  const int64_t n = 6 * nxg * nyg * nzg;
  const int64_t gid = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (gid >= n) return;
  const int64_t X = gid % nxg, Y = (gid / nxg) % nyg, Z = (gid / (nxg * nyg)) % nzg;
  const int c = static_cast<int>(gid / (nxg * nyg * nzg));
  G.F[gid] = newell_fn(c, X, Y, Z, G);
}

// grid value with the parity of component c; offsets beyond the grid (not
// reached by the near field) are evaluated directly
__device__ DD newell_at(int c, int64_t X, int64_t Y, int64_t Z, const NewellGrid& G) {
  const int64_t ax = X < 0 ? -X : X, ay = Y < 0 ? -Y : Y, az = Z < 0 ? -Z : Z;
  if (ax > G.ex || ay > G.ey || az > G.ez) return newell_fn(c, X, Y, Z, G);
  const DD v = G.F[((static_cast<int64_t>(c) * (G.ez + 1) + az) * (G.ey + 1) + ay) * (G.ex + 1) + ax];
  const bool flip = (odd_axis(c, 0) && X < 0) ^ (odd_axis(c, 1) && Y < 0) ^ (odd_axis(c, 2) && Z < 0);
  return flip ? dd::neg(v) : v;
}

// dipolar_tensor_xx / _xy (atomistic/demag.jl:106-138) * V / (4 pi), permuted
// per component, in double-double
__device__ DD newell_dipole(int c, DD x, DD y, DD z, const DD& V4pi) {
  const DD x2 = dd::mul(x, x), y2 = dd::mul(y, y), z2 = dd::mul(z, z);
  const DD r2 = dd::add(dd::add(x2, y2), z2);
  DD num;
  switch (c) {
    case 0: num = dd::neg(dd::sub(dd::sub(dd::scale2(x2, 2.0), y2), z2)); break;
    case 1: num = dd::neg(dd::sub(dd::sub(dd::scale2(y2, 2.0), x2), z2)); break;
    case 2: num = dd::neg(dd::sub(dd::sub(dd::scale2(z2, 2.0), y2), x2)); break;
    case 3: num = dd::mul(dd::mul(x, y), -3.0); break;
    case 4: num = dd::mul(dd::mul(x, z), -3.0); break;
    default: num = dd::mul(dd::mul(y, z), -3.0); break;
  }
  return dd::mul(dd::div(num, dd::mul(dd::mul(r2, r2), dd::sqrt(r2))), V4pi);
}

// tensors_kernel_*!  src/micro/demag.jl:298-386: one thread per (component,
// cell offset), summing the macro-PBC images
__global__ void k_newell(double* __restrict__ out, int nx, int ny, int nz, int Nx, int Ny, int Nz, NewellGrid G) {
  const int64_t N = static_cast<int64_t>(nx) * ny * nz;
  const int64_t gid = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (gid >= 6 * N) return;
  const int c = static_cast<int>(gid / N);
  const int64_t I = gid - c * N;
  const int i = static_cast<int>(I % nx), j = static_cast<int>((I / nx) % ny),
            k = static_cast<int>(I / (static_cast<int64_t>(nx) * ny));
  const double mx = fmax(G.dx, fmax(G.dy, G.dz));
  const DD V = dd::mul(dd::two_prod(G.dx, G.dy), G.dz);
  const DD pi4 = dd::scale2(DD{dd::kPiHi, dd::kPiLo}, 4.0);
  const DD inv_near = dd::div(dd::mk(1.0), dd::mul(pi4, V));  // 1 / (4 pi dx dy dz)
  const DD V4pi = dd::div(V, pi4);
  DD sum = dd::mk(0.0);
  for (int p = -Nx; p <= Nx; ++p)
    for (int q = -Ny; q <= Ny; ++q)
      for (int r = -Nz; r <= Nz; ++r) {
        const int64_t X = i + static_cast<int64_t>(p) * nx, Y = j + static_cast<int64_t>(q) * ny,
                      Z = k + static_cast<int64_t>(r) * nz;
        // the switch as the reference evaluates it: FP64 coordinates, no contraction
        const double xd = __dmul_rn(static_cast<double>(X), G.dx), yd = __dmul_rn(static_cast<double>(Y), G.dy),
                     zd = __dmul_rn(static_cast<double>(Z), G.dz);
        const double Rc = __ddiv_rn(__dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(xd, xd), __dmul_rn(yd, yd)),
                                                          __dmul_rn(zd, zd))),
                                    mx);
        if (Rc > 60) {
          const DD x = dd::two_prod(static_cast<double>(X), G.dx), y = dd::two_prod(static_cast<double>(Y), G.dy),
                   z = dd::two_prod(static_cast<double>(Z), G.dz);
          sum = dd::add(sum, newell_dipole(c, x, y, z, V4pi));
          continue;
        }
        // 27-point second difference, 1-D weights w(0) = 2, w(+-1) = -1
        DD s = dd::mk(0.0);
        for (int a = -1; a <= 1; ++a)
          for (int b = -1; b <= 1; ++b)
            for (int e = -1; e <= 1; ++e) {
              const double w = (a == 0 ? 2.0 : -1.0) * (b == 0 ? 2.0 : -1.0) * (e == 0 ? 2.0 : -1.0);
              const DD v = newell_at(c, X + a, Y + b, Z + e, G);
              s = dd::add(s, DD{v.hi * w, v.lo * w});
            }
        sum = dd::add(sum, dd::mul(s, inv_near));
      }
  out[gid] = dd::to_double(sum);
}

int newell_tensor_device(int nx, int ny, int nz, double dx, double dy, double dz, int Nx, int Ny,
                         int Nz, double* out_dev, cudaStream_t st) {
  const double mx = std::max(dx, std::max(dy, dz));
  NewellGrid G;
  G.dx = dx / mx;
  G.dy = dy / mx;
  G.dz = dz / mx;
  // near-field offsets |X| dx <= 60 (R <= 60 cells), plus the stencil's +-1,
  // within the offsets the mesh and its images reach
  auto extent = [](double d, int n, int Nimg) {
    const double e = std::floor(60.0 / d) + 2.0;
    const double reach = static_cast<double>(n - 1) + static_cast<double>(Nimg) * n + 1.0;
    return static_cast<int>(std::min(e, reach));
  };
  G.ex = extent(G.dx, nx, Nx);
  G.ey = extent(G.dy, ny, Ny);
  G.ez = extent(G.dz, nz, Nz);
  const int64_t ng = 6LL * (G.ex + 1) * (G.ey + 1) * (G.ez + 1);
  G.F = nullptr;
  cudaError_t e = cudaMalloc(reinterpret_cast<void**>(&G.F), sizeof(DD) * ng);
  if (e != cudaSuccess) return static_cast<int>(e);
  const int T = 128;
  k_newell_grid<<<static_cast<unsigned>((ng + T - 1) / T), T, 0, st>>>(G);
  const int64_t tot = 6 * static_cast<int64_t>(nx) * ny * nz;
  k_newell<<<static_cast<unsigned>((tot + T - 1) / T), T, 0, st>>>(out_dev, nx, ny, nz, Nx, Ny, Nz, G);
  e = cudaGetLastError();
  const cudaError_t es = cudaStreamSynchronize(st);
  cudaFree(G.F);
  return static_cast<int>(e != cudaSuccess ? e : es);
}


// ============================================================ host side ====
LaunchRecorder*& launch_recorder() {
  thread_local LaunchRecorder* r = nullptr;
  return r;
}

bool pdl_enabled() {
  static const bool on = [] {
    const char* e = getenv("MMCUDA_PDL");
    return !(e && e[0] == '0');
  }();
  return on;
}

void smem_optin(const void* kernel) {
  static std::mutex mu;
  static std::set<std::pair<const void*, int>> done;
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lk(mu);
  if (done.count({kernel, dev})) return;
  // the opt-in limit covers static and dynamic shared memory together
  cudaFuncAttributes fa{};
  cudaFuncGetAttributes(&fa, kernel);
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       static_cast<int>(kMaxSmem) - static_cast<int>(fa.sharedSizeBytes));
  done.insert({kernel, dev});
}

// exp(-2 pi i t / L)
template <typename C> static C unit_root(int64_t t, int L) {
  const long double a = -2.0L * 3.141592653589793238462643383279502884L * static_cast<long double>(t) / L;
  C c;
  c.x = static_cast<decltype(C::x)>(static_cast<double>(cosl(a)));
  c.y = static_cast<decltype(C::x)>(static_cast<double>(sinl(a)));
  return c;
}

// exp(-2 pi i t / L), t < L
template <typename C> static std::vector<C> twiddle_table(int L) {
  std::vector<C> h(L);
  for (int t = 0; t < L; ++t) h[t] = unit_root<C>(t, L);
  return h;
}

template <typename C> static C* upload_table(const std::vector<C>& h, size_t& bytes, cudaStream_t st) {
  const size_t n = sizeof(C) * h.size();
  C* d = nullptr;
  if (cudaMalloc(&d, n) != cudaSuccess) return nullptr;
  bytes += n;
  cudaMemcpyAsync(d, h.data(), n, cudaMemcpyHostToDevice, st);
  cudaStreamSynchronize(st);
  return d;
}

// the table of length L; Q > 0 (L = 64 Q, the register passes): followed by
// their table exp(-2 pi i q k / (L / 2)) at k Q + q, k < 32, q < Q
template <typename C>
static C* upload_twiddles(std::vector<C> h, size_t& bytes, cudaStream_t st, int Q = 0) {
  for (int k = 0; k < (Q > 0 ? 32 : 0); ++k)
    for (int q = 0; q < Q; ++q) h.push_back(C(h[2 * q * k]));
  return upload_table(h, bytes, st);
}
template <typename C>
static C* upload_twiddles(int L, size_t& bytes, cudaStream_t st) {
  return upload_table(twiddle_table<C>(L), bytes, st);
}

template <typename R>
DemagPlan<R>::~DemagPlan() {
  cudaFree(X);
  cudaFree(Y);
  cudaFree(S);
  cudaFree(Zx);
  cudaFree(Zx2);
  cudaFree(Nhat);
  cudaFree(twx);
  cudaFree(twy);
  cudaFree(twz);
  cudaFree(rtab);
}

// The compile-time passes (mm_rf.cuh) where they apply, unless MMCUDA_RFFT=0
// (or the persistent step kernel, which runs the run-time-length bodies) keeps
// the run-time-length passes
static bool rfft_enabled() {
  static const bool on = [] {
    const char* e = getenv("MMCUDA_RFFT");
    return !(e && e[0] == '0');
  }();
  return on && !persist_enabled();
}
// Smaller meshes keep the run-time-length passes: their kernels are the same for
// every length, so a batch of uneven ones is a few merged launches.  The line is
// not the fastest one: with it at 64 cells a step of a 64 x 64 film took 45 us
// instead of 66 (FP32; 51 and 59 in FP64), and 32 films of 24 to 60 cells a side
// 0.14 ms in 352 launches instead of 0.22 in 16.
constexpr int64_t kRfftCells = 8192;

// tw2[(r-1) R1 + k] = w_{R1 R2}^(r k), tw3[(q-1) R1 R2 + i] = w_L^(q i), from
// the plan's table of length step L (sines of their own took 0.25 ms of the 5.5
// ms that add_demag takes for a 1000 x 1000 film)
template <typename C>
static void fill_rf_twiddles(const rf::Radices& f, const std::vector<C>& table, int step, std::vector<C>& out, size_t& o2,
                             size_t& o3) {
  const int L = f.r1 * f.r2 * f.r3, M = f.r1 * f.r2;
  o2 = out.size();
  for (int r = 1; r < f.r2; ++r)
    for (int k = 0; k < f.r1; ++k) out.push_back(unit_root<C>(r * k % M, M));
  o3 = out.size();
  for (int q = 1; q < f.r3; ++q)
    for (int i = 0; i < M; ++i) out.push_back(table[static_cast<int64_t>(q) * i % L * step]);
}

template <typename R>
int DemagPlan<R>::init(int nx, int ny, int nz, cudaStream_t st, char* err, size_t nerr, bool runtime_len) {
  constexpr bool f64 = sizeof(R) == 8;
  g.nx = nx; g.ny = ny; g.nz = nz;
  g.gate = nullptr;
  g.Px = padded_fft_len(nx, true);
  g.Py = padded_fft_len(ny, false);
  g.Pz = padded_fft_len(nz, false);
  // compile-time lengths: not for the power-of-two meshes of the register
  // passes (mm_wreg.cu), nor where a line has no instantiation
  rfft = rfft_z = runtime_ok = false;
  if (!runtime_len && rfft_enabled() && nx >= 8 && ny >= 8 && static_cast<int64_t>(nx) * ny * nz >= kRfftCells) {
    const bool zc2 = (g.Pz & (g.Pz - 1)) == 0 && g.Pz >= 4 && (g.Pz <= 128 || (!f64 && g.Pz == 256));
    const bool reg = nz > 1 && zc2 && wreg_enabled() && wreg_applies(nx, ny, nz, g.Px, g.Py, f64);
    const int lx = rf::next_length(rf::KX, f64, nx);
    const int ly = rf::next_length(nz == 1 ? rf::KC : rf::KY, f64, 2 * ny - 1);
    const int lz = nz >= 6 ? rf::next_length(rf::KZ, f64, 2 * nz - 1) : g.Pz;
    if (!reg && lx && ly && lz) {
      rfft = true;
      runtime_ok = nz == 1 && g.Px == 2 * lx && g.Py == ly &&
                   6 * sizeof(C) * static_cast<size_t>(padded_line_stride(ly)) <= kMaxSmem;
      g.Px = 2 * lx;
      g.Py = ly;
      g.Pz = lz;
      rfft_z = nz >= 6 && (f64 || !zpair_enabled() || lz != 32);  // FP32 Pz = 32: register z convolution
    }
  }
  g.Lc = g.Px > 1 ? g.Px / 2 : 0;
  g.Hx = g.Px > 1 ? g.Lc + 1 : 1;
  g.Tyq = g.Py / 2 + 1;
  g.Tzq = g.Pz / 2 + 1;
  g.Tys = g.Tyq;
  // one line (x, y; the three components of a z line) with its ping-pong
  // buffer must fit one block's shared memory, in the FP64 tensor passes too
  // x and y lines longer than one block holds (FP64 tensor passes included)
  // run as global-memory stages; z lines must fit
  const size_t c64 = sizeof(double2), cR = sizeof(C);
  long_x = 2 * c64 * static_cast<size_t>(g.Lc | 1) > kMaxSmem;
  long_y = 2 * c64 * static_cast<size_t>(g.Py | 1) > kMaxSmem;
  const bool fit_z = 2 * c64 * static_cast<size_t>(g.Pz | 1) <= kMaxSmem &&
                     2 * 3 * cR * static_cast<size_t>(g.Pz | 1) <= kMaxSmem;
  if (!fit_z) {
    snprintf(err, nerr, "demag: mesh %dx%dx%d exceeds the FFT pass limit (padded z <= %d)", nx, ny, nz,
             static_cast<int>(kMaxSmem / (6 * cR)) - 1);
    return -1;
  }
  // films: the y transform, tensor product and inverse of a column run in one
  // block when its three lines (two buffers) fit the tile budget, or, in the
  // column-major layout, one block's shared memory (one column per block);
  // longer film columns run the y transforms as global-memory stages
  // (coalesced across kx) instead of one-column shared-memory tiles
  const bool cols_ok = g.Px > 1 && !long_x;  // the global-memory x stages keep rows
  fused2d = !long_y && (g.Pz == 1) &&
            (2 * 3 * (g.Py | 1) * sizeof(C) <= static_cast<size_t>(smem_budget_bytes()) ||
             (cols_ok && 2 * 3 * static_cast<size_t>(padded_line_stride(g.Py)) * sizeof(C) <= kMaxSmem));
  if (rfft) fused2d = g.Pz == 1;
  if (g.Pz == 1 && !fused2d && cols_ok) long_y = true;
  g.xT = fused2d && cols_ok ? 1 : 0;
  // 3-D meshes whose shared-memory y lines leave row tiles narrower than 8
  // columns (16- to 64-byte row segments) keep the spectra column-major
  // (DemagGeom::yT) when the z convolution is the fused power-of-two kernel
  g.yT = 0;
  const bool zc2 = (g.Pz & (g.Pz - 1)) == 0 && g.Pz >= 4 && (g.Pz <= 128 || (sizeof(R) == 4 && g.Pz == 256));
  if (g.Pz > 1 && !rfft && !long_y && cols_ok && zc2 && cols3d_enabled()) {
    FftPlan1 py;
    make_fft_plan(g.Py, py, sizeof(R) == 4 ? fp32_max_radix() : 8);
    if (lines_tile<R>(g.Hx, g.Py, 1, std::max(1, line_fft_buffers(py))) < 8) g.yT = g.xT = 1;
  }
  g.wreg = 0;
  if (g.Pz > 1 && !rfft && !long_x && !long_y && zc2 && wreg_enabled() &&
      wreg_applies(nx, ny, nz, g.Px, g.Py, sizeof(R) == 8))
    g.wreg = g.yT = g.xT = 1;
  if ((long_x && !make_fft_plan(g.Lc, gplx, 8)) || (long_y && !make_fft_plan(g.Py, gply, 8))) {
    snprintf(err, nerr, "demag: no radix plan");
    return -1;
  }
  const int maxr = sizeof(R) == 4 ? fp32_max_radix() : 8;
  if (!make_fft_plan(g.Lc > 0 ? g.Lc : 1, g.plx, maxr) || !make_fft_plan(g.Py, g.ply, maxr) ||
      !make_fft_plan(g.Pz, g.plz, maxr)) {
    snprintf(err, nerr, "demag: no radix plan");
    return -1;
  }
  g.fLc = make_fastdiv(std::max(1, g.Lc));
  g.fHx = make_fastdiv(g.Hx);
  g.fPy = make_fastdiv(g.Py);
  g.fPz = make_fastdiv(g.Pz);
  g.fny = make_fastdiv(ny);
  g.fnz = make_fastdiv(nz);
  g.frows = make_fastdiv(ny * nz);
  g.fpady = make_fastdiv(std::max(1, g.Py - ny));
  g.fpadz = make_fastdiv(std::max(1, g.Pz - nz));
  wreg_set_attrs();
  const int64_t nX = 3LL * nz * ny * g.Hx;
  if (cudaMalloc(&X, sizeof(C) * nX) != cudaSuccess) return 2;
  bytes_ += sizeof(C) * nX;
  if (!fused2d) {
    const int64_t nY = 3LL * nz * g.Py * g.Hx;
    if (cudaMalloc(&Y, sizeof(C) * nY) != cudaSuccess) return 2;
    bytes_ += sizeof(C) * nY;
    if (long_y && !rfft) {
      if (cudaMalloc(&S, sizeof(C) * nY) != cudaSuccess) return 2;
      bytes_ += sizeof(C) * nY;
    }
  }
  if (long_x) {
    const int64_t nZ = 3LL * ny * nz * g.Lc;
    if (cudaMalloc(&Zx, sizeof(C) * nZ) != cudaSuccess || cudaMalloc(&Zx2, sizeof(C) * nZ) != cudaSuccess) return 2;
    bytes_ += 2 * sizeof(C) * nZ;
  }
  if (sizeof(R) == 4 && g.yT && zpair_enabled() && zpair_applies(g)) g.Tys = (g.Tyq + 3) & ~3;
  const int64_t nT = 6LL * g.Tzq * g.Tys * g.Hx;
  if (cudaMalloc(&Nhat, sizeof(R) * nT) != cudaSuccess) return 2;
  bytes_ += sizeof(R) * nT;
  cudaMemsetAsync(Nhat, 0, sizeof(R) * nT, st);
  if constexpr (sizeof(R) == 4) {
    if (g.yT && zpair_enabled() && zpair_applies(g) && !zpair_tensor_map(g, Nhat, zmap)) {
      snprintf(err, nerr, "demag: tensor map of the z convolution could not be encoded");
      return -1;
    }
  }
  const std::vector<C> hx = twiddle_table<C>(g.Px), hy = twiddle_table<C>(g.Py), hz = twiddle_table<C>(g.Pz);
  if (g.Px > 1 && !(twx = upload_twiddles<C>(hx, bytes_, st, g.wreg ? nx / 32 : 0))) return 2;
  if (!(twy = upload_twiddles<C>(hy, bytes_, st, g.wreg ? ny / 32 : 0))) return 2;
  if (!(twz = upload_twiddles<C>(hz, bytes_, st))) return 2;
  if (rfft) {
    std::vector<C> h;
    size_t o[6] = {};
    fill_rf_twiddles(rf::plan_of(rf::KX, f64, g.Lc), hx, 2, h, o[0], o[1]);  // Px = 2 Lc
    fill_rf_twiddles(rf::plan_of(fused2d ? rf::KC : rf::KY, f64, g.Py), hy, 1, h, o[2], o[3]);
    if (rfft_z) fill_rf_twiddles(rf::plan_of(rf::KZ, f64, g.Pz), hz, 1, h, o[4], o[5]);
    if (!(rtab = upload_table(h, bytes_, st))) return 2;
    rtx = {rtab + o[0], rtab + o[1]};
    rty = {rtab + o[2], rtab + o[3]};
    rtz = {rtab + o[4], rtab + o[5]};
  }
  return static_cast<int>(cudaGetLastError());
}

// ---- long lines: self-sorting Stockham stages through global memory -------
// For lines longer than one block's shared memory holds (two buffers), each
// radix stage is one launch that reads a whole spectrum array and writes the
// other of a ping-pong pair: y lines of [cz][Py][Hx] arrays (element stride
// Hx, the kx column fastest across threads) and x lines of [line][Lc] arrays
// (element stride 1, the butterfly fastest).  Same butterflies, twiddles and
// stage order as the shared-memory passes.
template <typename R, int RADIX, bool INV, bool ROWS>
__global__ void __launch_bounds__(256) k_gstage(const cplx_t<R>* __restrict__ src, cplx_t<R>* __restrict__ dst,
                                                int L, int64_t outer, int inner, int64_t los, int64_t es, int p,
                                                const cplx_t<R>* __restrict__ tw, int tw_mul, const int* __restrict__ gate) {
  using C = cplx_t<R>;
  if (gate && !*gate) return;
  const int T = L / RADIX;
  const int64_t total = outer * inner * static_cast<int64_t>(T);
  const int twstep = L / (p * RADIX) * tw_mul;
  for (int64_t idx = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    int64_t o;
    int w, i;
    if (ROWS) {  // x lines: butterfly fastest
      i = static_cast<int>(idx % T);
      const int64_t r = idx / T;
      w = static_cast<int>(r % inner);
      o = r / inner;
    } else {  // y lines: kx column fastest
      w = static_cast<int>(idx % inner);
      const int64_t r = idx / inner;
      i = static_cast<int>(r % T);
      o = r / T;
    }
    const int64_t base = o * los + w;
    const int k = i % p;
    C v[RADIX];
#pragma unroll
    for (int r = 0; r < RADIX; ++r) v[r] = src[base + static_cast<int64_t>(i + r * T) * es];
    if (p > 1) {
#pragma unroll
      for (int r = 1; r < RADIX; ++r) {
        C t = __ldg(tw + r * k * twstep);
        if (INV) t.y = -t.y;
        v[r] = cmul(v[r], t);
      }
    }
    dftR<RADIX, INV>(v);
    const int oo = (i - k) * RADIX + k;
#pragma unroll
    for (int r = 0; r < RADIX; ++r) dst[base + static_cast<int64_t>(oo + r * p) * es] = v[r];
  }
}

template <typename R, bool INV, bool ROWS>
static void launch_gstage(int radix, const cplx_t<R>* src, cplx_t<R>* dst, int L, int64_t outer, int inner,
                          int64_t los, int64_t es, int p, const cplx_t<R>* tw, int tw_mul, const int* gate,
                          cudaStream_t st) {
  const int64_t total = outer * inner * static_cast<int64_t>(L / radix);
  const int blocks = static_cast<int>(std::min<int64_t>((total + 255) / 256, 148 * 16));
  switch (radix) {
    case 8: k_gstage<R, 8, INV, ROWS><<<blocks, 256, 0, st>>>(src, dst, L, outer, inner, los, es, p, tw, tw_mul, gate); break;
    case 7: k_gstage<R, 7, INV, ROWS><<<blocks, 256, 0, st>>>(src, dst, L, outer, inner, los, es, p, tw, tw_mul, gate); break;
    case 5: k_gstage<R, 5, INV, ROWS><<<blocks, 256, 0, st>>>(src, dst, L, outer, inner, los, es, p, tw, tw_mul, gate); break;
    case 4: k_gstage<R, 4, INV, ROWS><<<blocks, 256, 0, st>>>(src, dst, L, outer, inner, los, es, p, tw, tw_mul, gate); break;
    case 3: k_gstage<R, 3, INV, ROWS><<<blocks, 256, 0, st>>>(src, dst, L, outer, inner, los, es, p, tw, tw_mul, gate); break;
    default: k_gstage<R, 2, INV, ROWS><<<blocks, 256, 0, st>>>(src, dst, L, outer, inner, los, es, p, tw, tw_mul, gate); break;
  }
}

// all stages of plan pl (radix <= 8) over the lines of buffer `a`, with `b`
// as the other buffer of the pair; returns the buffer holding the result
template <typename R, bool INV, bool ROWS>
static cplx_t<R>* glines_fft(const FftPlan1& pl, cplx_t<R>* a, cplx_t<R>* b, int64_t outer, int inner, int64_t los,
                             int64_t es, const cplx_t<R>* tw, int tw_mul, cudaStream_t st,
                             const int* gate = nullptr) {
  int p = 1;
  for (int s = 0; s < pl.nst; ++s) {
    const int R_ = plan_radix(pl, s);
    launch_gstage<R, INV, ROWS>(R_, a, b, pl.L, outer, inner, los, es, p, tw, tw_mul, gate, st);
    p *= R_;
    std::swap(a, b);
  }
  return a;
}

// y lines of the rows y < ny of X[cz][ny][Hx] into Y[cz][Py][Hx]: zero padded,
// or (tensor) mirrored with sign tsign (rows j >= Py - ny + 1 take row Py - j)
template <typename R>
__global__ void k_gy_expand(const cplx_t<R>* __restrict__ X, cplx_t<R>* __restrict__ Y, int ny, int Py, int Hx,
                            int64_t ncz, int tensor_sign, const int* __restrict__ gate = nullptr) {
  using C = cplx_t<R>;
  if (gate && !*gate) return;
  const int64_t total = ncz * Py * static_cast<int64_t>(Hx);
  for (int64_t e = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; e < total;
       e += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int kx = static_cast<int>(e % Hx);
    const int64_t r = e / Hx;
    const int j = static_cast<int>(r % Py);
    const int64_t cz = r / Py;
    C v = cmk<C>(R(0), R(0));
    if (j < ny) {
      v = X[(cz * ny + j) * Hx + kx];
    } else if (tensor_sign != 0 && j >= Py - ny + 1) {
      v = X[(cz * ny + (Py - j)) * Hx + kx];
      if (tensor_sign < 0) v = cmk<C>(-v.x, -v.y);
    }
    Y[e] = v;
  }
}

// rows y < ny of Y[cz][Py][Hx] back into X[cz][ny][Hx]
template <typename R>
__global__ void k_gy_extract(const cplx_t<R>* __restrict__ Y, cplx_t<R>* __restrict__ X, int ny, int Py, int Hx,
                             int64_t ncz, const int* __restrict__ gate) {
  if (gate && !*gate) return;
  const int64_t total = ncz * ny * static_cast<int64_t>(Hx);
  for (int64_t e = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; e < total;
       e += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int kx = static_cast<int>(e % Hx);
    const int64_t r = e / Hx;
    const int j = static_cast<int>(r % ny);
    const int64_t cz = r / ny;
    X[e] = Y[(cz * Py + j) * Hx + kx];
  }
}

// real part of ky <= Py/2 of Y[Py][Hx] times scale into Tq[Tyq][Hx] (films)
__global__ void k_gy_quadrant(const double2* __restrict__ Y, double* __restrict__ Tq, int Tyq, int Hx, double scale) {
  const int64_t total = static_cast<int64_t>(Tyq) * Hx;
  for (int64_t e = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; e < total;
       e += static_cast<int64_t>(gridDim.x) * blockDim.x)
    Tq[e] = Y[e].x * scale;
}

// film convolution in the y spectrum: H(kx, ky) = Nhat(kx, ky, kz = 0) M(kx, ky)
// for the three components of Y[c][Py][Hx] (nz = 1), tensor quadrant unfolded
template <typename R>
__global__ void k_gproduct_film(cplx_t<R>* __restrict__ Y, const R* __restrict__ Nhat, int Py, int Hx, int Tyq,
                                const int* __restrict__ gate) {
  using C = cplx_t<R>;
  if (gate && !*gate) return;
  const int64_t total = static_cast<int64_t>(Py) * Hx;
  const int64_t Ts = static_cast<int64_t>(Tyq) * Hx;  // Tzq = 1
  for (int64_t e = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; e < total;
       e += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int kx = static_cast<int>(e % Hx);
    const int ky = static_cast<int>(e / Hx);
    const bool fy = ky > Py / 2;
    const int kyq = fy ? Py - ky : ky;
    const R sy = fy ? R(-1) : R(1);
    const int64_t b = static_cast<int64_t>(kyq) * Hx + kx;
    const R xx = Nhat[b], yy = Nhat[Ts + b], zz = Nhat[2 * Ts + b];
    const R xy = sy * Nhat[3 * Ts + b], xz = Nhat[4 * Ts + b], yz = sy * Nhat[5 * Ts + b];
    const C p0 = Y[e], p1 = Y[total + e], p2 = Y[2 * total + e];
    Y[e] = cmk<C>(xx * p0.x + xy * p1.x + xz * p2.x, xx * p0.y + xy * p1.y + xz * p2.y);
    Y[total + e] = cmk<C>(xy * p0.x + yy * p1.x + yz * p2.x, xy * p0.y + yy * p1.y + yz * p2.y);
    Y[2 * total + e] = cmk<C>(xz * p0.x + yz * p1.x + zz * p2.x, xz * p0.y + yz * p1.y + zz * p2.y);
  }
}

static int gblocks(int64_t n) { return static_cast<int>(std::min<int64_t>((n + 255) / 256, 148 * 16)); }

// x lines longer than a block holds: pack the real rows (Ms*m, or the
// mirrored tensor row) as Lc complex pairs, transform, then the even/odd
// split of k_fwd_x; the inverse undoes it as k_inv_x does
template <typename R, int MODE>
__global__ void k_gx_pack(const R* __restrict__ m, const R* __restrict__ Ms, const double* __restrict__ Tr, int tsign,
                          cplx_t<R>* __restrict__ Z, int rows, int nx, int Lc, int Px, int64_t lines,
                          const int* __restrict__ gate = nullptr) {
  using C = cplx_t<R>;
  if (gate && !*gate) return;
  const int64_t N = static_cast<int64_t>(rows) * nx, total = lines * Lc;
  for (int64_t e = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; e < total;
       e += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int t = static_cast<int>(e % Lc);
    const int64_t line = e / Lc;
    const int64_t c = line / rows, row = line - c * rows;
    R v[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int u = 2 * t + h;
      R x = R(0);
      const int64_t I = row * nx;
      if (MODE == XM_MAGN) {
        if (u < nx) x = m[c * N + I + u] * Ms[I + u];
      } else {
        if (u < nx) x = static_cast<R>(Tr[I + u]);
        else if (u >= Px - nx + 1) x = static_cast<R>(tsign * Tr[I + (Px - u)]);
      }
      v[h] = x;
    }
    Z[e] = cmk<C>(v[0], v[1]);
  }
}

template <typename R>
__global__ void k_gx_post(const cplx_t<R>* __restrict__ Z, cplx_t<R>* __restrict__ X, int Lc, int Hx, int64_t lines,
                          const cplx_t<R>* __restrict__ twx, const int* __restrict__ gate = nullptr) {
  using C = cplx_t<R>;
  if (gate && !*gate) return;
  const int64_t total = lines * Hx;
  const R one_half = R(0.5);
  for (int64_t e = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; e < total;
       e += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int k = static_cast<int>(e % Hx);
    const int64_t l = e / Hx;
    const C* z = Z + l * Lc;
    const C zk = z[k == Lc ? 0 : k];
    const C zc = cconj(z[k == 0 ? 0 : Lc - k]);
    const C ev = cscale(cadd(zk, zc), one_half);
    const C od = crot<false>(cscale(csub(zk, zc), one_half));
    X[e] = cadd(ev, cmul(__ldg(twx + k), od));
  }
}

template <typename R>
__global__ void k_gx_pre(const cplx_t<R>* __restrict__ X, cplx_t<R>* __restrict__ Z, int Lc, int Hx, int64_t lines,
                         const cplx_t<R>* __restrict__ twx, const int* __restrict__ gate) {
  using C = cplx_t<R>;
  if (gate && !*gate) return;
  const int64_t total = lines * Lc;
  for (int64_t e = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; e < total;
       e += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int k = static_cast<int>(e % Lc);
    const int64_t l = e / Lc;
    const C* xr = X + l * Hx;
    const C a = xr[k];
    const C b = cconj(xr[Lc - k]);
    const C w = cconj(__ldg(twx + k));
    Z[e] = cadd(cadd(a, b), crot<true>(cmul(csub(a, b), w)));
  }
}

template <typename R>
__global__ void k_gx_unpack(const cplx_t<R>* __restrict__ Z, R* __restrict__ H, int rows, int nx, int Lc,
                            int64_t lines, const int* __restrict__ gate) {
  if (gate && !*gate) return;
  const int64_t N = static_cast<int64_t>(rows) * nx, total = lines * Lc;
  for (int64_t e = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; e < total;
       e += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int t = static_cast<int>(e % Lc);
    const int64_t line = e / Lc;
    const int64_t c = line / rows, row = line - c * rows;
    const auto z = Z[e];
    const int u = 2 * t;
    R* out = H + c * N + row * nx;
    if (u < nx) out[u] = z.x;
    if (u + 1 < nx) out[u + 1] = z.y;
  }
}

// ---- launch helpers shared by apply() and the tensor assembly ------------
template <typename R, int MODE, int NT>
static void launch_ypass(const DemagGeom& g, const cplx_t<R>* in, cplx_t<R>* out, const R* Nhat, double* Tq,
                         int ncompc, int ncomp, const cplx_t<R>* twy, int tsign, double tscale, cudaStream_t st) {
  using C = cplx_t<R>;
  const int W = floor_pow2(std::max(1, std::min(g.Hx, PassCfg<R, NT>::cap / (ncompc * g.Py))));
  dim3 grid((g.Hx + W - 1) / W, g.nz, ncomp / ncompc);
  const int half = ncompc * W * (g.Py | 1);
  const size_t sm = 2 * sizeof(C) * half;
  if (sm > 48 * 1024) smem_optin(reinterpret_cast<const void*>(&k_ypass<R, MODE, NT>));
  k_ypass<R, MODE, NT><<<grid, NT, sm, st>>>(in, out, Nhat, Tq, g, ilog2(W), ncompc, twy, tsign, tscale, half);
}

template <typename R, int MODE, int NT>
static void launch_zpass(const DemagGeom& g, cplx_t<R>* Y, const R* Nhat, double* Tq, int ncompc, int kyrows,
                         const cplx_t<R>* twz, int tsign, double tscale, cudaStream_t st) {
  using C = cplx_t<R>;
  const int nrow = (MODE == ZM_CONV && g.Py > 2) ? 2 : 1;  // ky and its mirror row
  const int W = floor_pow2(std::max(1, std::min(g.Hx, PassCfg<R, NT>::cap / (nrow * ncompc * g.Pz))));
  dim3 grid((g.Hx + W - 1) / W, kyrows, 1);
  const int half = nrow * ncompc * W * (g.Pz | 1);
  const size_t sm = 2 * sizeof(C) * half;
  if (sm > 48 * 1024) smem_optin(reinterpret_cast<const void*>(&k_zpass<R, MODE, NT>));
  k_zpass<R, MODE, NT><<<grid, NT, sm, st>>>(Y, Nhat, Tq, g, ilog2(W), ncompc, twz, tsign, tscale, half);
}

template <typename R>
static bool run_pass(const DemagPlan<R>& p, DemagGeom g, int which, const R* m, const R* mu0Ms, R* Hd,
                     cudaStream_t st, bool runtime_len = false) {
  using C = cplx_t<R>;
  constexpr int NT = kHotNT;
  const int64_t xlines = 3LL * g.ny * g.nz, ncz = 3LL * g.nz;
  if (g.wreg && which != 2) {
    launch_wreg(which, g, m, mu0Ms, p.X, p.Y, Hd, p.twx, p.twy, st);
    return true;
  }
  if (p.rfft && !runtime_len) {
    const int rows = g.ny * g.nz;
    switch (which) {
      case 0: rf::fwd_x<R>(g.Lc, m, mu0Ms, p.X, p.rtx, p.twx, g.gate, g.nx, rows, g.xT, st); return true;
      case 1:
        if (p.fused2d) return false;
        rf::fwd_y<R>(g.Py, p.X, p.Y, p.rty, g.gate, g.ny, g.nz, g.Hx, st);
        return true;
      case 2:
        if (p.fused2d) rf::conv_film<R>(g.Py, p.X, p.Nhat, p.rty, g.gate, g.ny, g.Hx, st);
        else if (p.rfft_z) rf::conv_z<R>(g.Pz, p.Y, p.Nhat, p.rtz, g.gate, g.nz, g.Hx, g.Py, st);
        else launch_zconv<R>(g, p.Y, p.Nhat, p.twz, st, p.tile[2], p.zmap);
        return true;
      case 3:
        if (p.fused2d) return false;
        rf::inv_y<R>(g.Py, p.Y, p.X, p.rty, g.gate, g.ny, g.nz, g.Hx, st);
        return true;
      case 4: rf::inv_x<R>(g.Lc, p.X, Hd, p.rtx, p.twx, g.gate, g.nx, rows, g.xT, st); return true;
      default: return false;
    }
  }
  switch (which) {
    case 0:
      if (p.long_x) {
        k_gx_pack<R, XM_MAGN><<<gblocks(xlines * g.Lc), 256, 0, st>>>(m, mu0Ms, nullptr, 1, p.Zx, g.ny * g.nz, g.nx,
                                                                     g.Lc, g.Px, xlines, g.gate);
        C* z = glines_fft<R, false, true>(p.gplx, p.Zx, p.Zx2, xlines, 1, g.Lc, 1, p.twx, 2, st, g.gate);
        k_gx_post<R><<<gblocks(xlines * g.Hx), 256, 0, st>>>(z, p.X, g.Lc, g.Hx, xlines, p.twx, g.gate);
        return true;
      }
      launch_fwd_x<R, XM_MAGN, NT>(g, m, mu0Ms, nullptr, 1, p.X, 3, p.twx, st);
      return true;
    case 1:
      if (p.fused2d) return false;
      if (p.long_y) {
        // start in the buffer that leaves the result in Y after nst stages
        C* a = (p.gply.nst & 1) ? p.S : p.Y;
        k_gy_expand<R><<<gblocks(ncz * g.Py * g.Hx), 256, 0, st>>>(p.X, a, g.ny, g.Py, g.Hx, ncz, 0, g.gate);
        glines_fft<R, false, false>(p.gply, a, a == p.Y ? p.S : p.Y, ncz, g.Hx, static_cast<int64_t>(g.Py) * g.Hx,
                                    g.Hx, p.twy, 1, st, g.gate);
        return true;
      }
      launch_ylines<R, YL_FWD>(g, p.X, p.Y, p.Nhat, p.twy, st, p.tile[1]);
      return true;
    case 2:
      if (p.fused2d) launch_ylines<R, YL_CONV2D>(g, p.X, p.X, p.Nhat, p.twy, st, runtime_len ? 0 : p.tile[2]);
      else if (p.long_y && g.Pz == 1)
        k_gproduct_film<R><<<gblocks(static_cast<int64_t>(g.Py) * g.Hx), 256, 0, st>>>(p.Y, p.Nhat, g.Py, g.Hx, g.Tyq,
                                                                                    g.gate);
      else launch_zconv<R>(g, p.Y, p.Nhat, p.twz, st, p.tile[2], p.zmap);
      return true;
    case 3:
      if (p.fused2d) return false;
      if (p.long_y) {
        C* r = glines_fft<R, true, false>(p.gply, p.Y, p.S, ncz, g.Hx, static_cast<int64_t>(g.Py) * g.Hx, g.Hx,
                                          p.twy, 1, st, g.gate);
        k_gy_extract<R><<<gblocks(ncz * g.ny * g.Hx), 256, 0, st>>>(r, p.X, g.ny, g.Py, g.Hx, ncz, g.gate);
        return true;
      }
      launch_ylines<R, YL_INV>(g, p.Y, p.X, p.Nhat, p.twy, st, p.tile[3]);
      return true;
    case 4: {
      const int lines = 3 * g.ny * g.nz;
      if (p.long_x) {
        k_gx_pre<R><<<gblocks(xlines * g.Lc), 256, 0, st>>>(p.X, p.Zx, g.Lc, g.Hx, xlines, p.twx, g.gate);
        C* z = glines_fft<R, true, true>(p.gplx, p.Zx, p.Zx2, xlines, 1, g.Lc, 1, p.twx, 2, st, g.gate);
        k_gx_unpack<R><<<gblocks(xlines * g.Lc), 256, 0, st>>>(z, Hd, g.ny * g.nz, g.nx, g.Lc, xlines, g.gate);
        return true;
      }
      if (g.Px == 1) {
        k_inv_x1<R><<<(lines + 255) / 256, 256, 0, st>>>(p.X, Hd, lines, g.gate);
      } else {
        launch_inv_x<R>(g, p.X, Hd, p.twx, st);
      }
      return true;
    }
    default:
      return false;
  }
}

template <typename R>
void DemagPlan<R>::apply(const R* m, const R* mu0Ms, R* Hd, cudaStream_t st, const int* gate, bool runtime_len) {
  DemagGeom gg = this->g;
  gg.gate = gate;
  for (int which = 0; which < 5; ++which) run_pass(*this, gg, which, m, mu0Ms, Hd, st, runtime_len && runtime_ok);
}

template <typename R>
bool DemagPlan<R>::launch_pass(int which, const R* m, const R* mu0Ms, R* Hd, cudaStream_t st) {
  return run_pass(*this, this->g, which, m, mu0Ms, Hd, st);
}

// ---- tile autotuner ---------------------------------------------------------
// For each strided pass the plan uses, time every valid tile width W (powers
// of two up to a 128-byte row segment, within the 200 KB shared-memory limit
// and, for the fused-middle z kernel, W * RA <= threads) on the plan's own
// buffers and keep the fastest.  Results are cached per (form, kind of
// lengths, mesh shape), so a batch of equal meshes tunes once.  MMCUDA_AUTOTUNE=0 keeps the static
// rule.
struct TileKey {
  int w;
  bool rfft;
  int nx, ny, nz;
  bool operator<(const TileKey& o) const {
    return std::tie(w, rfft, nx, ny, nz) < std::tie(o.w, o.rfft, o.nx, o.ny, o.nz);
  }
};
static std::mutex g_tile_mu;
static std::map<TileKey, std::array<int, 5>> g_tile_cache;

template <typename R>
int DemagPlan<R>::autotune(const R* m, const R* mu0Ms, R* Hd, cudaStream_t st) {
  using C = cplx_t<R>;
  const char* env = getenv("MMCUDA_AUTOTUNE");
  if (env && env[0] == '0') return 0;
  const TileKey key{static_cast<int>(sizeof(R)), rfft, g.nx, g.ny, g.nz};
  {
    std::lock_guard<std::mutex> lk(g_tile_mu);
    auto it = g_tile_cache.find(key);
    if (it != g_tile_cache.end()) {
      for (int i = 0; i < 5; ++i) tile[i] = it->second[i];
      return 0;
    }
  }
  cudaEvent_t e0, e1;
  if (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess) return -1;
  const int wmax = 128 / static_cast<int>(sizeof(C));
  const int ra = zconv2_ra(g.Pz);
  const bool zc2 = !fused2d && pass_smem<R>(g, 2, false, 1) == sizeof(C) * 3 * (g.Pz | 1);
  for (int which = 1; which <= 3; ++which) {
    if (fused2d && which != 2) continue;
    if (rfft && (which != 2 || fused2d || rfft_z)) {  // one width a length
      const rf::Kind k = which != 2 ? rf::KY : (fused2d ? rf::KC : rf::KZ);
      tile[which] = rf::tile_width(k, sizeof(R) == 8, which == 2 && !fused2d ? g.Pz : g.Py);
      continue;
    }
    if (long_y && (which != 2 || g.Pz == 1)) continue;  // global-memory stages have no tile
    if (g.wreg && which != 2) continue;                  // register passes have no tile
    if (which == 2 && (sizeof(R) == 4 ? zpair_enabled() && zpair_applies(g) : zquad_applies(g))) continue;
    // the static rule's W is the incumbent; another W must be 3 % faster
    // (timing noise, e.g. under a profiler, then cannot move the choice)
    tile[which] = 0;
    int W0 = 1;
    {
      const int nb = which == 2 ? (fused2d ? 2 : (zc2 ? 1 : 2)) : std::max(1, line_fft_buffers(g.ply));
      W0 = which == 2 && !fused2d ? lines_tile<R>(g.yT ? g.Py : g.Hx, g.Pz, 3, nb)
                                  : lines_tile<R>(g.Hx, g.Py, which == 2 ? 3 : 1, nb);
      if (which == 2 && zc2)
        while (W0 * ra > zconv2_nt<R>()) W0 /= 2;
    }
    float ms0 = 0.f, best = 1e30f;
    int bestW = W0;
    for (int W = 1; W <= wmax; W *= 2) {
      if (W / 2 >= (which == 2 && g.yT ? g.Py : g.Hx)) break;
      if (pass_smem<R>(g, which, fused2d, W) > kMaxSmem) break;
      if (which == 2 && zc2 && W * ra > zconv2_nt<R>()) break;
      tile[which] = W;
      for (int r = 0; r < 2; ++r) run_pass(*this, g, which, m, mu0Ms, Hd, st);
      cudaEventRecord(e0, st);
      for (int r = 0; r < 6; ++r) run_pass(*this, g, which, m, mu0Ms, Hd, st);
      cudaEventRecord(e1, st);
      if (cudaEventSynchronize(e1) != cudaSuccess) break;
      float ms = 0.f;
      cudaEventElapsedTime(&ms, e0, e1);
      if (W == W0) ms0 = ms;
      if (ms < best) {
        best = ms;
        bestW = W;
      }
    }
    if (ms0 > 0.f && best > 0.97f * ms0) {
      bestW = W0;
      best = ms0;
    }
    tile[which] = bestW;
    tile_ms[which] = best / 6;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  const cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) return static_cast<int>(err);
  std::lock_guard<std::mutex> lk(g_tile_mu);
  g_tile_cache[key] = {tile[0], tile[1], tile[2], tile[3], tile[4]};
  return 0;
}

template <typename R>
double DemagPlan<R>::pass_bytes(int which) const {
  const double w = sizeof(R), cw = 2.0 * sizeof(R);
  const double rows = static_cast<double>(g.ny) * g.nz, N = rows * g.nx;
  const double nX = 3.0 * rows * g.Hx, nY = 3.0 * g.nz * g.Py * g.Hx;
  const double Ts = static_cast<double>(g.Tzq) * g.Tyq * g.Hx;
  switch (which) {
    case 0: return 4.0 * N * w + nX * cw;
    case 1: return fused2d ? 0.0 : (nX + nY) * cw;
    case 2: return (fused2d ? 2.0 * nX : 2.0 * nY) * cw + 6.0 * Ts * w;
    case 3: return fused2d ? 0.0 : (nX + nY) * cw;
    case 4: return nX * cw + 3.0 * N * w;
    default: return 0.0;
  }
}

template <typename R>
bool DemagPlan<R>::batchable() const {
  // the paths of run_pass that launch FwdX, YLines, ZConv and InvX only
  if (long_x || (long_y && !rfft) || g.Px == 1 || g.wreg) return false;
  if (fused2d || rfft_z) return true;
  if (sizeof(R) == 4 && zpair_enabled() && zpair_applies(g)) return false;
  switch (g.Pz) {
    case 4: case 8: case 16: case 32: case 64: case 128: return false;  // k_zconv2
    case 256: return sizeof(R) != 4;
    default: return true;
  }
}

template <typename R>
int DemagPlan<R>::launches_per_apply() const {
  if (fused2d) return 3;
  int n = 1;                                          // conv
  n += long_x ? 2 * (gplx.nst + 2) : 2;               // x forward / inverse
  n += long_y ? 2 * (gply.nst + 1) : 2;               // y forward / inverse
  return n;
}

// Tensor spectrum: for each component, forward r2c-x / y / z transforms of
// the mirrored, padded real-space tensor in FP64, real part of the
// (kx, ky<=Py/2, kz<=Pz/2) quadrant, scaled by -1/(mu0 Px Py Pz).
template <typename R>
int DemagPlan<R>::set_tensor(const double* T6N, cudaStream_t st) {
  using C64 = double2;
  constexpr int NT = kTensorNT;
  size_t b64 = 0;
  C64 *tx = nullptr, *ty = nullptr, *tz = nullptr, *X64 = nullptr, *Y64 = nullptr;
  double* Tq = nullptr;
  const int64_t N = static_cast<int64_t>(g.nx) * g.ny * g.nz;
  const int64_t nX = static_cast<int64_t>(g.nz) * g.ny * g.Hx;
  const int64_t nY = static_cast<int64_t>(g.nz) * g.Py * g.Hx;
  const int64_t Ts = static_cast<int64_t>(g.Tzq) * g.Tyq * g.Hx;
  // FP64 plans (radix <= 8) for the same lengths
  DemagGeom g64 = g;
  make_fft_plan(g.Lc > 0 ? g.Lc : 1, g64.plx, 8);
  make_fft_plan(g.Py, g64.ply, 8);
  make_fft_plan(g.Pz, g64.plz, 8);
  int rc = 0;
  if (g.Px > 1 && !(tx = upload_twiddles<C64>(g.Px, b64, st))) rc = 2;
  if (!rc && !(ty = upload_twiddles<C64>(g.Py, b64, st))) rc = 2;
  if (!rc && !(tz = upload_twiddles<C64>(g.Pz, b64, st))) rc = 2;
  C64 *Z64 = nullptr, *Z64b = nullptr, *S64 = nullptr;
  const int64_t nZ = static_cast<int64_t>(g.ny) * g.nz * g.Lc;
  if (!rc && cudaMalloc(&X64, sizeof(C64) * nX) != cudaSuccess) rc = 2;
  if (!rc && (g.Pz > 1 || long_y) && cudaMalloc(&Y64, sizeof(C64) * nY) != cudaSuccess) rc = 2;
  if (!rc && long_y && cudaMalloc(&S64, sizeof(C64) * nY) != cudaSuccess) rc = 2;
  if (!rc && long_x && (cudaMalloc(&Z64, sizeof(C64) * nZ) != cudaSuccess || cudaMalloc(&Z64b, sizeof(C64) * nZ) != cudaSuccess))
    rc = 2;
  if (!rc && cudaMalloc(&Tq, sizeof(double) * 6 * Ts) != cudaSuccess) rc = 2;
  if (!rc) {
    const double scale = -1.0 / (kMu0 * static_cast<double>(g.Px) * g.Py * g.Pz);
    const int64_t rows = static_cast<int64_t>(g.ny) * g.nz;
    for (int c = 0; c < 6; ++c) {
      const int sx = odd_axis(c, 0) ? -1 : 1, sy = odd_axis(c, 1) ? -1 : 1, sz = odd_axis(c, 2) ? -1 : 1;
      if (long_x) {
        k_gx_pack<double, XM_TENSOR><<<gblocks(rows * g.Lc), 256, 0, st>>>(nullptr, nullptr, T6N + c * N, sx, Z64,
                                                                          static_cast<int>(rows), g.nx, g.Lc, g.Px,
                                                                          rows);
        C64* z = glines_fft<double, false, true>(gplx, Z64, Z64b, rows, 1, g.Lc, 1, tx, 2, st);
        k_gx_post<double><<<gblocks(rows * g.Hx), 256, 0, st>>>(z, X64, g.Lc, g.Hx, rows, tx);
      } else {
        launch_fwd_x<double, XM_TENSOR, NT>(g64, nullptr, nullptr, T6N + c * N, sx, X64, 1, tx, st);
      }
      if (long_y) {
        // mirrored y lines in global memory; the result lands in Y64
        C64* a = (gply.nst & 1) ? S64 : Y64;
        k_gy_expand<double><<<gblocks(static_cast<int64_t>(g.nz) * g.Py * g.Hx), 256, 0, st>>>(
            X64, a, g.ny, g.Py, g.Hx, g.nz, sy);
        glines_fft<double, false, false>(gply, a, a == Y64 ? S64 : Y64, g.nz, g.Hx,
                                         static_cast<int64_t>(g.Py) * g.Hx, g.Hx, ty, 1, st);
        if (g.Pz == 1)
          k_gy_quadrant<<<gblocks(static_cast<int64_t>(g.Tyq) * g.Hx), 256, 0, st>>>(Y64, Tq + c * Ts, g.Tyq, g.Hx,
                                                                                      scale);
        else
          launch_zpass<double, ZM_TENSOR_Q, NT>(g64, Y64, nullptr, Tq + c * Ts, 1, g.Tyq, tz, sz, scale, st);
      } else if (g.Pz == 1) {
        launch_ypass<double, YM_TENSOR_Q, NT>(g64, X64, nullptr, nullptr, Tq + c * Ts, 1, 1, ty, sy, scale, st);
      } else {
        launch_ypass<double, YM_TENSOR, NT>(g64, X64, Y64, nullptr, nullptr, 1, 1, ty, sy, 0.0, st);
        launch_zpass<double, ZM_TENSOR_Q, NT>(g64, Y64, nullptr, Tq + c * Ts, 1, g.Tyq, tz, sz, scale, st);
      }
    }
    if (g.xT || g.yT) k_cast_cols<R><<<1024, 256, 0, st>>>(Tq, Nhat, g.Tyq, g.Tys, g.Hx, g.Tzq);
    else k_cast<R><<<1024, 256, 0, st>>>(Tq, Nhat, 6 * Ts);
    rc = static_cast<int>(cudaGetLastError());
    cudaStreamSynchronize(st);
  }
  cudaFree(tx); cudaFree(ty); cudaFree(tz); cudaFree(X64); cudaFree(Y64); cudaFree(Tq);
  cudaFree(S64); cudaFree(Z64); cudaFree(Z64b);
  return rc;
}

template class DemagPlan<float>;
template class DemagPlan<double>;

}  // namespace mm
