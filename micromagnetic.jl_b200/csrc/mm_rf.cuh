// mm_rf.cuh -- which line lengths the compile-time passes take, and their
// launchers (internal; kernels in mm_rfpass.cuh, instantiated by mm_rf_*.cu).
#pragma once
#include "mm_rfft.cuh"

namespace mm {
namespace rf {

enum Kind { KX = 0, KY = 1, KZ = 2, KC = 3 };  // x half length, y of 3-D meshes, z, film columns

// Smallest instantiated length >= n of a kind, 0 when there is none.
int next_length(Kind k, bool f64, int n);
// Radices of that length (the twiddle tables follow from them).
Radices plan_of(Kind k, bool f64, int L);
// Columns (lines) one block of the y, z or film kernel takes.
int tile_width(Kind k, bool f64, int L);

template <typename R> struct Tw {  // twiddle tables of one length
  const cplx_t<R>*tw2, *tw3;
};

template <typename R>
void fwd_x(int L, const R* m, const R* Ms, cplx_t<R>* X, Tw<R> t, const cplx_t<R>* twx, const int* gate, int nx,
           int rows, int cols, cudaStream_t st);
template <typename R>
void inv_x(int L, const cplx_t<R>* X, R* H, Tw<R> t, const cplx_t<R>* twx, const int* gate, int nx, int rows, int cols,
           cudaStream_t st);
template <typename R>
void fwd_y(int L, const cplx_t<R>* X, cplx_t<R>* Y, Tw<R> t, const int* gate, int ny, int nz, int Hx, cudaStream_t st);
template <typename R>
void inv_y(int L, const cplx_t<R>* Y, cplx_t<R>* X, Tw<R> t, const int* gate, int ny, int nz, int Hx, cudaStream_t st);
template <typename R>
void conv_z(int L, cplx_t<R>* Y, const R* Nhat, Tw<R> t, const int* gate, int nz, int Hx, int Py, cudaStream_t st);
template <typename R>
void conv_film(int L, cplx_t<R>* X, const R* Nhat, Tw<R> t, const int* gate, int ny, int Hx, cudaStream_t st);

}  // namespace rf
}  // namespace mm
