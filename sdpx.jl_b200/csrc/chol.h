// Batched Cholesky / triangular kernels (chol.cu).
#pragma once
#include <algorithm>

#include "common.cuh"

namespace sdpx {

template <class T>
struct MatDesc {
  T* a;     // column-major n×n, leading dimension ld
  int n;
  int ld;
};

// Lower Cholesky in place of every matrix in d_mats (device array of nmat
// descriptors, largest order nmax), one launch (potrf_flow.cu): a CTA per matrix
// runs the pivot chain, sms/nmat − 1 others its remaining tiles, ordered by tile
// flags.  info[b] = 0 on success, else the 1-based index of the first non-positive
// pivot (the no-throw contract of SDPX's `kchol!`, src/kernels/generic.jl:133-155),
// or −1 when a wait for a tile gave up (about a second).  dmin/dmax receive min/max
// |L_ii|.  The strict upper triangle is zeroed unless zero_upper is false (positive-
// definiteness tests that only read info/dmin/dmax).  `flags`
// (potrf_flow_flag_words(nmat, nmax) words) must not be shared by concurrent calls.
size_t potrf_flow_flag_words(int nmat, int nmax);
void potrf_flow(const MatDesc<double>* d_mats, int nmat, int nmax, int* info, double* dmin,
                double* dmax, unsigned* flags, int sms, cudaStream_t st, bool zero_upper = true);

// W_b = L_b^{-1} for lower-triangular L_b (W zero-initialised by the caller).
template <class T, int NB>
void trinv_batched(const MatDesc<T>* d_L, const MatDesc<T>* d_W, int nmat, int nmax,
                   cudaStream_t st);

// Inverses of the 64×64 diagonal tiles of a lower factor L (n×n): Dinv[s]
// (64×64, column-major), and into the diagonal tiles of Linv (n×n) unless null.
void factor_diag_inverses(const double* L, long long ld, int n, double* Dinv, double* Linv,
                          cudaStream_t st);

// rhs ← (L Lᵀ)^{-1} rhs by blocked forward/backward substitution (work: n).
template <class T, int NB>
void cholesky_solve(const T* L, long long ld, int n, const T* Dinv, T* rhs, T* work,
                    cudaStream_t st);

// Linv = L⁻¹ (n×n, column-major, ld n) by recursive doubling over 64×64 tiles.
// Dinv: ceil(n/64)·64·64 scratch, tmp: n·n scratch.
void trinv_recursive_f64(const double* L, int n, double* Linv, double* Dinv, double* tmp,
                         cudaStream_t st);

}  // namespace sdpx
