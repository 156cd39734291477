// Chains of block products for dense blocks of order at most 64 (small_blocks.cu).
#pragma once
#include "common.cuh"

namespace sdpx {

constexpr int kSmallOrder = 64;

// For every block b (k_b ≤ kSmallOrder, at off_b in the stacked arrays):
//   out = X⁻¹·T,  T = sign·(M·Y − R),  X⁻¹ = WᵀW  (W = L_X⁻¹, zeros above its diagonal),
// R may be null (T = sign·M·Y); sym: out ← (out + outᵀ)/2.  out may be R.
void block_xinv_my(const long long* d_off, const int* d_k, int nb, int kmax, const double* M, const double* Y,
                   const double* R, double sign, const double* W, double* out, bool sym, cudaStream_t st);

// G_s = W_s·D_s·W_sᵀ for the blocks of list (indices into d_off, d_k) and s = 0, 1.
struct Congruence {
  const double *W[2], *D[2];
  double* G[2];
};
void block_congruence(const long long* d_off, const int* d_k, const int* d_list, int n, int kmax,
                      const Congruence& q, cudaStream_t st);

}  // namespace sdpx
