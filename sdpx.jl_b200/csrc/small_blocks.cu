// Chains of block products for dense blocks of order at most 64, one CTA per block and all
// matrices in shared tiles (small_blocks.h).
//
// What bounds them is the latency of a launch: a product of order 64 is 2 µs of one SM's
// FP64 tensor pipe, as a launch of its own 5.5 µs and 1.5 to the next, and the host
// issues it in 4.  A right-hand side or direction took three such launches (and a
// symmetrisation): 16 µs and the gaps at order 50, 11 at order 12; one takes 13 and 4.8.
// The Newton step of m = 24, k = 12 went from 590 to 505 µs, of k = 61 + 17 from 1437 to
// 1410.
#include "small_blocks.h"
#include "tile64.cuh"

#include <algorithm>

namespace sdpx {
using namespace tile64;
namespace {

__global__ void __launch_bounds__(FT) k_block_xinv_my(const long long* __restrict__ off,
                                                      const int* __restrict__ kk, const double* M,
                                                      const double* Y, const double* R, double sign,
                                                      const double* W, double* out, int sym) {
  extern __shared__ __align__(16) double fsm[];
  const int k = kk[blockIdx.x], nb = (k + 7) >> 3, tile = 8 * nb * FLD;
  const long long o = off[blockIdx.x];
  double *S0 = fsm, *S1 = S0 + tile, *S2 = S1 + tile, *S3 = S2 + tile;
  cta_load_tile(S0, M + o, k);
  cta_load_tile(S1, Y + o, k);
  cta_load_tile(S2, W + o, k);
  __syncthreads();
  cta_tile_gemm<false, kFull>(S0, S1, nb, [&](int r, int c, double v) {
    S3[c * FLD + r] = sign * (R && r < k && c < k ? v - R[o + r + c * k] : v);
  });
  __syncthreads();
  if (!sym) {
    cta_tile_cholsolve(S2, S3, S0, nb, [&](int r, int c, double v) {
      if (r < k && c < k) out[o + r + c * k] = v;
    });
    return;
  }
  cta_tile_cholsolve(S2, S3, S0, nb, [&](int r, int c, double v) { S1[c * FLD + r] = v; });
  __syncthreads();
  for (int e = threadIdx.x; e < 64 * k; e += FT) {
    const int r = e & 63, c = e >> 6;
    if (r < k) out[o + r + c * k] = r == c ? S1[c * FLD + r] : (S1[c * FLD + r] + S1[r * FLD + c]) / 2;
  }
}

__global__ void __launch_bounds__(FT) k_block_congruence(const long long* __restrict__ off,
                                                         const int* __restrict__ kk,
                                                         const int* __restrict__ list, const Congruence q) {
  extern __shared__ __align__(16) double fsm[];
  const int b = list[blockIdx.x], s = blockIdx.y, k = kk[b], nb = (k + 7) >> 3, tile = 8 * nb * FLD;
  const long long o = off[b];
  double *S0 = fsm, *S1 = S0 + tile, *S2 = S1 + tile, *S3 = S2 + tile;
  cta_load_tile(S0, q.W[s] + o, k);
  cta_load_tile(S1, q.D[s] + o, k);
  cta_load_tile(S2, q.W[s] + o, k, true);
  __syncthreads();
  cta_tile_gemm<false, kLower>(S0, S1, nb, [&](int r, int c, double v) { S3[c * FLD + r] = v; });
  __syncthreads();
  cta_tile_gemm<false, kFull>(S3, S2, nb, [&](int r, int c, double v) {
    if (r < k && c < k) q.G[s][o + r + c * k] = v;
  });
}

size_t chain_smem(int kmax) { return 4 * sizeof(double) * (size_t)((kmax + 7) / 8 * 8) * FLD; }

}  // namespace

void block_xinv_my(const long long* d_off, const int* d_k, int nb, int kmax, const double* M, const double* Y,
                   const double* R, double sign, const double* W, double* out, bool sym, cudaStream_t st) {
  if (nb == 0) return;
  ensure_smem(k_block_xinv_my, chain_smem(kmax));
  k_block_xinv_my<<<nb, FT, chain_smem(kmax), st>>>(d_off, d_k, M, Y, R, sign, W, out, sym ? 1 : 0);
  SDPX_LAUNCH_CHECK();
}

void block_congruence(const long long* d_off, const int* d_k, const int* d_list, int n, int kmax,
                      const Congruence& q, cudaStream_t st) {
  if (n == 0) return;
  ensure_smem(k_block_congruence, chain_smem(kmax));
  k_block_congruence<<<dim3(n, 2), FT, chain_smem(kmax), st>>>(d_off, d_k, d_list, q);
  SDPX_LAUNCH_CHECK();
}

}  // namespace sdpx
