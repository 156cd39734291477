// Triangular inverses and solves with a lower Cholesky factor (the factorization
// itself: potrf_flow.cu).
#include "chol.h"
#include "blas_f64.h"

namespace sdpx {

// ---------------------------------------------------------------------------
// Triangular inverse W = L^{-1} (lower), blocked by NB.  Step 0 inverts every
// diagonal tile; step i fills block row i:  W[i,j] = -W[i,i] Σ_{p=j}^{i-1} L[i,p] W[p,j].
// W must be zero-initialised (its strict upper triangle stays zero).
// ---------------------------------------------------------------------------
template <class T, int NB>
__global__ void k_trinv_diag(const MatDesc<T>* Ls, const MatDesc<T>* Ws) {
  __shared__ T Lt[NB][NB + 1];
  __shared__ T Wt[NB][NB + 1];
  const MatDesc<T> L = Ls[blockIdx.y], W = Ws[blockIdx.y];
  const int s0 = blockIdx.x * NB;
  if (s0 >= L.n) return;
  const int w = min(NB, L.n - s0);
  for (int e = threadIdx.x; e < w * w; e += blockDim.x) {
    int r = e % w, c = e / w;
    Lt[c][r] = L.a[(size_t)(s0 + c) * L.ld + s0 + r];
  }
  __syncthreads();
  for (int c = threadIdx.x; c < w; c += blockDim.x) {
    Wt[c][c] = T(1) / Lt[c][c];
    for (int r = c + 1; r < w; ++r) {
      T s = T(0);
      for (int p = c; p < r; ++p) s += Lt[p][r] * Wt[c][p];
      Wt[c][r] = -s / Lt[r][r];
    }
    for (int r = 0; r < c; ++r) Wt[c][r] = T(0);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < w * w; e += blockDim.x) {
    int r = e % w, c = e / w;
    W.a[(size_t)(s0 + c) * W.ld + s0 + r] = Wt[c][r];
  }
}

template <class T, int NB>
__global__ void k_trinv_row(const MatDesc<T>* Ls, const MatDesc<T>* Ws, int i) {
  __shared__ T Acc[NB][NB + 1];
  __shared__ T Lt[NB][NB + 1];
  __shared__ T Wt[NB][NB + 1];
  const MatDesc<T> L = Ls[blockIdx.y], W = Ws[blockIdx.y];
  const int nt = (L.n + NB - 1) / NB;
  if (i >= nt) return;
  const int j = blockIdx.x;
  if (j >= i) return;
  const int r0 = i * NB, h = min(NB, L.n - r0);
  for (int e = threadIdx.x; e < NB * NB; e += blockDim.x) Acc[e / NB][e % NB] = T(0);
  for (int p = j; p < i; ++p) {
    const int p0 = p * NB;
    __syncthreads();
    for (int e = threadIdx.x; e < NB * NB; e += blockDim.x) {
      int r = e % NB, c = e / NB;
      Lt[c][r] = (r < h) ? L.a[(size_t)(p0 + c) * L.ld + r0 + r] : T(0);       // L[i,p]
      Wt[c][r] = W.a[(size_t)(j * NB + c) * W.ld + p0 + r];                     // W[p,j]
    }
    __syncthreads();
    for (int e = threadIdx.x; e < NB * NB; e += blockDim.x) {
      int r = e % NB, c = e / NB;
      T s = T(0);
#pragma unroll 8
      for (int q = 0; q < NB; ++q) s += Lt[q][r] * Wt[c][q];
      Acc[c][r] += s;
    }
  }
  __syncthreads();
  // W[i,j] = -W[i,i] · Acc
  for (int e = threadIdx.x; e < NB * NB; e += blockDim.x) {
    int r = e % NB, c = e / NB;
    Wt[c][r] = (r < h && c < h) ? W.a[(size_t)(r0 + c) * W.ld + r0 + r] : T(0);  // W[i,i]
  }
  __syncthreads();
  for (int e = threadIdx.x; e < h * NB; e += blockDim.x) {
    int r = e % h, c = e / h;
    T s = T(0);
    for (int q = 0; q < h; ++q) s += Wt[q][r] * Acc[c][q];
    W.a[(size_t)(j * NB + c) * W.ld + r0 + r] = -s;
  }
}

template <class T, int NB>
void trinv_batched(const MatDesc<T>* d_L, const MatDesc<T>* d_W, int nmat, int nmax,
                   cudaStream_t st) {
  if (nmat == 0 || nmax == 0) return;
  const int nt = ceil_div(nmax, NB);
  k_trinv_diag<T, NB><<<dim3(nt, nmat), 128, 0, st>>>(d_L, d_W);
  for (int i = 1; i < nt; ++i) k_trinv_row<T, NB><<<dim3(i, nmat), 256, 0, st>>>(d_L, d_W, i);
  SDPX_LAUNCH_CHECK_N(nt);
}
template void trinv_batched<double, 32>(const MatDesc<double>*, const MatDesc<double>*, int, int,
                                        cudaStream_t);

// Forward step s of L y = r:  y_s = Dinv_s r_s ;  r[rows below] -= L[rows, s] y_s.
// CTA 0 writes y_s; CTAs ≥ 1 each update ROWS rows below block s.  r and y are
// distinct buffers so no CTA reads a value written in the same launch.
template <class T, int NB, int ROWS>
__global__ void k_trsv_fwd_step(const T* L, long long ld, int n, const T* Dinv, int s, T* r, T* y) {
  __shared__ T ys[NB];
  const int s0 = s * NB, w = min(NB, n - s0);
  const T* Di = Dinv + (size_t)s * NB * NB;
  for (int t = threadIdx.x; t < NB; t += blockDim.x) {
    T acc = T(0);
    if (t < w)
      for (int p = 0; p < w; ++p) acc += Di[t + p * NB] * r[s0 + p];
    ys[t] = acc;
  }
  __syncthreads();
  if (blockIdx.x == 0) {
    for (int t = threadIdx.x; t < w; t += blockDim.x) y[s0 + t] = ys[t];
    return;
  }
  const int base = s0 + w + (blockIdx.x - 1) * ROWS;
  for (int row = base + threadIdx.x; row < min(n, base + ROWS); row += blockDim.x) {
    T acc = T(0);
    for (int p = 0; p < w; ++p) acc += L[(size_t)(s0 + p) * ld + row] * ys[p];
    r[row] -= acc;
  }
}

// Backward step s of Lᵀ x = y: x_s = Dinv_sᵀ y_s ; y[rows above] -= L[s-block, rows]ᵀ x_s.
template <class T, int NB, int ROWS>
__global__ void k_trsv_bwd_step(const T* L, long long ld, int n, const T* Dinv, int s, T* yv, T* x) {
  __shared__ T xs[NB];
  const int s0 = s * NB, w = min(NB, n - s0);
  const T* Di = Dinv + (size_t)s * NB * NB;
  for (int t = threadIdx.x; t < NB; t += blockDim.x) {
    T acc = T(0);
    if (t < w)
      for (int p = 0; p < w; ++p) acc += Di[p + t * NB] * yv[s0 + p];
    xs[t] = acc;
  }
  __syncthreads();
  if (blockIdx.x == 0) {
    for (int t = threadIdx.x; t < w; t += blockDim.x) x[s0 + t] = xs[t];
    return;
  }
  const int base = (blockIdx.x - 1) * ROWS;
  const int end = min(s0, base + ROWS);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int row = base + warp; row < end; row += nw) {
    T acc = T(0);
    for (int p = lane; p < w; p += 32) acc += L[(size_t)row * ld + s0 + p] * xs[p];
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) yv[row] -= acc;
  }
}

template <class T, int NB>
void cholesky_solve(const T* L, long long ld, int n, const T* Dinv, T* rhs, T* work,
                    cudaStream_t st) {
  // rhs ← (L Lᵀ)^{-1} rhs.  `work` (n) receives the intermediate y.
  constexpr int ROWS = 256;
  const int nt = ceil_div(n, NB);
  for (int s = 0; s < nt; ++s) {
    int below = n - std::min(n, (s + 1) * NB);
    int grid = 1 + ceil_div(below, ROWS);
    k_trsv_fwd_step<T, NB, ROWS><<<grid, 256, 0, st>>>(L, ld, n, Dinv, s, rhs, work);
  }
  for (int s = nt - 1; s >= 0; --s) {
    int above = s * NB;
    int grid = 1 + ceil_div(above, ROWS);
    k_trsv_bwd_step<T, NB, ROWS><<<grid, 256, 0, st>>>(L, ld, n, Dinv, s, work, rhs);
  }
  SDPX_LAUNCH_CHECK_N(2 * nt);
}

// ---------------------------------------------------------------------------
// Explicit inverse of a lower-triangular factor by recursive doubling:
//   inv([A 0; B C]) = [A⁻¹ 0; −C⁻¹ B A⁻¹  C⁻¹],
// leaves are the 64×64 diagonal tiles (inverted in shared memory); every
// combination is two DMMA GEMMs with triangular K ranges.
// ---------------------------------------------------------------------------
void trinv_recursive_f64(const double* L, int n, double* Linv, double* Dinv, double* tmp,
                         cudaStream_t st) {
  SDPX_CUDA(cudaMemsetAsync(Linv, 0, sizeof(double) * (size_t)n * n, st));
  factor_diag_inverses(L, n, n, Dinv, Linv, st);
  const int nt = ceil_div(n, 64);
  auto sub = [&](const double* base, int r0, int c0, int rows, int cols, bool kcontig) {
    Opnd o;
    o.base = base + r0 + (size_t)c0 * n;
    o.inner = 1 << 30;
    o.outer_stride = 0;
    if (kcontig) {  // operand as B: (kk = row, nn = col)
      o.kstride = 1;
      o.inner_stride = n;
      o.mn_extent = cols;
      o.k_extent = rows;
    } else {  // operand as A: (mm = row, kk = col)
      o.kstride = n;
      o.inner_stride = 1;
      o.mn_extent = rows;
      o.k_extent = cols;
    }
    return o;
  };
  auto out = [&](double* base, int r0, int c0, int rows, int cols) {
    OutDesc d;
    d.base = base + r0 + (size_t)c0 * n;
    d.row_inner_stride = 1;
    d.row_outer_stride = 0;
    d.row_inner = 1 << 30;
    d.col_inner_stride = n;
    d.col_outer_stride = 0;
    d.col_inner = 1 << 30;
    d.rows = rows;
    d.cols = cols;
    return d;
  };
  // The pairs of one doubling level are independent: their first products
  // go out as grouped launches, then their second products.
  for (int g = 1; g < nt; g *= 2) {
    GemmGroups first, second;
    auto flush = [&]() {
      gemm_f64_grouped(first, false, true, st);
      gemm_f64_grouped(second, false, true, st);
      first.n = second.n = 0;
    };
    for (int i0 = 0; i0 < nt; i0 += 2 * g) {
      const int a0 = i0 * 64, a1 = std::min(n, (i0 + g) * 64);
      const int c0 = a1, c1 = std::min(n, (i0 + 2 * g) * 64);
      if (c0 >= n) continue;
      const int ra = a1 - a0, rc = c1 - c0;
      if (first.n == kGemmGroups) flush();
      // T = B · A⁻¹   (B = L[c0:c1, a0:a1], A⁻¹ lower: k ≥ col)
      const int q = first.n++;
      first.A[q] = sub(L, c0, a0, rc, ra, false);
      first.B[q] = sub(Linv, a0, a0, ra, ra, true);
      first.C[q] = out(tmp, c0, a0, rc, ra);
      first.alpha[q] = 1.0;
      first.beta[q] = 0.0;
      first.mode[q] = KR_B_LOWER;
      // Linv[c0:c1, a0:a1] = −C⁻¹ · T   (C⁻¹ lower: k ≤ row)
      second.n++;
      second.A[q] = sub(Linv, c0, c0, rc, rc, false);
      second.B[q] = sub(tmp, c0, a0, rc, ra, true);
      second.C[q] = out(Linv, c0, a0, rc, ra);
      second.alpha[q] = -1.0;
      second.beta[q] = 0.0;
      second.mode[q] = KR_A_LOWER;
    }
    flush();
  }
}
template void cholesky_solve<double, 64>(const double*, long long, int, const double*, double*,
                                         double*, cudaStream_t);

}  // namespace sdpx
