// Triangular inverses and solves with a lower Cholesky factor (the factorization
// itself: potrf_flow.cu).
#include "chol.h"
#include "blas_f64.h"

namespace sdpx {

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
// Explicit inverses of lower-triangular factors by recursive doubling:
//   inv([A 0; B C]) = [A⁻¹ 0; −C⁻¹ B A⁻¹  C⁻¹],
// leaves are the 64×64 diagonal tiles (inverted in shared memory); every
// combination is two DMMA GEMMs with triangular K ranges.  The pairs of one
// doubling level, of all matrices, are independent: their first products go out as
// grouped launches, then their second products.
// ---------------------------------------------------------------------------
void trinv(const TrinvList& list, cudaStream_t st) {
  invert_diag_tiles(list, st);
  int nmax = 0;
  for (int b = 0; b < list.count; ++b) nmax = std::max(nmax, list.n[b]);
  const int nt = ceil_div(nmax, 64);
  for (int g = 1; g < nt; g *= 2) {
    GemmGroups first, second;
    auto flush = [&]() {
      gemm_f64_grouped(first, false, true, st);
      gemm_f64_grouped(second, false, true, st);
      first.n = second.n = 0;
    };
    for (int b = 0; b < list.count; ++b) {
      const int n = list.n[b];
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
      const double* L = list.L[b];
      double *W = list.W[b], *tmp = list.tmp[b];
      for (int a0 = 0; a0 + 64 * g < n; a0 += 128 * g) {
        const int c0 = a0 + 64 * g, c1 = std::min(n, c0 + 64 * g);
        const int ra = c0 - a0, rc = c1 - c0;
        if (first.n == kGemmGroups) flush();
        // T = B · A⁻¹   (B = L[c0:c1, a0:c0], A⁻¹ lower: k ≥ col)
        const int q = first.n++;
        first.A[q] = sub(L, c0, a0, rc, ra, false);
        first.B[q] = sub(W, a0, a0, ra, ra, true);
        first.C[q] = out(tmp, c0, a0, rc, ra);
        first.alpha[q] = 1.0;
        first.beta[q] = 0.0;
        first.mode[q] = KR_B_LOWER;
        // W[c0:c1, a0:c0] = −C⁻¹ · T   (C⁻¹ lower: k ≤ row)
        second.n++;
        second.A[q] = sub(W, c0, c0, rc, rc, false);
        second.B[q] = sub(tmp, c0, a0, rc, ra, true);
        second.C[q] = out(W, c0, a0, rc, ra);
        second.alpha[q] = -1.0;
        second.beta[q] = 0.0;
        second.mode[q] = KR_A_LOWER;
      }
    }
    flush();
  }
}
template void cholesky_solve<double, 64>(const double*, long long, int, const double*, double*,
                                         double*, cudaStream_t);

}  // namespace sdpx
