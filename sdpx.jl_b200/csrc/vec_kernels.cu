// Memory-bound kernels over the stacked constraint matrix 𝒜 (K×m, column i =
// vec(A_i) of every block, 1×1 blocks gathered at the end) and over stacked
// block vectors (length K, same row offsets as 𝒜).
#include "dd.cuh"
#include "vec_kernels.h"

#include <type_traits>

namespace sdpx {

// ---------------------------------------------------------------- gemv ----
// out[row] = Σ_i A[row + i·K]·x[i], column range split into `chunks` partial
// sums (written to part[chunk·K + row]) then reduced in fixed order.
__global__ void k_gemv_n_part(const double* __restrict__ A, long long K, int m,
                              const double* __restrict__ x, int chunks, double* __restrict__ part) {
  long long row = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  int ch = blockIdx.y;
  if (row >= K) return;
  int per = (m + chunks - 1) / chunks;
  int i0 = ch * per, i1 = min(m, i0 + per);
  const double* p = A + row;
  double s0 = 0, s1 = 0, s2 = 0, s3 = 0;
  int i = i0;
  for (; i + 3 < i1; i += 4) {
    s0 += p[(long long)i * K] * x[i];
    s1 += p[(long long)(i + 1) * K] * x[i + 1];
    s2 += p[(long long)(i + 2) * K] * x[i + 2];
    s3 += p[(long long)(i + 3) * K] * x[i + 3];
  }
  for (; i < i1; ++i) s0 += p[(long long)i * K] * x[i];
  part[(long long)ch * K + row] = (s0 + s1) + (s2 + s3);
}

__global__ void k_gemv_n_reduce(const double* __restrict__ part, long long K, int chunks,
                                double* __restrict__ out) {
  long long row = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (row >= K) return;
  double s = 0;
  for (int c = 0; c < chunks; ++c) s += part[(long long)c * K + row];
  out[row] = s;
}

// The same partial sums with 128-bit loads: each thread owns the row pair
// (2q, 2q+1) and reads one double2 per column (K even and A 16-byte aligned,
// so every column starts on a 16-byte boundary).  Each row accumulates its
// columns in exactly the order of k_gemv_n_part, so the results are identical.
__global__ void k_gemv_n_part2(const double* __restrict__ A, long long K, int m,
                               const double* __restrict__ x, int chunks, double* __restrict__ part) {
  const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long K2 = K >> 1;
  if (q >= K2) return;
  const int ch = blockIdx.y;
  const int per = (m + chunks - 1) / chunks;
  const int i0 = ch * per, i1 = min(m, i0 + per);
  const double2* p = reinterpret_cast<const double2*>(A) + q;
  double2 s0 = {0, 0}, s1 = {0, 0}, s2 = {0, 0}, s3 = {0, 0};
  int i = i0;
  for (; i + 3 < i1; i += 4) {
    const double2 a0 = __ldg(p + (long long)i * K2), a1 = __ldg(p + (long long)(i + 1) * K2);
    const double2 a2 = __ldg(p + (long long)(i + 2) * K2), a3 = __ldg(p + (long long)(i + 3) * K2);
    const double x0 = x[i], x1 = x[i + 1], x2 = x[i + 2], x3 = x[i + 3];
    s0.x += a0.x * x0; s0.y += a0.y * x0;
    s1.x += a1.x * x1; s1.y += a1.y * x1;
    s2.x += a2.x * x2; s2.y += a2.y * x2;
    s3.x += a3.x * x3; s3.y += a3.y * x3;
  }
  for (; i < i1; ++i) {
    const double2 a = __ldg(p + (long long)i * K2);
    s0.x += a.x * x[i];
    s0.y += a.y * x[i];
  }
  double2 r;
  r.x = (s0.x + s1.x) + (s2.x + s3.x);
  r.y = (s0.y + s1.y) + (s2.y + s3.y);
  reinterpret_cast<double2*>(part + (long long)ch * K)[q] = r;
}

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// Partial sums of 𝒜·x over `chunks` column ranges: the 128-bit variant when
// the stride allows it, else one row per thread.
static void gemv_n_partials(const double* A, long long K, int m, const double* x, int chunks,
                            double* part, cudaStream_t st) {
  if ((K & 1) == 0 && aligned16(A) && aligned16(part)) {
    dim3 g(ceil_div(K / 2, 256), chunks);
    k_gemv_n_part2<<<g, 256, 0, st>>>(A, K, m, x, chunks, part);
  } else {
    dim3 g(ceil_div(K, 256), chunks);
    k_gemv_n_part<<<g, 256, 0, st>>>(A, K, m, x, chunks, part);
  }
}

void gemv_n(const double* A, long long K, int m, const double* x, double* out, double* part,
            int chunks, cudaStream_t st) {
  if (K == 0) return;
  gemv_n_partials(A, K, m, x, chunks, part, st);
  k_gemv_n_reduce<<<ceil_div(K, 256), 256, 0, st>>>(part, K, chunks, out);
  SDPX_LAUNCH_CHECK_N(2);
}

// ------------------------------------------- lower-triangle constraints ---
// Ap[q + i·Kt] = A[rows[q] + i·K]: the rows kept by the packed copy.
__global__ void k_pack_rows(const double* __restrict__ A, long long K, int m,
                            const long long* __restrict__ rows, long long Kt,
                            double* __restrict__ Ap) {
  const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (q >= Kt) return;
  const long long src = rows[q];
  for (int i = blockIdx.y; i < m; i += gridDim.y) Ap[q + (long long)i * Kt] = A[src + (long long)i * K];
}
void pack_rows(const double* A, long long K, int m, const long long* rows, long long Kt, double* Ap,
               cudaStream_t st) {
  if (Kt == 0 || m == 0) return;
  dim3 g(ceil_div(Kt, 256), std::min(m, 64));
  k_pack_rows<<<g, 256, 0, st>>>(A, K, m, rows, Kt, Ap);
  SDPX_LAUNCH_CHECK();
}

// Row sums of the column-chunk partials, written to both stacked positions.
__global__ void k_gemv_n_reduce_sym(const double* __restrict__ part, long long Kt, int chunks,
                                    const long long* __restrict__ lo,
                                    const long long* __restrict__ up, double* __restrict__ out) {
  const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (q >= Kt) return;
  double s = 0;
  for (int c = 0; c < chunks; ++c) s += part[(long long)c * Kt + q];
  out[lo[q]] = s;
  out[up[q]] = s;
}
void gemv_n_sym(const double* Ap, long long Kt, int m, const double* x, const long long* lo,
                const long long* up, double* out, double* part, int chunks, cudaStream_t st) {
  if (Kt == 0) return;
  gemv_n_partials(Ap, Kt, m, x, chunks, part, st);
  k_gemv_n_reduce_sym<<<ceil_div(Kt, 256), 256, 0, st>>>(part, Kt, chunks, lo, up, out);
  SDPX_LAUNCH_CHECK_N(2);
}

// zf[q] = z[lo] + z[up] off the diagonal, z[lo] on it: ⟨A_i, Z⟩ over the
// lower triangle of a symmetric A_i.
__global__ void k_fold_sym(long long Kt, const double* __restrict__ z,
                           const long long* __restrict__ lo, const long long* __restrict__ up,
                           double* __restrict__ zf) {
  const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (q >= Kt) return;
  const long long a = lo[q], b = up[q];
  zf[q] = a == b ? z[a] : z[a] + z[b];
}
void fold_sym(long long Kt, const double* z, const long long* lo, const long long* up, double* zf,
              cudaStream_t st) {
  if (Kt == 0) return;
  k_fold_sym<<<ceil_div(Kt, 256), 256, 0, st>>>(Kt, z, lo, up, zf);
  SDPX_LAUNCH_CHECK();
}

// out[i] = alpha·(A[:,i] · z) + beta·base[i]   (one CTA per column).
__global__ void k_gemv_t(const double* __restrict__ A, long long K, int m,
                         const double* __restrict__ z, double alpha, const double* __restrict__ base,
                         double beta, double* __restrict__ out) {
  __shared__ double red[32];
  int i = blockIdx.x;
  const double* col = A + (long long)i * K;
  double s0 = 0, s1 = 0;
  long long r = threadIdx.x;
  for (; r + blockDim.x < K; r += 2 * blockDim.x) {
    s0 += col[r] * z[r];
    s1 += col[r + blockDim.x] * z[r + blockDim.x];
  }
  if (r < K) s0 += col[r] * z[r];
  double s = block_sum(s0 + s1, red);
  if (threadIdx.x == 0) out[i] = alpha * s + (base ? beta * base[i] : 0.0);
}

// 128-bit variant (K even, A and z 16-byte aligned): thread t reads the
// double2 pairs t, t + 512, …, two accumulators per lane of the pair.
__global__ void k_gemv_t2(const double* __restrict__ A, long long K, int m,
                          const double* __restrict__ z, double alpha,
                          const double* __restrict__ base, double beta, double* __restrict__ out) {
  __shared__ double red[32];
  const int i = blockIdx.x;
  const long long K2 = K >> 1;
  const double2* col = reinterpret_cast<const double2*>(A + (long long)i * K);
  const double2* z2 = reinterpret_cast<const double2*>(z);
  double s0 = 0, s1 = 0, s2 = 0, s3 = 0;
  long long r = threadIdx.x;
  for (; r + blockDim.x < K2; r += 2 * blockDim.x) {
    const double2 a = __ldg(col + r), b = __ldg(col + r + blockDim.x);
    const double2 u = __ldg(z2 + r), v = __ldg(z2 + r + blockDim.x);
    s0 += a.x * u.x;
    s1 += a.y * u.y;
    s2 += b.x * v.x;
    s3 += b.y * v.y;
  }
  if (r < K2) {
    const double2 a = __ldg(col + r), u = __ldg(z2 + r);
    s0 += a.x * u.x;
    s1 += a.y * u.y;
  }
  const double s = block_sum((s0 + s1) + (s2 + s3), red);
  if (threadIdx.x == 0) out[i] = alpha * s + (base ? beta * base[i] : 0.0);
}

void gemv_t(const double* A, long long K, int m, const double* z, double alpha, const double* base,
            double beta, double* out, cudaStream_t st) {
  if (m == 0) return;
  if ((K & 1) == 0 && aligned16(A) && aligned16(z))
    k_gemv_t2<<<m, 512, 0, st>>>(A, K, m, z, alpha, base, beta, out);
  else
    k_gemv_t<<<m, 512, 0, st>>>(A, K, m, z, alpha, base, beta, out);
  SDPX_LAUNCH_CHECK();
}

// ------------------------------------------------ compensated residuals ---
// Dot2 of Ogita, Rump and Oishi ("Accurate sum and dot product", SIAM J. Sci.
// Comput. 26(6), 2005): every term enters as its exact product p + e (FMA),
// the running sum is advanced by TwoSum and the rounding errors (TwoSum's and
// the products') collect in a second accumulator; partial accumulators merge
// by TwoSum the same way, and the result s + c is rounded once.  The value is
// as accurate as if computed in twice the working precision, so it does not
// depend on the order of the terms.
struct Dot2 {
  double s, c;
};
__device__ __forceinline__ void dot2_fma(Dot2& a, double x, double y) {
  const ddv p = dd_two_prod(x, y);
  const ddv t = dd_two_sum(a.s, p.hi);
  a.s = t.hi;
  a.c += t.lo + p.lo;
}
__device__ __forceinline__ void dot2_add(Dot2& a, double v) {
  const ddv t = dd_two_sum(a.s, v);
  a.s = t.hi;
  a.c += t.lo;
}
__device__ __forceinline__ void dot2_merge(Dot2& a, const Dot2& b) {
  const ddv t = dd_two_sum(a.s, b.s);
  a.s = t.hi;
  a.c += t.lo + b.c;
}

// Partials of 𝒜·x over `chunks` column ranges as Dot2 pairs: sums at
// part[ch·K + row], error terms at part[(chunks + ch)·K + row]; 128-bit loads
// of the row pair (2q, 2q+1) when K is even and A 16-byte aligned.
__global__ void k_gemv_n_part2_acc(const double* __restrict__ A, long long K, int m,
                                   const double* __restrict__ x, int chunks,
                                   double* __restrict__ part) {
  const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long K2 = K >> 1;
  if (q >= K2) return;
  const int ch = blockIdx.y;
  const int per = (m + chunks - 1) / chunks;
  const int i0 = ch * per, i1 = min(m, i0 + per);
  const double2* p = reinterpret_cast<const double2*>(A) + q;
  Dot2 a0{0, 0}, a1{0, 0}, b0{0, 0}, b1{0, 0};
  int i = i0;
  for (; i + 1 < i1; i += 2) {
    const double2 u = __ldg(p + (long long)i * K2), v = __ldg(p + (long long)(i + 1) * K2);
    const double x0 = x[i], x1 = x[i + 1];
    dot2_fma(a0, u.x, x0);
    dot2_fma(b0, u.y, x0);
    dot2_fma(a1, v.x, x1);
    dot2_fma(b1, v.y, x1);
  }
  if (i < i1) {
    const double2 u = __ldg(p + (long long)i * K2);
    dot2_fma(a0, u.x, x[i]);
    dot2_fma(b0, u.y, x[i]);
  }
  dot2_merge(a0, a1);
  dot2_merge(b0, b1);
  reinterpret_cast<double2*>(part + (long long)ch * K)[q] = make_double2(a0.s, b0.s);
  reinterpret_cast<double2*>(part + (long long)(chunks + ch) * K)[q] = make_double2(a0.c, b0.c);
}
__global__ void k_gemv_n_part_acc(const double* __restrict__ A, long long K, int m,
                                  const double* __restrict__ x, int chunks,
                                  double* __restrict__ part) {
  const long long row = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (row >= K) return;
  const int ch = blockIdx.y;
  const int per = (m + chunks - 1) / chunks;
  const int i0 = ch * per, i1 = min(m, i0 + per);
  Dot2 a0{0, 0}, a1{0, 0};
  int i = i0;
  for (; i + 1 < i1; i += 2) {
    dot2_fma(a0, A[row + (long long)i * K], x[i]);
    dot2_fma(a1, A[row + (long long)(i + 1) * K], x[i + 1]);
  }
  if (i < i1) dot2_fma(a0, A[row + (long long)i * K], x[i]);
  dot2_merge(a0, a1);
  part[(long long)ch * K + row] = a0.s;
  part[(long long)(chunks + ch) * K + row] = a0.c;
}

// out[r] = Σ_chunks partials − X[r] − C[r] (X, C may be null), rounded once;
// with lo/up (packed rows) the row's value goes to both stacked positions.
__global__ void k_gemv_n_reduce_acc(const double* __restrict__ part, long long K, int chunks,
                                    const double* __restrict__ X, const double* __restrict__ C,
                                    const long long* __restrict__ lo,
                                    const long long* __restrict__ up, double* __restrict__ out) {
  const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (q >= K) return;
  Dot2 a{0, 0};
  for (int c = 0; c < chunks; ++c)
    dot2_merge(a, Dot2{part[(long long)c * K + q], part[(long long)(chunks + c) * K + q]});
  const long long r0 = lo ? lo[q] : q, r1 = up ? up[q] : q;
  Dot2 b = a;
  if (X) dot2_add(a, -X[r0]);
  if (C) dot2_add(a, -C[r0]);
  out[r0] = a.s + a.c;
  if (r1 != r0) {
    if (X) dot2_add(b, -X[r1]);
    if (C) dot2_add(b, -C[r1]);
    out[r1] = b.s + b.c;
  }
}

static void gemv_n_partials_acc(const double* A, long long K, int m, const double* x, int chunks,
                                double* part, cudaStream_t st) {
  if ((K & 1) == 0 && aligned16(A) && aligned16(part)) {
    dim3 g(ceil_div(K / 2, 256), chunks);
    k_gemv_n_part2_acc<<<g, 256, 0, st>>>(A, K, m, x, chunks, part);
  } else {
    dim3 g(ceil_div(K, 256), chunks);
    k_gemv_n_part_acc<<<g, 256, 0, st>>>(A, K, m, x, chunks, part);
  }
}

void gemv_n_acc(const double* A, long long K, int m, const double* x, const double* X,
                const double* C, double* out, double* part, int chunks, cudaStream_t st) {
  if (K == 0) return;
  gemv_n_partials_acc(A, K, m, x, chunks, part, st);
  k_gemv_n_reduce_acc<<<ceil_div(K, 256), 256, 0, st>>>(part, K, chunks, X, C, nullptr, nullptr,
                                                         out);
  SDPX_LAUNCH_CHECK_N(2);
}

void gemv_n_sym_acc(const double* Ap, long long Kt, int m, const double* x, const long long* lo,
                    const long long* up, const double* X, const double* C, double* out,
                    double* part, int chunks, cudaStream_t st) {
  if (Kt == 0) return;
  gemv_n_partials_acc(Ap, Kt, m, x, chunks, part, st);
  k_gemv_n_reduce_acc<<<ceil_div(Kt, 256), 256, 0, st>>>(part, Kt, chunks, X, C, lo, up, out);
  SDPX_LAUNCH_CHECK_N(2);
}

// Block-wide merge of the Dot2 pairs (every thread receives the total).
__device__ __forceinline__ Dot2 block_dot2(Dot2 a, double* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const Dot2 b{__shfl_xor_sync(0xffffffffu, a.s, o), __shfl_xor_sync(0xffffffffu, a.c, o)};
    dot2_merge(a, b);
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  __syncthreads();
  if (lane == 0) {
    red[w] = a.s;
    red[32 + w] = a.c;
  }
  __syncthreads();
  if (w == 0) {
    a = lane < nw ? Dot2{red[lane], red[32 + lane]} : Dot2{0, 0};
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const Dot2 b{__shfl_xor_sync(0xffffffffu, a.s, o), __shfl_xor_sync(0xffffffffu, a.c, o)};
      dot2_merge(a, b);
    }
  }
  return a;  // valid in thread 0
}

// out[i] = alpha·(A[:,i]·z) + beta·base[i] from one double-double value,
// rounded once (one CTA per column; 128-bit loads when K is even and A, z
// are 16-byte aligned).
template <bool VEC>
__global__ void k_gemv_t_acc(const double* __restrict__ A, long long K, int m,
                             const double* __restrict__ z, double alpha,
                             const double* __restrict__ base, double beta,
                             double* __restrict__ out) {
  __shared__ double red[64];
  const int i = blockIdx.x;
  Dot2 a0{0, 0}, a1{0, 0};
  if (VEC) {
    const long long K2 = K >> 1;
    const double2* col = reinterpret_cast<const double2*>(A + (long long)i * K);
    const double2* z2 = reinterpret_cast<const double2*>(z);
    for (long long r = threadIdx.x; r < K2; r += blockDim.x) {
      const double2 u = __ldg(col + r), v = __ldg(z2 + r);
      dot2_fma(a0, u.x, v.x);
      dot2_fma(a1, u.y, v.y);
    }
  } else {
    const double* col = A + (long long)i * K;
    for (long long r = threadIdx.x; r < K; r += blockDim.x) dot2_fma(a0, col[r], z[r]);
  }
  dot2_merge(a0, a1);
  const Dot2 t = block_dot2(a0, red);
  if (threadIdx.x == 0) {
    ddv v = dd_mul_d(dd_two_sum(t.s, t.c), alpha);
    if (base) v = dd_add(v, dd_two_prod(beta, base[i]));
    out[i] = v.hi + v.lo;
  }
}

void gemv_t_acc(const double* A, long long K, int m, const double* z, double alpha,
                const double* base, double beta, double* out, cudaStream_t st) {
  if (m == 0) return;
  if ((K & 1) == 0 && aligned16(A) && aligned16(z))
    k_gemv_t_acc<true><<<m, 512, 0, st>>>(A, K, m, z, alpha, base, beta, out);
  else
    k_gemv_t_acc<false><<<m, 512, 0, st>>>(A, K, m, z, alpha, base, beta, out);
  SDPX_LAUNCH_CHECK();
}

// ------------------------------------------------------- elementwise -------
__global__ void k_axpbypcz(long long n, double a, const double* x, double b, const double* y,
                           double c, const double* z, double* out) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n;
       e += (long long)gridDim.x * blockDim.x) {
    double v = a * x[e];
    if (y) v += b * y[e];
    if (z) v += c * z[e];
    out[e] = v;
  }
}
// 128-bit variant over element pairs (every operand 16-byte aligned); the odd
// last element, if any, is done by thread 0 of block 0.  Same arithmetic per
// element as k_axpbypcz.
__global__ void k_axpbypcz2(long long n, double a, const double* x, double b, const double* y,
                            double c, const double* z, double* out) {
  const long long n2 = n >> 1;
  const double2* x2 = reinterpret_cast<const double2*>(x);
  const double2* y2 = reinterpret_cast<const double2*>(y);
  const double2* z2 = reinterpret_cast<const double2*>(z);
  double2* o2 = reinterpret_cast<double2*>(out);
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n2;
       e += (long long)gridDim.x * blockDim.x) {
    const double2 xv = x2[e];
    double2 v = {a * xv.x, a * xv.y};
    if (y) {
      const double2 yv = y2[e];
      v.x += b * yv.x;
      v.y += b * yv.y;
    }
    if (z) {
      const double2 zv = z2[e];
      v.x += c * zv.x;
      v.y += c * zv.y;
    }
    o2[e] = v;
  }
  if ((n & 1) && blockIdx.x == 0 && threadIdx.x == 0) {
    const long long e = n - 1;
    double v = a * x[e];
    if (y) v += b * y[e];
    if (z) v += c * z[e];
    out[e] = v;
  }
}
void axpbypcz(long long n, double a, const double* x, double b, const double* y, double c,
              const double* z, double* out, cudaStream_t st) {
  if (n == 0) return;
  if (aligned16(x) && aligned16(out) && (!y || aligned16(y)) && (!z || aligned16(z))) {
    const int g = std::min(4096, (int)std::max<long long>(1, ceil_div(n / 2, 256)));
    k_axpbypcz2<<<g, 256, 0, st>>>(n, a, x, b, y, c, z, out);
  } else {
    const int g = std::min(4096, ceil_div(n, 256));
    k_axpbypcz<<<g, 256, 0, st>>>(n, a, x, b, y, c, z, out);
  }
  SDPX_LAUNCH_CHECK();
}

// x ← x + t·d   (the reference's trial_combine!: dest[i] = X[i] + t*dX[i])
__global__ void k_combine(long long n, double* x, double t, const double* d) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n;
       e += (long long)gridDim.x * blockDim.x)
    x[e] = x[e] + t * d[e];
}
__global__ void k_combine2(long long n, double* x, double t, const double* d) {
  const long long n2 = n >> 1;
  double2* x2 = reinterpret_cast<double2*>(x);
  const double2* d2 = reinterpret_cast<const double2*>(d);
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n2;
       e += (long long)gridDim.x * blockDim.x) {
    double2 xv = x2[e];
    const double2 dv = d2[e];
    xv.x = xv.x + t * dv.x;
    xv.y = xv.y + t * dv.y;
    x2[e] = xv;
  }
  if ((n & 1) && blockIdx.x == 0 && threadIdx.x == 0) x[n - 1] = x[n - 1] + t * d[n - 1];
}
void combine(long long n, double* x, double t, const double* d, cudaStream_t st) {
  if (n == 0) return;
  if (aligned16(x) && aligned16(d))
    k_combine2<<<std::min(4096, (int)std::max<long long>(1, ceil_div(n / 2, 256))), 256, 0, st>>>(
        n, x, t, d);
  else
    k_combine<<<std::min(4096, ceil_div(n, 256)), 256, 0, st>>>(n, x, t, d);
  SDPX_LAUNCH_CHECK();
}

__global__ void k_scale(long long n, double* x, double f) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n;
       e += (long long)gridDim.x * blockDim.x)
    x[e] *= f;
}
void scale(long long n, double* x, double f, cudaStream_t st) {
  if (n == 0) return;
  k_scale<<<std::min(4096, ceil_div(n, 256)), 256, 0, st>>>(n, x, f);
  SDPX_LAUNCH_CHECK();
}

__global__ void k_zero_list(const __grid_constant__ ZeroList q) {
  double* p = q.p[blockIdx.y];
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < q.len[blockIdx.y];
       e += (long long)gridDim.x * blockDim.x)
    p[e] = 0.0;
}
void zero_list(const ZeroList& q, cudaStream_t st) {
  long long most = 0;
  for (int i = 0; i < q.n; ++i) most = std::max(most, q.len[i]);
  if (most == 0) return;
  k_zero_list<<<dim3(std::min(256, ceil_div(most, 256)), q.n), 256, 0, st>>>(q);
  SDPX_LAUNCH_CHECK();
}

// ----------------------------------------------------------- reductions ----
// out[slot] = max(out[slot], max|x|) ; finiteness folded in (NaN → +inf).
__global__ void k_absmax(long long n, const double* x, double* out) {
  __shared__ double red[32];
  double v = 0.0;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n;
       e += (long long)gridDim.x * blockDim.x) {
    double a = fabs(x[e]);
    if (!(a == a)) a = 1.0 / 0.0;
    v = fmax(v, a);
  }
  v = block_max(v, red);
  if (threadIdx.x == 0) atomic_max_nonneg(out, v);
}
void absmax(long long n, const double* x, double* out, cudaStream_t st) {
  if (n == 0) return;
  k_absmax<<<std::min(1024, ceil_div(n, 256)), 256, 0, st>>>(n, x, out);
  SDPX_LAUNCH_CHECK();
}

// max|x_e| of several vectors, delivered by the last block to finish (atomic ticket): a
// launch in place of a clear, one launch per vector and a copy back, whose gaps and host
// calls took 15-25 µs for vectors that need under 2.
void NormList::add(long long len_, const double* x_, double* out_) {
  if (len_ == 0) {
    *out_ = 0.0;
    return;
  }
  len[n] = len_;
  x[n] = x_;
  out[n] = out_;
  first[n + 1] = first[n] + (int)std::min<long long>(512, ceil_div(len_, 1024));
  ++n;
}
__global__ void __launch_bounds__(256) k_absmax_list(const __grid_constant__ NormList q, NormWork* w) {
  __shared__ double red[32];
  __shared__ bool last;
  int e = 0;
  while ((int)blockIdx.x >= q.first[e + 1]) ++e;
  const double* x = q.x[e];
  const long long n = q.len[e], step = (long long)(q.first[e + 1] - q.first[e]) * blockDim.x;
  double v = 0.0;
  for (long long i = (long long)(blockIdx.x - q.first[e]) * blockDim.x + threadIdx.x; i < n; i += step) {
    double a = fabs(x[i]);
    if (!(a == a)) a = 1.0 / 0.0;
    v = fmax(v, a);
  }
  v = block_max(v, red);
  if (threadIdx.x == 0) {
    atomic_max_nonneg(&w->v[e], v);
    __threadfence();
    last = atomicAdd(&w->done, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  if (threadIdx.x < q.n) {
    __threadfence();
    *q.out[threadIdx.x] = __ldcg(&w->v[threadIdx.x]);
    w->v[threadIdx.x] = 0.0;
  }
  if (threadIdx.x == 0) w->done = 0;
}
void absmax_list(const NormList& q, NormWork* work, cudaStream_t st) {
  if (q.n == 0) return;
  k_absmax_list<<<q.first[q.n], 256, 0, st>>>(q, work);
  SDPX_LAUNCH_CHECK();
}

// Segmented dot products: out[s] = Σ (x + tx·dx)(y + ty·dy) over segment s (dx/dy may be
// null).  One CTA per chunk of at most kSegChunk rows; the last CTA to finish adds the
// chunks of a segment, a warp each, in an order of its own (the same every time).
__global__ void __launch_bounds__(256) k_seg_dot(const SegChunk* __restrict__ chunks,
                                                 const int* __restrict__ first, int nseg,
                                                 const double* __restrict__ x, const double* __restrict__ dx,
                                                 double tx, const double* __restrict__ y,
                                                 const double* __restrict__ dy, double ty, double* part,
                                                 unsigned* done, double* out) {
  __shared__ double red[32];
  __shared__ bool last;
  const SegChunk q = chunks[blockIdx.x];
  constexpr int PER = kSegChunk / 256;
  double acc = 0.0;
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    const long long i = q.start + threadIdx.x + u * 256;
    if (i >= q.end) break;
    double a = x[i];
    if (dx) a += tx * dx[i];
    double c = y[i];
    if (dy) c += ty * dy[i];
    acc += a * c;
  }
  acc = block_sum(acc, red);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = acc;
    __threadfence();
    last = atomicAdd(done, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int s = threadIdx.x; s < nseg; s += 256)
    if (first[s + 1] - first[s] == 1) out[s] = __ldcg(part + first[s]);
  for (int s = warp; s < nseg; s += 8) {
    const int b = first[s], e = first[s + 1];
    if (e - b == 1) continue;
    double t = 0.0;
    for (int i = b + lane; i < e; i += 32) t += __ldcg(part + i);
    t = warp_sum(t);
    if (lane == 0) out[s] = t;
  }
  if (threadIdx.x == 0) *done = 0;
}
void seg_dot(const SegChunk* d_chunks, int nchunk, const int* d_first, int nseg, const double* x,
             const double* dx, double tx, const double* y, const double* dy, double ty, double* part,
             unsigned* done, double* out, cudaStream_t st) {
  if (nseg == 0 || nchunk == 0) return;
  k_seg_dot<<<nchunk, 256, 0, st>>>(d_chunks, d_first, nseg, x, dx, tx, y, dy, ty, part, done, out);
  SDPX_LAUNCH_CHECK();
}

// Diagonal entries of every dense block plus the 1×1 entries: out[t] = trace.
__global__ void k_block_trace(const long long* off, const int* kk, int nseg, const double* M,
                              double* out) {
  __shared__ double red[32];
  int s = blockIdx.x;
  int k = kk[s];
  double acc = 0.0;
  for (int i = threadIdx.x; i < k; i += blockDim.x) acc += M[off[s] + i + (long long)i * k];
  acc = block_sum(acc, red);
  if (threadIdx.x == 0) out[s] = acc;
}
void block_trace(const long long* d_off, const int* d_k, int nseg, const double* M, double* out,
                 cudaStream_t st) {
  if (nseg == 0) return;
  k_block_trace<<<nseg, 128, 0, st>>>(d_off, d_k, nseg, M, out);
  SDPX_LAUNCH_CHECK();
}

// M_block += shift_s · I for each segment s (dense blocks) — shifts[s] per block.
__global__ void k_add_diag(const long long* off, const int* kk, int nseg, double* M,
                           const double* shifts, double uniform) {
  int s = blockIdx.y;
  if (s >= nseg) return;
  int k = kk[s];
  double sh = shifts ? shifts[s] : uniform;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < k; i += gridDim.x * blockDim.x)
    M[off[s] + i + (long long)i * k] += sh;
}
void add_diag(const long long* d_off, const int* d_k, int nseg, int kmax, double* M,
              const double* d_shifts, double uniform, cudaStream_t st) {
  if (nseg == 0 || kmax == 0) return;
  k_add_diag<<<dim3(ceil_div(kmax, 256), nseg), 256, 0, st>>>(d_off, d_k, nseg, M, d_shifts, uniform);
  SDPX_LAUNCH_CHECK();
}

struct Shifts {
  double v[kShiftInline];
};
__global__ void k_add_diag_inline(const long long* off, const int* kk, double* M,
                                  const __grid_constant__ Shifts sh) {
  const int s = blockIdx.y, k = kk[s];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < k; i += gridDim.x * blockDim.x)
    M[off[s] + i + (long long)i * k] += sh.v[s];
}
void add_diag_host(const long long* d_off, const int* d_k, int nseg, int kmax, double* M,
                   const double* shifts, double* d_tmp, cudaStream_t st) {
  if (nseg == 0 || kmax == 0) return;
  if (nseg > kShiftInline) {
    SDPX_CUDA(cudaMemcpyAsync(d_tmp, shifts, sizeof(double) * nseg, cudaMemcpyHostToDevice, st));
    add_diag(d_off, d_k, nseg, kmax, M, d_tmp, 0.0, st);
    return;
  }
  Shifts sh{};
  std::copy(shifts, shifts + nseg, sh.v);
  k_add_diag_inline<<<dim3(ceil_div(kmax, 256), nseg), 256, 0, st>>>(d_off, d_k, M, sh);
  SDPX_LAUNCH_CHECK();
}

// Symmetrize every dense block in place: M ← (M + Mᵀ)/2.
__global__ void k_symmetrize(const long long* off, const int* kk, int nseg, double* M) {
  int s = blockIdx.y;
  if (s >= nseg) return;
  int k = kk[s];
  long long tot = (long long)k * k;
  double* B = M + off[s];
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < tot;
       e += (long long)gridDim.x * blockDim.x) {
    int i = (int)(e % k), j = (int)(e / k);
    if (i < j) {
      double avg = (B[i + (long long)j * k] + B[j + (long long)i * k]) / 2;
      B[i + (long long)j * k] = avg;
      B[j + (long long)i * k] = avg;
    }
  }
}
void symmetrize(const long long* d_off, const int* d_k, int nseg, int kmax, double* M,
                cudaStream_t st) {
  if (nseg == 0) return;
  int g = std::max(1, std::min(512, ceil_div((long long)kmax * kmax, 256)));
  k_symmetrize<<<dim3(g, nseg), 256, 0, st>>>(d_off, d_k, nseg, M);
  SDPX_LAUNCH_CHECK();
}

// Gershgorin lower bound, finiteness and max |lower entry| per dense block
// (lower triangle authoritative, src/cold_start.jl:152-201).  One CTA per row;
// out_bound[row-major offset] collects per-row candidates, reduced on the host side.
__global__ void k_gershgorin_rows(const long long* off, const int* kk, int nseg, const double* M,
                                  double* cand, double* scale, int* nonfinite,
                                  const long long* cand_off) {
  __shared__ double red[32];
  int s = blockIdx.y, i = blockIdx.x;
  if (s >= nseg) return;
  int k = kk[s];
  if (i >= k) return;
  const double* B = M + off[s];
  double rad = 0.0, mx = 0.0;
  int bad = 0;
  for (int j = threadIdx.x; j < k; j += blockDim.x) {
    double v = (j <= i) ? B[i + (long long)j * k] : B[j + (long long)i * k];
    if (!isfinite(v)) bad = 1;
    if (j != i) rad += fabs(v);
    if (j <= i) mx = fmax(mx, fabs(v));
  }
  rad = block_sum(rad, red);
  double m2 = block_max(mx, red);
  int anybad = __syncthreads_or(bad);
  if (threadIdx.x == 0) {
    cand[cand_off[s] + i] = B[i + (long long)i * k] - rad;
    atomic_max_nonneg(scale + s, m2);
    if (anybad) nonfinite[s] = 1;
  }
}
void gershgorin(const long long* d_off, const int* d_k, int nseg, int kmax, const double* M,
                double* d_cand, const long long* d_cand_off, double* d_scale, int* d_nonfinite,
                cudaStream_t st) {
  if (nseg == 0) return;
  k_gershgorin_rows<<<dim3(kmax, nseg), 128, 0, st>>>(d_off, d_k, nseg, M, d_cand, d_scale,
                                                      d_nonfinite, d_cand_off);
  SDPX_LAUNCH_CHECK();
}

// ------------------------------------------------------ 1×1 block group ----
// Entries j = 0..nd-1 at stacked offset od.  mu_user / user index per entry.
__global__ void k_diag_residual_R(int nd, long long od, const double* X, const double* Y,
                                  const double* mu_user, const int* user, int use_affine, double* R) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= nd) return;
  long long e = od + j;
  double v = -(X[e] * Y[e]);
  if (!use_affine) v += mu_user[user[j]];
  R[e] = v;
}
void diag_residual_R(int nd, long long od, const double* X, const double* Y, const double* mu_user,
                     const int* user, int use_affine, double* R, cudaStream_t st) {
  if (nd == 0) return;
  k_diag_residual_R<<<ceil_div(nd, 256), 256, 0, st>>>(nd, od, X, Y, mu_user, user, use_affine, R);
  SDPX_LAUNCH_CHECK();
}

// LX = sqrt(X), MY = sqrt(Y); fail flag if a value is not positive.
__global__ void k_diag_factor(int nd, long long od, const double* X, const double* Y, double* LX,
                              double* MY, int* fail) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= nd) return;
  long long e = od + j;
  double x = X[e], y = Y[e];
  if (!(x > 0) || !(y > 0)) *fail = 1;  // (may be pinned host memory)
  LX[e] = sqrt(x);
  MY[e] = sqrt(y);
}
void diag_factor(int nd, long long od, const double* X, const double* Y, double* LX, double* MY,
                 int* fail, cudaStream_t st) {
  if (nd == 0) return;
  k_diag_factor<<<ceil_div(nd, 256), 256, 0, st>>>(nd, od, X, Y, LX, MY, fail);
  SDPX_LAUNCH_CHECK();
}

// Z = (P·Y − R) / l / l  with l = LX  (kcholsolve 1×1: M / l11 / l11)
__global__ void k_diag_rhs_Z(int nd, long long od, const double* P, const double* Y, const double* R,
                             const double* LX, double* Z) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= nd) return;
  long long e = od + j;
  double l = LX[e];
  Z[e] = (P[e] * Y[e] - R[e]) / l / l;
}
void diag_rhs_Z(int nd, long long od, const double* P, const double* Y, const double* R,
                const double* LX, double* Z, cudaStream_t st) {
  if (nd == 0) return;
  k_diag_rhs_Z<<<ceil_div(nd, 256), 256, 0, st>>>(nd, od, P, Y, R, LX, Z);
  SDPX_LAUNCH_CHECK();
}

// dY = (R − dX·Y) / l / l
__global__ void k_diag_dY(int nd, long long od, const double* R, const double* dX, const double* Y,
                          const double* LX, double* dY) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= nd) return;
  long long e = od + j;
  double l = LX[e];
  dY[e] = (R[e] - dX[e] * Y[e]) / l / l;
}
void diag_dY(int nd, long long od, const double* R, const double* dX, const double* Y,
             const double* LX, double* dY, cudaStream_t st) {
  if (nd == 0) return;
  k_diag_dY<<<ceil_div(nd, 256), 256, 0, st>>>(nd, od, R, dX, Y, LX, dY);
  SDPX_LAUNCH_CHECK();
}

// R = target − X·Y − dX·dY  (Mehrotra, 1×1) with per-entry target
__global__ void k_diag_corrector_R(int nd, long long od, const double* X, const double* Y,
                                   const double* dX, const double* dY, const double* target_user,
                                   const int* user, double* R) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= nd) return;
  long long e = od + j;
  double v = -(X[e] * Y[e]);
  v = v - dX[e] * dY[e];
  R[e] = v + target_user[user[j]];
}
void diag_corrector_R(int nd, long long od, const double* X, const double* Y, const double* dX,
                      const double* dY, const double* target_user, const int* user, double* R,
                      cudaStream_t st) {
  if (nd == 0) return;
  k_diag_corrector_R<<<ceil_div(nd, 256), 256, 0, st>>>(nd, od, X, Y, dX, dY, target_user, user, R);
  SDPX_LAUNCH_CHECK();
}

// Schur panel rows of the 1×1 group:  P̂[od+j, i] = (A[od+j, i] / LX_j) · MY_j
__global__ void k_diag_panel(long long K, int m, int nd, long long od, const double* A,
                             const double* LX, const double* MY, double* Pc) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  int i = blockIdx.y;
  if (j >= nd || i >= m) return;
  long long e = od + j;
  long long a = e + (long long)i * K;
  Pc[a] = (A[a] / LX[e]) * MY[e];
}
void diag_panel(long long K, int m, int nd, long long od, const double* A, const double* LX,
                const double* MY, double* Pc, cudaStream_t st) {
  if (nd == 0) return;
  k_diag_panel<<<dim3(ceil_div(nd, 256), m), 256, 0, st>>>(K, m, nd, od, A, LX, MY, Pc);
  SDPX_LAUNCH_CHECK();
}

// ----------------------------------------------------- line-search trials ---
// 1×1 group: for candidate steps t[c] (c < n), fail[c] = 1 unless X + t dX > 0 in every entry.
// margin > 0 additionally requires a finite square root (SDPX's 1×1
// `trial_has_cholesky_margin!`).
__global__ void k_diag_trial(int nd, long long od, const double* X, const double* dX,
                             const __grid_constant__ DiagSteps q, int margin, int* fail) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  int c = blockIdx.y;
  if (j >= nd) return;
  long long e = od + j;
  double v = X[e] + q.t[c] * dX[e];
  bool ok = v > 0;
  if (ok && margin) ok = isfinite(sqrt(v));
  if (!ok) fail[c] = 1;
}
void diag_trial(int nd, long long od, const double* X, const double* dX, const DiagSteps& q, int margin, int* fail,
                cudaStream_t st) {
  if (nd == 0 || q.n == 0) return;
  k_diag_trial<<<dim3(ceil_div(nd, 256), q.n), 256, 0, st>>>(nd, od, X, dX, q, margin, fail);
  SDPX_LAUNCH_CHECK();
}

// 1×1 fraction-to-boundary: min_j (d < 0 ? min(1, −X/d) : 1)  (src/kernels/generic.jl:355-357).
// Single CTA so the minimum is exact.
__global__ void k_diag_ftb(int nd, long long od, const double* X, const double* dX, double* out) {
  __shared__ double red[32];
  double v = 1.0;
  for (int j = threadIdx.x; j < nd; j += blockDim.x) {
    double d = dX[od + j];
    double b = (d < 0) ? fmin(1.0, -X[od + j] / d) : 1.0;
    v = fmin(v, b);
  }
  double m = -block_max(-v, red);
  if (threadIdx.x == 0) *out = m;
}
void diag_ftb(int nd, long long od, const double* X, const double* dX, double* d_out,
              cudaStream_t st) {
  if (nd == 0) return;
  k_diag_ftb<<<1, 1024, 0, st>>>(nd, od, X, dX, d_out);
  SDPX_LAUNCH_CHECK();
}

// Trial matrices from a descriptor list: out_q = X_q + t_q·dX_q (k_q × k_q).
struct TrialFew {
  TrialDesc t[kTrialInline];
};
__global__ void k_make_trials_list(const __grid_constant__ TrialFew few, const TrialDesc* d, int n) {
  const int q = blockIdx.y;
  const TrialDesc T = n <= kTrialInline ? few.t[q] : d[q];
  const long long tot = (long long)T.k * T.k;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < tot;
       e += (long long)gridDim.x * blockDim.x)
    T.out[e] = T.X[e] + T.t * T.dX[e];
}
void make_trials_list(const TrialDesc* list, TrialDesc* d_list, int n, int kmax, cudaStream_t st) {
  if (n == 0) return;
  TrialFew few{};
  if (n <= kTrialInline) std::copy(list, list + n, few.t);
  else SDPX_CUDA(cudaMemcpyAsync(d_list, list, sizeof(TrialDesc) * n, cudaMemcpyHostToDevice, st));
  int g = std::max(1, std::min(64, ceil_div((long long)kmax * kmax, 256)));
  k_make_trials_list<<<dim3(g, n), 256, 0, st>>>(few, d_list, n);
  SDPX_LAUNCH_CHECK();
}

// ------------------------------------------------------------ permutation --
__global__ void k_gather(long long n, const long long* map, const double* src, double* dst) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n;
       e += (long long)gridDim.x * blockDim.x)
    dst[e] = src[map[e]];
}
__global__ void k_scatter(long long n, const long long* map, const double* src, double* dst) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n;
       e += (long long)gridDim.x * blockDim.x)
    dst[map[e]] = src[e];
}
void gather(long long n, const long long* map, const double* src, double* dst, cudaStream_t st) {
  if (n == 0) return;
  k_gather<<<std::min(4096, ceil_div(n, 256)), 256, 0, st>>>(n, map, src, dst);
  SDPX_LAUNCH_CHECK();
}
void scatter(long long n, const long long* map, const double* src, double* dst, cudaStream_t st) {
  if (n == 0) return;
  k_scatter<<<std::min(4096, ceil_div(n, 256)), 256, 0, st>>>(n, map, src, dst);
  SDPX_LAUNCH_CHECK();
}

__global__ void k_scatter_axpby(long long n, const long long* map, double a, const double* x, double b,
                                const double* y, double* dst) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n;
       e += (long long)gridDim.x * blockDim.x)
    dst[map[e]] = a * x[e] + b * y[e];
}
void scatter_axpby(long long n, const long long* map, double a, const double* x, double b, const double* y,
                   double* dst, cudaStream_t st) {
  if (n == 0) return;
  k_scatter_axpby<<<std::min(4096, ceil_div(n, 256)), 256, 0, st>>>(n, map, a, x, b, y, dst);
  SDPX_LAUNCH_CHECK();
}

// --------------------------------------------------------- dense S helpers --
// Full symmetric S from its lower triangle (upper ← lower).
__global__ void k_mirror_lower(int m, double* S) {
  long long tot = (long long)m * m;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < tot;
       e += (long long)gridDim.x * blockDim.x) {
    int i = (int)(e % m), j = (int)(e / m);
    if (i < j) S[e] = S[j + (long long)i * m];
  }
}
void mirror_lower(int m, double* S, cudaStream_t st) {
  k_mirror_lower<<<std::min(4096, ceil_div((long long)m * m, 256)), 256, 0, st>>>(m, S);
  SDPX_LAUNCH_CHECK();
}

// Sf = S (lower) with diagonal += reg·max(|S_ii|, 1)   (src/kkt.jl:1419-1445)
__global__ void k_copy_reg(int m, const double* S, double* Sf, double reg, const int* err, int* err_out) {
  if (err && blockIdx.x == 0 && threadIdx.x == 0) *err_out = *err;
  long long tot = (long long)m * m;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < tot;
       e += (long long)gridDim.x * blockDim.x) {
    int i = (int)(e % m), j = (int)(e / m);
    double v = (i >= j) ? S[e] : 0.0;
    if (i == j && reg != 0.0) v += reg * fmax(fabs(S[e]), 1.0);
    Sf[e] = v;
  }
}
void copy_reg(int m, const double* S, double* Sf, double reg, cudaStream_t st, const int* err, int* err_out) {
  k_copy_reg<<<std::min(4096, ceil_div((long long)m * m, 256)), 256, 0, st>>>(m, S, Sf, reg, err, err_out);
  SDPX_LAUNCH_CHECK();
}

__global__ void k_copy_pair(long long n, const double* s0, double* d0, const double* s1, double* d1) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n;
       e += (long long)gridDim.x * blockDim.x) {
    const double a = s0[e], b = s1[e];
    d0[e] = a;
    d1[e] = b;
  }
}
void copy_pair(long long n, const double* s0, double* d0, const double* s1, double* d1, cudaStream_t st) {
  if (n == 0) return;
  k_copy_pair<<<std::min(4096, ceil_div(n, 256)), 256, 0, st>>>(n, s0, d0, s1, d1);
  SDPX_LAUNCH_CHECK();
}

// y = alpha·S·x + beta·b for symmetric S stored full (column i = row i).
__global__ void k_symv_full(int m, const double* S, const double* x, double alpha, const double* b,
                            double beta, double* y) {
  int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= m) return;
  const double* col = S + (long long)warp * m;
  double acc = 0.0;
  for (int j = lane; j < m; j += 32) acc += col[j] * x[j];
  acc = warp_sum(acc);
  if (lane == 0) y[warp] = alpha * acc + (b ? beta * b[warp] : 0.0);
}
void symv_full(int m, const double* S, const double* x, double alpha, const double* b, double beta,
               double* y, cudaStream_t st) {
  k_symv_full<<<ceil_div((long long)m * 32, 256), 256, 0, st>>>(m, S, x, alpha, b, beta, y);
  SDPX_LAUNCH_CHECK();
}

// --------------------------------------------------------- equilibration ---
// Ruiz passes on the unscaled data with the factors of the passes before: a pass only
// reads 𝒜, which is written once at the end, every entry multiplied by one pass's
// e_r·e_c after the other, as if each pass had scaled it.  (Scaling 𝒜 in every pass and C
// on the host took 6.5 + 2.6 ms of kernels for m = 2000, k = 400 + 200, four passes, a
// copy of 𝒜 and a round trip of C a pass.)  F holds the factors of pass p at p·rows.
//
// rn[r] = max(rn[r], max |A_i[r,c]·…|) over the columns i of 𝒜 and C (i = m), for a dense
// block, after NP passes.  CTA i walks A_i's k×k block column by column with thread r
// holding row r's maximum in a register (each column read coalesced, no index
// division, no shared-memory atomics), then one atomic per row.  NaN counts as +inf.
template <int NP>
__global__ void k_ruiz_rowmax_dense(const double* __restrict__ A, const double* __restrict__ C, long long K,
                                    int m, long long off, int k, const double* __restrict__ F, int rows,
                                    const int* __restrict__ active, double* rn) {
  if (!*active) return;
  const double* blk = ((int)blockIdx.x < m ? A + (long long)blockIdx.x * K : C) + off;
  for (int r = threadIdx.x; r < k; r += blockDim.x) {
    double er[NP + 1];
#pragma unroll
    for (int p = 0; p < NP; ++p) er[p] = F[p * rows + r];
    double mx = 0.0;
#pragma unroll 8
    for (int c = 0; c < k; ++c) {
      double v = blk[(long long)c * k + r];
#pragma unroll
      for (int p = 0; p < NP; ++p) v *= er[p] * F[p * rows + c];
      v = fabs(v);
      if (!(v == v)) v = 1.0 / 0.0;
      mx = fmax(mx, v);
    }
    atomic_max_nonneg(rn + r, mx);
  }
}
// The same for the 1×1 group, the constraints split into chunks of 16 across blockIdx.y
// (an atomic per chunk) so that the pass is spread over the whole GPU rather than one
// thread per j.
constexpr int kRuizDiagChunk = 16;
template <int NP>
__global__ void k_ruiz_rowmax_diag(const double* __restrict__ A, const double* __restrict__ C, long long K,
                                   int m, long long od, int nd, const double* __restrict__ F, int rows,
                                   const int* __restrict__ active, double* rn) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= nd || !active[j]) return;
  double e2[NP + 1];
#pragma unroll
  for (int p = 0; p < NP; ++p) e2[p] = F[p * rows + j] * F[p * rows + j];
  for (int i0 = blockIdx.y * kRuizDiagChunk; i0 <= m; i0 += gridDim.y * kRuizDiagChunk) {
    const int i1 = min(m + 1, i0 + kRuizDiagChunk);
    double v = 0.0;
    for (int i = i0; i < i1; ++i) {
      double a = i < m ? A[od + j + (long long)i * K] : C[od + j];
#pragma unroll
      for (int p = 0; p < NP; ++p) a *= e2[p];
      a = fabs(a);
      if (!(a == a)) a = 1.0 / 0.0;
      v = fmax(v, a);
    }
    atomic_max_nonneg(rn + j, v);
  }
}
// f(integral_constant<n>) for a run-time 0 ≤ n ≤ 8.
template <int N = 0, class F>
static void with_passes(int n, F f) {
  if constexpr (N <= 8) {
    if (n == N) return f(std::integral_constant<int, N>());
    with_passes<N + 1>(n, f);
  }
}
void ruiz_rowmax_dense(const double* A, const double* C, long long K, int m, long long off, int k, int np,
                       const double* F, int rows, const int* active, double* rn, cudaStream_t st) {
  if (k == 0) return;
  const int threads = std::min(512, ceil_div(k, 32) * 32);
  with_passes(np, [&](auto n) {
    k_ruiz_rowmax_dense<decltype(n)::value><<<m + 1, threads, 0, st>>>(A, C, K, m, off, k, F, rows, active, rn);
  });
  SDPX_LAUNCH_CHECK();
}
void ruiz_rowmax_diag(const double* A, const double* C, long long K, int m, long long od, int nd, int np,
                      const double* F, int rows, const int* active, double* rn, cudaStream_t st) {
  if (nd == 0) return;
  dim3 grid(ceil_div(nd, 128), std::min(65535, ceil_div(m + 1, kRuizDiagChunk)));
  with_passes(np, [&](auto n) {
    k_ruiz_rowmax_diag<decltype(n)::value><<<grid, 128, 0, st>>>(A, C, K, m, od, nd, F, rows, active, rn);
  });
  SDPX_LAUNCH_CHECK();
}

// End of pass `it`: factors f_r = 1/√rn_r (where positive, else 1) of the active blocks
// into F, E_r ← E_r·f_r; a block becomes inactive from the second pass on when every
// |log rn_r| ≤ 1/20; rn ← 0.  One CTA per dense block, then 256 of the 1×1 blocks each.
// used = last pass of a block; *any (pinned) = it while a block stays active.
__global__ void __launch_bounds__(256) k_ruiz_update(int it, int nb, const int* __restrict__ kk,
                                                     const int* __restrict__ row0, int nd, double* rn,
                                                     double* F, double* E, int* active, int* used, int* any) {
  const int b = blockIdx.x;
  const bool dense = b < nb;
  const int j = dense ? 0 : (b - nb) * 256 + (int)threadIdx.x;
  const int blk = dense ? b : nb + j, r0 = dense ? row0[b] : row0[nb] + j;
  const int n = dense ? kk[b] : j < nd ? 1 : 0;
  const bool act = n > 0 && active[blk];
  bool ok = true;  // every |log rn| within the limit
  for (int r = dense ? threadIdx.x : 0; r < n; r += 256) {
    const double v = act ? rn[r0 + r] : 0.0;
    double f = 1.0;
    if (v > 0) {
      ok = ok && isfinite(v) && fabs(log(v)) <= 1.0 / 20.0;
      f = 1.0 / sqrt(v);
    }
    rn[r0 + r] = 0.0;
    F[r0 + r] = f;
    E[r0 + r] *= f;
  }
  const bool conv = (dense ? __syncthreads_and(ok) : ok) && it >= 2;
  if (!act || (dense && threadIdx.x != 0)) return;
  used[blk] = it;
  if (conv) active[blk] = 0;
  else *any = it;
}
void ruiz_update(int it, int nb, const int* d_k, const int* d_row0, int nd, double* rn, double* F, double* E,
                 int* active, int* used, int* any, cudaStream_t st) {
  k_ruiz_update<<<nb + ceil_div(nd, 256), 256, 0, st>>>(it, nb, d_k, d_row0, nd, rn, F, E, active, used, any);
  SDPX_LAUNCH_CHECK();
}

// w[p·K + q] = e_r·e_c of pass p (blockIdx.z) for every stacked entry q.
__global__ void k_ruiz_weights(int nb, const int* __restrict__ kk, const long long* __restrict__ off,
                               const int* __restrict__ row0, int nd, long long od, long long K,
                               const double* __restrict__ F, int rows, double* w) {
  const int b = blockIdx.y;
  const double* e = F + (long long)blockIdx.z * rows + row0[b];
  w += blockIdx.z * K;
  if (b == nb) {
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < nd; j += gridDim.x * blockDim.x) w[od + j] = e[j] * e[j];
    return;
  }
  const int k = kk[b];
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < (long long)k * k;
       q += (long long)gridDim.x * blockDim.x)
    w[off[b] + q] = e[q % k] * e[q / k];
}
void ruiz_weights(int nb, const int* d_k, const long long* d_off, const int* d_row0, int kmax, int nd,
                  long long od, long long K, int np, const double* F, int rows, double* w, cudaStream_t st) {
  const long long most = std::max<long long>((long long)kmax * kmax, nd);
  k_ruiz_weights<<<dim3(std::min(256, std::max(1, ceil_div(most, 256))), nb + 1, np), 256, 0, st>>>(
      nb, d_k, d_off, d_row0, nd, od, K, F, rows, w);
  SDPX_LAUNCH_CHECK();
}

// Column max of the scaled |A[:, i]| → out[i]
template <int NP>
__global__ void k_colmax(const double* __restrict__ A, const double* __restrict__ w, long long K, double* out) {
  __shared__ double red[32];
  int i = blockIdx.x;
  const double* col = A + (long long)i * K;
  double v = 0.0;
#pragma unroll 4
  for (long long r = threadIdx.x; r < K; r += blockDim.x) {
    double a = col[r];
#pragma unroll
    for (int p = 0; p < NP; ++p) a *= w[p * K + r];
    a = fabs(a);
    if (!(a == a)) a = 1.0 / 0.0;
    v = fmax(v, a);
  }
  v = block_max(v, red);
  if (threadIdx.x == 0) out[i] = v;
}
void colmax(const double* A, const double* w, int np, long long K, int m, double* out, cudaStream_t st) {
  if (m == 0) return;
  with_passes(np, [&](auto n) { k_colmax<decltype(n)::value><<<m, 512, 0, st>>>(A, w, K, out); });
  SDPX_LAUNCH_CHECK();
}

// A0 ← A (unless null), A[q, i] ← A[q, i]·w_q… / s_i (s null: 1): a thread keeps its row's
// weights for eight columns, whose loads are in flight together.
constexpr int kScaleCols = 8;
template <int NP>
__global__ void k_scale_store(double* __restrict__ A, double* __restrict__ A0, long long K, int m,
                              const double* __restrict__ w, const double* __restrict__ s) {
  const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (q >= K) return;
  double wq[NP + 1];
#pragma unroll
  for (int p = 0; p < NP; ++p) wq[p] = w[p * K + q];
  for (int i0 = blockIdx.y * kScaleCols; i0 < m; i0 += gridDim.y * kScaleCols) {
    double v[kScaleCols];
#pragma unroll
    for (int u = 0; u < kScaleCols; ++u) v[u] = i0 + u < m ? A[(i0 + u) * K + q] : 0.0;
#pragma unroll
    for (int u = 0; u < kScaleCols; ++u) {
      if (i0 + u >= m) break;
      if (A0) A0[(i0 + u) * K + q] = v[u];
#pragma unroll
      for (int p = 0; p < NP; ++p) v[u] *= wq[p];
      A[(i0 + u) * K + q] = s ? v[u] / s[i0 + u] : v[u];
    }
  }
}
void scale_store(double* A, double* A0, long long K, int m, const double* w, int np, const double* s,
                 cudaStream_t st) {
  if (K == 0 || m == 0) return;
  const dim3 grid(ceil_div(K, 256), std::min(65535, ceil_div(m, kScaleCols)));
  with_passes(np, [&](auto n) { k_scale_store<decltype(n)::value><<<grid, 256, 0, st>>>(A, A0, K, m, w, s); });
  SDPX_LAUNCH_CHECK();
}

}  // namespace sdpx
