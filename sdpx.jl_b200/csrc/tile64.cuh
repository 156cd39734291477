// A 64×64 FP64 tile in shared memory, worked on by eight warps: its Cholesky factor
// and the triangular solve against it.
//
// Warp w owns rows 8w … 8w+7 (a strip); as DMMA accumulators lane 4g+t holds row g,
// columns 8f+2t and 8f+2t+1 of fragment f.  Orders below 64 use the first nb strips, the
// tile padded with the identity to 8·nb.  The arithmetic of every element is the
// unblocked right-looking factorization's: products subtracted one by one in
// increasing column order, columns scaled by the reciprocal pivot (LAPACK's dpotf2).
#pragma once
#include "common.cuh"

namespace sdpx {
namespace tile64 {

constexpr int FB = 64;        // tile order
constexpr int FLD = FB + 4;   // leading dimension: ≡ 4 (mod 16) doubles, so the fragment
                              // reads (4 k × 4 rows per half-warp) hit 16 banks
constexpr int FT = 256;       // threads
constexpr int kNoFail = 1 << 30;

__device__ __forceinline__ void bar_sync(int id, int n) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int n) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory");
}
// dmma_8x8x4 without the ordering of a volatile asm.
__device__ __forceinline__ void mma8(double& c0, double& c1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
      : "+d"(c0), "+d"(c1)
      : "d"(a), "d"(b));
}

// Rows 8b … 8b+7 (columns 8p … 8p+7 and below) as B operand, X's strip as A:
// x −= X_p·L_{b,p}ᵀ for p < np, one product after the other.
__device__ __forceinline__ void subtract_products(double (&x)[2], const double* Xr, const double* L, int b,
                                                  int np) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const double *a = Xr + t * FLD + g, *l = L + t * FLD + 8 * b + g;
#pragma unroll 2
  for (int k = 0; k < 2 * np; ++k, a += 4 * FLD, l += 4 * FLD) mma8(x[0], x[1], -*a, *l);
}

// Eight columns of a strip (block b, in x) solved against the 8×8 diagonal block
// of L (D[c·FLD + r] = L[r][c], inv = reciprocal pivots): x_c ← x_c·inv_c, then
// x_q −= x_c·L[q][c] for q > c, into the strip's place in X.  One lane per row:
// the chain is a product and an fma a column, where the four lanes of a row in
// fragment layout would add a shuffle.
__device__ __forceinline__ void solve8(const double (&x)[2], double* Xr, const double* D, const double* inv,
                                       int b) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  double* xs = Xr + (8 * b) * FLD;
  xs[(2 * t) * FLD + g] = x[0];
  xs[(2 * t + 1) * FLD + g] = x[1];
  __syncwarp();
  if (lane < 8) {
    const double* d = D + (8 * b) * FLD + 8 * b;
    double v[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) v[c] = xs[c * FLD + lane];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      v[c] *= inv[8 * b + c];
#pragma unroll
      for (int q = (c + 1) & ~1; q < 8; q += 2) {  // rows q, q+1 in one 16-byte load
        const double2 l = *reinterpret_cast<const double2*>(d + c * FLD + q);
        if (q > c) v[q] -= v[c] * l.x;
        v[q + 1] -= v[c] * l.y;
      }
    }
#pragma unroll
    for (int c = 0; c < 8; ++c) xs[c * FLD + lane] = v[c];
  }
  __syncwarp();
}

// X ← X·L⁻ᵀ for the warp's strip of X, L the lower tile in D (its first nb strips).
__device__ __forceinline__ void solve_strip(double* X, const double* D, const double* inv, int nb = 8) {
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  double* Xr = X + 8 * wp;
#pragma unroll 1
  for (int b = 0; b < nb; ++b) {
    double x[2] = {Xr[(8 * b + 2 * t) * FLD + g], Xr[(8 * b + 2 * t + 1) * FLD + g]};
    subtract_products(x, Xr, D, b, b);
    solve8(x, Xr, D, inv, b);
  }
}

// l = √a and 1/l, both correctly rounded, for normal a far from the ends of the
// range: y = a^(-1/2) from the hardware's approximation y0 by the series of
// (1 − e)^(-1/2), e = 1 − a·y0², then l = s + (a − s²)·y/2 with s = a·y and
// 1/l = y + (1 − l·y)·y (Markstein, "Computation of elementary functions on the IBM
// RISC System/6000", 1990).  No branch; about 105 cycles where sqrt() and a division
// take 153 one after the other.  Equal to those bit for bit on 6e9 values but for
// the reciprocal of l = 2 − 2⁻⁵² (times powers of two), which is 1 ulp off.
__device__ __forceinline__ void sqrt_rcp(double a, double& l, double& inv) {
  double y0;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(a));
  const double e = fma(-(a * y0), y0, 1.0);
  const double y = fma(y0 * e, fma(e, 0.375, 0.5), y0), s = a * y;
  l = fma(fma(-s, s, a), 0.5 * y, s);
  inv = fma(fma(-l, y, 1.0), y, y);
}

// The 8×8 diagonal block at d (leading dimension FLD, lower part), factored by
// every lane of one warp alike from broadcast reads: no shuffle in the chain, and
// the other products fill its gaps.  iv: reciprocal pivots.  Returns the failing
// column or −1; nothing is written unless it is −1.  careful = false assumes
// pivots in (2⁻⁸³⁰, 2⁸³⁰) and returns −2 when one was not: the caller then starts
// again with careful = true, so the usual case has no branch in its chain.
template <bool careful>
__device__ __forceinline__ int factor8(double* d, double* iv) {
  double B[8][8], v[8];
#pragma unroll
  for (int c = 0; c < 8; ++c)
#pragma unroll
    for (int r = c & ~1; r < 8; r += 2) {
      const double2 u = *reinterpret_cast<const double2*>(d + c * FLD + r);
      B[c][r] = u.x;
      B[c][r + 1] = u.y;
    }
  bool odd = false;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const double piv = B[c][c];
    if (careful) {
      if (!(piv > 0.0)) return c;
      B[c][c] = sqrt(piv);
      v[c] = 1.0 / B[c][c];
    } else {
      odd |= (unsigned)(__double2hiint(piv) - ((1023 - 830) << 20)) >= (1660u << 20);
      sqrt_rcp(piv, B[c][c], v[c]);
    }
#pragma unroll
    for (int r = c + 1; r < 8; ++r) B[c][r] *= v[c];
#pragma unroll
    for (int q = c + 1; q < 8; ++q)
#pragma unroll
      for (int r = q; r < 8; ++r) B[q][r] -= B[c][r] * B[c][q];
  }
  if (odd) return -2;
  __syncwarp();
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int c = 0; c < 8; ++c) {
#pragma unroll
      for (int r = c; r < 8; ++r) d[c * FLD + r] = B[c][r];
      iv[c] = v[c];
    }
  }
  __syncwarp();
  return -1;
}

// The tile in D (its first nb strips) factored in place, reciprocal pivots to inv.
// Warp b factors diagonal block b as soon as its own rows are up to date; the
// warps below solve their rows of block column b, and only then read each other's
// rows, to bring their next block up to date while warp b+1 factors.  So two named
// barriers per block suffice, and of the second the next warp to factor does not
// wait.  *sfail (kNoFail before) receives the failing column.
__device__ __forceinline__ void factor_tile(double* D, double* inv, int nb, int* sfail) {
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  if (wp >= nb) return;
  double* Dr = D + 8 * wp;
  double* dd = Dr + (8 * wp) * FLD;  // the warp's diagonal block
  double xd[2] = {dd[(2 * t) * FLD + g], dd[(2 * t + 1) * FLD + g]};
#pragma unroll 1
  for (int b = 0; b < wp; ++b) {
    double x[2] = {Dr[(8 * b + 2 * t) * FLD + g], Dr[(8 * b + 2 * t + 1) * FLD + g]};
    subtract_products(x, Dr, D, b, b);
    bar_sync(1 + (b & 1), 32 * (nb - b));  // block b is factored
    solve8(x, Dr, D, inv, b);
    const double* o = Dr + (8 * b + t) * FLD + g;  // the own rows on both sides
    mma8(xd[0], xd[1], -o[0], o[0]);
    mma8(xd[0], xd[1], -o[4 * FLD], o[4 * FLD]);
    if (wp == b + 1) bar_arrive(3 + (b & 1), 32 * (nb - 1 - b));
    else bar_sync(3 + (b & 1), 32 * (nb - 1 - b));
  }
  dd[(2 * t) * FLD + g] = xd[0];
  dd[(2 * t + 1) * FLD + g] = xd[1];
  __syncwarp();
  int fail = factor8<false>(dd, inv + 8 * wp);
  if (fail == -2) fail = factor8<true>(dd, inv + 8 * wp);
  if (fail >= 0) {  // the warps below go on with NaN pivots, and fail too
    if (lane < 8) inv[8 * wp + lane] = NAN;
    if (lane == 0) atomicMin(sfail, 8 * wp + fail);
    __syncwarp();
  }
  if (wp < nb - 1) bar_arrive(1 + (wp & 1), 32 * (nb - wp));
}

// ---- whole k×k matrices (k ≤ 64) by FT threads: column c at c·FLD, padded with the identity
// to 8·nb rows and columns, nb = ⌈k/8⌉, so the DMMA products need no guards and their
// fragment reads no bank conflicts.

// S ← G (k×k column-major, global); t: its transpose.  All loads are issued before the
// first shared store (one memory round trip a matrix).
__device__ __forceinline__ void cta_load_tile(double* S, const double* G, int k, bool t = false) {
  const int r = threadIdx.x & 63, cb = threadIdx.x >> 6, k8 = (k + 7) & ~7;
  double v[16];
#pragma unroll
  for (int u = 0; u < 16; ++u) {
    const int c = cb + 4 * u;
    v[u] = (r < k && c < k) ? G[r + c * k] : (r == c ? 1.0 : 0.0);
  }
  if (r < k8)
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      const int c = cb + 4 * u;
      if (c < k8) S[t ? r * FLD + c : c * FLD + r] = v[u];
    }
}
// f(r, c, Σ_p op(A)(r, p)·B(p, c)) over the 8·nb square, for tiles A, B; ta: A
// transposed.  first(i), last(i): the range of 8-blocks p that block row i needs (a
// triangular A).  Each warp takes pairs of 8×8 output blocks of a block row in
// turn, two chains to cover the pipe's latency.
enum TileTri { kFull, kLower, kUpper };  // op(A)
template <bool ta, TileTri tri, class F>
__device__ __forceinline__ void cta_tile_gemm(const double* A, const double* B, int nb, F f) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int pairs = (nb + 1) / 2;
  for (int u = warp; u < nb * pairs; u += FT / 32) {
    const int i = u % nb, c0 = 16 * (u / nb);
    const bool two = c0 + 8 < 8 * nb;
    const int p0 = tri == kUpper ? 2 * i : 0, p1 = tri == kLower ? 2 * i + 2 : 2 * nb;
    double acc[2][2] = {};
    for (int p = p0; p < p1; ++p) {
      const int q = 4 * p + t;
      const double a = ta ? A[(8 * i + g) * FLD + q] : A[q * FLD + 8 * i + g];
      mma8(acc[0][0], acc[0][1], a, B[(c0 + g) * FLD + q]);
      if (two) mma8(acc[1][0], acc[1][1], a, B[(c0 + 8 + g) * FLD + q]);
    }
#pragma unroll
    for (int v = 0; v < 2; ++v)
#pragma unroll
      for (int e = 0; e < 2; ++e)
        if (v == 0 || two) f(8 * i + g, c0 + 8 * v + 2 * t + e, acc[v][e]);
  }
}

// X⁻¹·B = Wᵀ·(W·B) for W = L_X⁻¹ in a tile: T (scratch) ← W·B, then f of the product.
template <class F>
__device__ __forceinline__ void cta_tile_cholsolve(const double* W, const double* B, double* T, int nb, F f) {
  cta_tile_gemm<false, kLower>(W, B, nb, [&](int r, int c, double v) { T[c * FLD + r] = v; });
  __syncthreads();
  cta_tile_gemm<true, kUpper>(W, T, nb, f);
}

}  // namespace tile64
}  // namespace sdpx
