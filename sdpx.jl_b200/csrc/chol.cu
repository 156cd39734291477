// Cholesky (lower, right-looking, panel width NB).  Orders whose NB-wide
// panel fits in shared memory (the line-search trials and block factors) take
// one launch per panel that factors the whole panel in place; larger orders
// factor the diagonal tile once (one CTA per matrix), solve the rows below it
// with one thread per row, and update the trailing lower tiles.  A matrix whose
// pivot is not positive (or NaN) records `info = pivot index + 1` and every
// later CTA of that matrix returns at once — the no-throw contract of SDPX's
// `kchol!` (src/kernels/generic.jl:133-155).
//
// Inside a panel the columns are processed in blocks of 8: l_cc = sqrt(a_cc),
// l_rc = a_rc · (1/l_cc) (the reciprocal scaling of LAPACK's dpotf2),
// a_rq -= l_rc · l_qc, every element updated in increasing column order.
#include "chol.h"
#include "blas_f64.h"

namespace sdpx {

// Right-looking factor of the leading w columns of the rows×w panel P (shared,
// column-major, leading dimension ld; rows ≥ w).  Returns the failing column
// or -1.  All threads of the CTA take part.
//
// Blocked by 8 columns: every thread factors the 8×8 diagonal block in its
// registers (l_cc = sqrt(a_cc), column below scaled by 1/l_cc, as LAPACK's
// unblocked dpotf2 does) — the same arithmetic in every thread, so the factor
// needs no publication and no barrier of its own; each row below the block is
// solved in registers (x = a · L_bb^{-T}); after one barrier the trailing
// columns of the panel receive the rank-8 update (the block's rows read as
// warp broadcasts) while thread 0 writes the factored block back.  Two
// barriers per 8 columns.  Every element sees its updates in increasing column
// order.
template <class T>
__device__ int factor_panel_smem(T* P, int ld, int rows, int w) {
  __syncthreads();
  for (int kb = 0; kb < w; kb += 8) {
    const int kw = min(8, w - kb);
    T D[8][8], inv[8];
#pragma unroll
    for (int c = 0; c < 8; ++c)
#pragma unroll
      for (int r = 0; r < 8; ++r)
        D[c][r] = (c < kw && r < kw && r >= c) ? P[(kb + c) * ld + kb + r] : T(0);
    int fail = -1;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      inv[c] = T(0);
      if (c < kw && fail < 0) {
        const T piv = D[c][c];
        if (!(piv > T(0))) {
          fail = c;
        } else {
          const T lc = sqrt(piv);
          inv[c] = T(1) / lc;
          D[c][c] = lc;
#pragma unroll
          for (int r = c + 1; r < 8; ++r) D[c][r] *= inv[c];
#pragma unroll
          for (int q = c + 1; q < 8; ++q)
#pragma unroll
            for (int r = q; r < 8; ++r) D[q][r] -= D[c][r] * D[c][q];
        }
      }
    }
    if (fail >= 0) return kb + fail;  // the same in every thread
    // rows below the block: x = a · L_bb^{-T}
    for (int r = kb + kw + threadIdx.x; r < rows; r += blockDim.x) {
      T x[8];
#pragma unroll
      for (int c = 0; c < 8; ++c) x[c] = (c < kw) ? P[(kb + c) * ld + r] : T(0);
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        if (c < kw) {
          x[c] *= inv[c];
#pragma unroll
          for (int q = c + 1; q < 8; ++q) x[q] -= x[c] * D[c][q];
        }
      }
#pragma unroll
      for (int c = 0; c < 8; ++c)
        if (c < kw) P[(kb + c) * ld + r] = x[c];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
      for (int c = 0; c < 8; ++c)
#pragma unroll
        for (int r = 0; r < 8; ++r)
          if (c < kw && r < kw && r >= c) P[(kb + c) * ld + kb + r] = D[c][r];
    }
    // trailing panel columns q ∈ [kb+kw, w), rows r ≥ q.  With fewer rows
    // than threads (the diagonal tiles, the short last panels) several threads
    // share a row and take every `slices`-th column of it; each element gets
    // the same sum in the same order either way.
    {
      const int r0 = kb + kw, nrow = rows - r0;
      const int slices = nrow > 0 ? max(1, (int)blockDim.x / nrow) : 1;
      for (int idx = threadIdx.x; idx < nrow * slices; idx += blockDim.x) {
        const int r = r0 + idx % nrow, sl = idx / nrow;
        T x[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) x[c] = (c < kw) ? P[(kb + c) * ld + r] : T(0);
        const int qe = min(w, r + 1);
        for (int q = r0 + sl; q < qe; q += slices) {
          T a = P[q * ld + r];
#pragma unroll
          for (int c = 0; c < 8; ++c)
            if (c < kw) a -= x[c] * P[(kb + c) * ld + q];
          P[q * ld + r] = a;
        }
      }
    }
    __syncthreads();
  }
  return -1;
}

template <class T>
__device__ void note_pivots(const T* P, int ld, int w, T* dmin, T* dmax, int b) {
  if (threadIdx.x != 0) return;
  T lo = dmin[b], hi = dmax[b];
  for (int c = 0; c < w; ++c) {
    T v = fabs(P[c * ld + c]);
    lo = fmin(lo, v);
    hi = fmax(hi, v);
  }
  dmin[b] = lo;
  dmax[b] = hi;
}

// The lower part of the w×w diagonal tile at (c0, c0) into shared D (column
// c at D[c·LD + …], zeros above the diagonal and outside w).  NT threads; each
// issues all of its NB·NB/NT loads before any shared store, so the tile costs
// one memory round trip.
template <class T, int NB, int NT>
__device__ __forceinline__ void load_diag_tile(T* D, int LD, const MatDesc<T>& M, int c0, int w) {
  constexpr int PER = NB * NB / NT;
  static_assert(NB * NB % NT == 0, "tile split");
  T v[PER];
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const int e = threadIdx.x + k * NT, r = e % NB, c = e / NB;
    v[k] = (r < w && c < w && r >= c) ? M.a[(size_t)(c0 + c) * M.ld + (c0 + r)] : T(0);
  }
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const int e = threadIdx.x + k * NT, r = e % NB, c = e / NB;
    if (r < w && c < w) D[c * LD + r] = v[k];
  }
}

// Tiled path, step 1: factor the diagonal tile of panel j (one CTA per matrix).
template <class T, int NB>
__global__ void __launch_bounds__(256) k_potrf_diag(const MatDesc<T>* mats, int j, int* info, T* dmin, T* dmax) {
  __shared__ T D[NB * (NB + 1)];
  constexpr int LD = NB + 1;
  const int b = blockIdx.x;
  const MatDesc<T> M = mats[b];
  const int c0 = j * NB;
  if (c0 >= M.n || info[b] != 0) return;
  const int w = min(NB, M.n - c0);
  load_diag_tile<T, NB, 256>(D, LD, M, c0, w);
  const int fail = factor_panel_smem<T>(D, LD, w, w);
  if (fail >= 0) {
    if (threadIdx.x == 0) info[b] = c0 + fail + 1;
    return;
  }
  for (int e = threadIdx.x; e < NB * NB; e += blockDim.x) {
    const int r = e % NB, c = e / NB;
    if (r < w && c < w && r >= c) M.a[(size_t)(c0 + c) * M.ld + (c0 + r)] = D[c * LD + r];
  }
  note_pivots(D, LD, w, dmin, dmax, b);
}

// Tiled path, step 2: rows below the diagonal tile, X = B · L_jj^{-T}, one
// thread per row with the row held in registers (forward substitution in the
// column order of the right-looking panel factor, scaling by the reciprocal
// pivots).
template <class T, int NB>
__global__ void __launch_bounds__(128) k_potrf_trsm_rows(const MatDesc<T>* mats, int j,
                                                         const int* info) {
  __shared__ T D[NB * (NB + 1)];
  constexpr int LD = NB + 1;
  const int b = blockIdx.y;
  const MatDesc<T> M = mats[b];
  const int c0 = j * NB;
  if (c0 >= M.n || info[b] != 0) return;
  const int w = min(NB, M.n - c0);
  const int first = c0 + w + blockIdx.x * blockDim.x;
  if (first >= M.n) return;
  load_diag_tile<T, NB, 128>(D, LD, M, c0, w);
  __shared__ T inv[NB];
  __syncthreads();  // the diagonal tile is loaded
  for (int c = threadIdx.x; c < w; c += blockDim.x) inv[c] = T(1) / D[c * LD + c];
  __syncthreads();
  const int r = first + threadIdx.x;
  if (r >= M.n) return;
  T x[NB];
#pragma unroll
  for (int c = 0; c < NB; ++c) x[c] = (c < w) ? M.a[(size_t)(c0 + c) * M.ld + r] : T(0);
#pragma unroll
  for (int c = 0; c < NB; ++c) {
    if (c < w) {
      x[c] *= inv[c];
#pragma unroll
      for (int q = c + 1; q < NB; ++q) x[q] -= x[c] * D[c * LD + q];
    }
  }
#pragma unroll
  for (int c = 0; c < NB; ++c)
    if (c < w) M.a[(size_t)(c0 + c) * M.ld + r] = x[c];
}

// Whole panel in shared memory (orders n with n·NB elements ≤ 224 KB): one CTA
// per matrix loads rows [c0, n) of panel j, factors it in place and writes it
// back; the trailing tiles are then updated by k_potrf_update.
template <class T, int NB>
__global__ void __launch_bounds__(512) k_potrf_panel_smem(const MatDesc<T>* mats, int j, int* info, T* dmin, T* dmax) {
  extern __shared__ __align__(16) unsigned char raw[];
  T* Pn = reinterpret_cast<T*>(raw);  // rows × NB, column-major with ld = rows | 1
  const MatDesc<T> M = mats[blockIdx.x];
  const int b = blockIdx.x;
  const int c0 = j * NB;
  if (c0 >= M.n || info[b] != 0) return;
  const int w = min(NB, M.n - c0);
  const int rows = M.n - c0;
  const int ld = rows | 1;  // odd stride: conflict-free column walks
  // A warp per column, lanes along the rows; each lane issues its PU loads of
  // a batch before storing any, so a column costs one memory round trip per
  // 32·PU rows instead of one per element.
  constexpr int PU = 8;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  for (int c = warp; c < w; c += nwarp) {
    const T* src = M.a + (size_t)(c0 + c) * M.ld + c0;
    for (int rb = 0; rb < rows; rb += 32 * PU) {
      T v[PU];
#pragma unroll
      for (int u = 0; u < PU; ++u) {
        const int r = rb + lane + 32 * u;
        v[u] = (r < rows && r >= c) ? src[r] : T(0);
      }
#pragma unroll
      for (int u = 0; u < PU; ++u) {
        const int r = rb + lane + 32 * u;
        if (r < rows) Pn[c * ld + r] = v[u];
      }
    }
  }
  const int fail = factor_panel_smem<T>(Pn, ld, rows, w);
  if (fail >= 0) {
    if (threadIdx.x == 0) info[b] = c0 + fail + 1;
    return;
  }
  for (int c = warp; c < w; c += nwarp) {
    T* dst = M.a + (size_t)(c0 + c) * M.ld + c0;
    for (int r = lane; r < rows; r += 32) dst[r] = (r >= c) ? Pn[c * ld + r] : T(0);
  }
  note_pivots(Pn, ld, w, dmin, dmax, b);
}

// Trailing update A[i,q] -= L[i,j] L[q,j]^T for j < q <= i (lower tiles).
template <class T, int NB>
__global__ void k_potrf_update(const MatDesc<T>* mats, int j, const int* info) {
  extern __shared__ __align__(16) unsigned char raw[];
  T* La = reinterpret_cast<T*>(raw);  // NB × (NB+1): rows of tile i, panel j
  T* Lb = La + NB * (NB + 1);          // rows of tile q
  constexpr int LD = NB + 1;
  const MatDesc<T> M = mats[blockIdx.y];
  if (info[blockIdx.y] != 0) return;
  const int nt = (M.n + NB - 1) / NB;
  if (j >= nt) return;
  const int rem = nt - j - 1;
  const int u = blockIdx.x;
  if (rem <= 0 || u >= rem * (rem + 1) / 2) return;
  int a = (int)((sqrt(8.0 * u + 1.0) - 1.0) * 0.5);
  while ((a + 1) * (a + 2) / 2 <= u) ++a;
  while (a * (a + 1) / 2 > u) --a;
  const int bq = u - a * (a + 1) / 2;
  const int i = j + 1 + a, q = j + 1 + bq;
  const int c0 = j * NB, r0 = i * NB, q0 = q * NB;
  const int w = min(NB, M.n - c0), h = min(NB, M.n - r0), hq = min(NB, M.n - q0);
  // Each thread owns an RB×RB block of outputs, RB = NB/16: 256 threads for
  // NB = 64 (4×4), 48 (3×3) and 32 (2×2).  Its outputs are read together with
  // the two operand tiles (each output tile belongs to this CTA alone), so the
  // read-modify-write at the end waits for no memory.
  constexpr int RB = NB / 16;
  constexpr int TPR = NB / RB;
  const int tr = threadIdx.x % TPR, tc = threadIdx.x / TPR;
  T cur[RB][RB];
#pragma unroll
  for (int x = 0; x < RB; ++x)
#pragma unroll
    for (int y = 0; y < RB; ++y) {
      const int r = tr + x * TPR, c = tc + y * TPR;
      cur[x][y] = (tc < TPR && r < h && c < hq) ? M.a[(size_t)(q0 + c) * M.ld + (r0 + r)] : T(0);
    }
  {
    // All loads of the two tiles are issued before the shared stores (one
    // memory round trip per tile instead of one per loop trip).
    constexpr int PER = NB * NB / 256;
    static_assert(NB * NB % 256 == 0, "tile load split");
    T va[PER], vb[PER];
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      const int e = threadIdx.x + k * 256, r = e % NB, c = e / NB;
      va[k] = (r < h && c < w) ? M.a[(size_t)(c0 + c) * M.ld + (r0 + r)] : T(0);
      vb[k] = (r < hq && c < w) ? M.a[(size_t)(c0 + c) * M.ld + (q0 + r)] : T(0);
    }
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      const int e = threadIdx.x + k * 256, r = e % NB, c = e / NB;
      La[c * LD + r] = va[k];
      Lb[c * LD + r] = vb[k];
    }
  }
  __syncthreads();
  if (tc < TPR) {
    T acc[RB][RB] = {};
    for (int p = 0; p < w; ++p) {
      T av[RB], bv[RB];
#pragma unroll
      for (int x = 0; x < RB; ++x) av[x] = La[p * LD + tr + x * TPR];
#pragma unroll
      for (int y = 0; y < RB; ++y) bv[y] = Lb[p * LD + tc + y * TPR];
#pragma unroll
      for (int x = 0; x < RB; ++x)
#pragma unroll
        for (int y = 0; y < RB; ++y) acc[x][y] += av[x] * bv[y];
    }
#pragma unroll
    for (int x = 0; x < RB; ++x)
#pragma unroll
      for (int y = 0; y < RB; ++y) {
        int r = tr + x * TPR, c = tc + y * TPR;
        if (r < h && c < hq) M.a[(size_t)(q0 + c) * M.ld + (r0 + r)] = cur[x][y] - acc[x][y];
      }
  }
}

// Strict upper triangle set to zero: a warp per column (rows 0 … c-1).
template <class T>
__global__ void k_zero_upper(const MatDesc<T>* mats) {
  const MatDesc<T> M = mats[blockIdx.y];
  const int lane = threadIdx.x & 31;
  for (int c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); c < M.n;
       c += gridDim.x * (blockDim.x >> 5)) {
    T* col = M.a + (size_t)c * M.ld;
    for (int r = lane; r < c; r += 32) col[r] = T(0);
  }
}

template <class T>
__global__ void k_init_stats(int n, int* info, T* dmin, T* dmax) {
  int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b < n) {
    info[b] = 0;
    dmin[b] = T(1.0 / 0.0);
    dmax[b] = T(0);
  }
}

template <class T, int NB>
void potrf_batched(const MatDesc<T>* d_mats, int nmat, int nmax, int* info, T* dmin, T* dmax,
                   cudaStream_t st, bool zero_upper) {
  if (nmat == 0 || nmax == 0) return;
  const size_t smem = 2 * sizeof(T) * NB * (NB + 1);
  ensure_smem(k_potrf_update<T, NB>, smem);
  k_init_stats<T><<<ceil_div(nmat, 128), 128, 0, st>>>(nmat, info, dmin, dmax);
  const int nt = ceil_div(nmax, NB);
  const int rows_pad = nmax | 1;
  const size_t panel_smem = sizeof(T) * (size_t)rows_pad * NB;
  const bool whole_panel = panel_smem <= 224 * 1024;
  if (whole_panel) ensure_smem(k_potrf_panel_smem<T, NB>, panel_smem);
  int launches = 1;  // k_init_stats
  for (int j = 0; j < nt; ++j) {
    int rem = nt - j - 1;
    if (whole_panel) {
      k_potrf_panel_smem<T, NB><<<nmat, 512, panel_smem, st>>>(d_mats, j, info, dmin, dmax);
      ++launches;
    } else {
      k_potrf_diag<T, NB><<<nmat, 256, 0, st>>>(d_mats, j, info, dmin, dmax);
      ++launches;
      const int below = nmax - (j + 1) * NB;
      if (below > 0) {
        dim3 gt(ceil_div(below, 128), nmat);
        k_potrf_trsm_rows<T, NB><<<gt, 128, 0, st>>>(d_mats, j, info);
        ++launches;
      }
    }
    if (rem > 0) {
      dim3 g2(rem * (rem + 1) / 2, nmat);
      k_potrf_update<T, NB><<<g2, 256, smem, st>>>(d_mats, j, info);
      ++launches;
    }
  }
  if (zero_upper) {
    dim3 gz(std::max(1, ceil_div(nmax, 8)), nmat);
    k_zero_upper<T><<<gz, 256, 0, st>>>(d_mats);
    ++launches;
  }
  SDPX_LAUNCH_CHECK_N(launches);
}

template void potrf_batched<float, 64>(const MatDesc<float>*, int, int, int*, float*, float*,
                                       cudaStream_t, bool);

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
