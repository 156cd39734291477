// Fraction-to-boundary bounds of M + t·dM from eigenvalues: with M = L·Lᵀ and
// G = L⁻¹·dM·L⁻ᵀ, the largest t ≤ 1 that keeps M + t·dM positive semidefinite is
// t* = −1/λ_min(G), or 1 when λ_min(G) ≥ −1 — the value that the 64-step bisection
// of Cholesky tests (`fraction_to_boundary_bound!`, src/kernels/generic.jl:350-422)
// approaches from below, up to the rounding of its tests.
//
// λ_min comes from a Householder tridiagonalisation and a Sturm-count
// multisection.  One cluster of C CTAs per matrix holds it, rows dealt out cyclically
// over the CTAs and their warps.  What bounds it is the chain of k reflections, so each
// has one pass over the rows and one wait: the pass applies the previous reflection's
// rank-2 update and multiplies with this reflection's vector, and its results go to
// every CTA together with the next column, counted by a barrier there.  Up to order 224
// rows and vectors live in registers and every warp forms the next reflection for
// itself (with CTA-wide sums and vectors in shared memory a reflection took 4700 cycles
// at k = 200, 4100 at 61 in one CTA; now 3100 and 2150).  Above it that code, unrolled over
// the order, is bound by instruction fetch: there the rows are in shared memory, the
// loops rolled, and one warp of its own forms the reflections.
//
// Against the bisection's 10 to 15 rounds of batched Cholesky tests (each with its
// uploads, factorizations and read-back), both sides of one iterate on the B200:
//   block orders       12        61 + 17    200       400 + 200
//   bisection rounds   0.45                 2.0       6.3 ms
//   CTA-wide sums      0.021     0.130      0.485     1.22 ms
//   here               0.017     0.074     0.306     1.10 ms
// and within 4e-15 of −1/λ_min in 64 bits where the bisection is, iterates of κ = 100.
#include "step_bound.h"
#include "lambda_bound.cuh"

#include <atomic>
#include <type_traits>

namespace sdpx {
namespace {

constexpr long long kBoundCycles = 1LL << 31;  // limit of a wait, about a second

__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// The address of the same shared location in CTA `rank` of the cluster.
__device__ __forceinline__ unsigned in_cluster(const void* p, unsigned rank) {
  unsigned b;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(b) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
  return b;
}
// (x, y) to a location of another CTA, counted by a barrier of that CTA.
__device__ __forceinline__ void send_pair(unsigned to, double x, double y, unsigned mbar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::"r"(to), "d"(x),
               "d"(y), "r"(mbar)
               : "memory");
}
__device__ __forceinline__ bool barrier_done(unsigned mbar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(mbar), "r"(parity)
      : "memory");
  return ok != 0;
}
// (The .aligned forms take whole warps: lanes may come from loops of different lengths.)
__device__ __forceinline__ void cluster_sync() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Sums over the lanes of N = 4 or 8 values at once: lane l returns that of value l mod N.
template <int N>
__device__ __forceinline__ double sum_many(double (&v)[N]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = N / 2; o >= 1; o >>= 1)
#pragma unroll
    for (int c = 0; c < o; ++c) {
      const bool up = lane & o;
      const double send = up ? v[c] : v[c + o], keep = up ? v[c + o] : v[c];
      v[c] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
#pragma unroll
  for (int o = N; o < 32; o *= 2) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
  return v[0];
}

// min(1, −1/λ_min) of the tridiagonal (d, e) by the whole CTA (BT threads), the same value in
// every thread; 0 when it is not finite.  scratch: 2k doubles.
template <int BT>
__device__ __forceinline__ double tridiagonal_bound(const double* d, const double* e, int k, double* scratch,
                                                    double* red) {
  // Gershgorin bounds
  double lo = INFINITY, hi = INFINITY, nrm = 0.0;
  for (int i = threadIdx.x; i < k; i += BT) {
    const double r = (i > 0 ? fabs(e[i - 1]) : 0.0) + (i + 1 < k ? fabs(e[i]) : 0.0);
    lo = fmin(lo, d[i] - r);
    hi = fmin(hi, d[i]);
    const double n = fabs(d[i]) + r;
    nrm = n == n ? fmax(nrm, n) : INFINITY;
  }
  lo = -block_max(-lo, red);
  hi = -block_max(-hi, red);
  nrm = block_max(nrm, red);
  if (!(nrm < 1e300)) return 0.0;  // non-finite direction: no step
  if (lo >= -1.0) return 1.0;
  const double f = 1.0 / nrm;  // nrm ≥ |lo| > 1
  double *ds = scratch, *es = scratch + k;
  for (int i = threadIdx.x; i < k; i += BT) {
    ds[i] = d[i] * f;
    es[i] = i + 1 < k ? fmax(e[i] * f * (e[i] * f), 1e-36) : 0.0;
  }
  __syncthreads();
  // thread 0 at −1: does the full step stay inside?
  if (!__syncthreads_or(threadIdx.x == 0 && minors_below(ds, es, k, -f) > 0)) return 1.0;
  double l = lo * f - 1e-15, h = fmin(hi * f + 1e-15, -f);
  for (int round = 0; round < 12; ++round) {
    const double step = (h - l) / (BT + 1);
    const int m = __syncthreads_count(minors_below(ds, es, k, l + step * (threadIdx.x + 1)) == 0);
    // counts are monotone: the first m shifts have no eigenvalue below them
    const double nl = m > 0 ? l + step * m : l, nh = m < BT ? l + step * (m + 1) : h;
    l = nl;
    h = nh;
    if (h - l <= 2e-16 * fabs(l)) break;
  }
  return bound_from_below(l / f);
}

// out[q] = bound of matrix q of the list (3 ≤ k ≤ 32·Q, at most R rows a warp): rows in
// registers, the vectors in every warp's, which forms the next reflection for itself.
template <int C, int NW, int Q, int R>
__global__ void __launch_bounds__(32 * NW, 1) k_step_bound_regs(const StepBoundDesc* list, double* out) {
  constexpr int BT = 32 * NW;  // threads
  extern __shared__ __align__(16) double bsm[];
  constexpr int N = R <= 4 ? 4 : 8;  // row sums made at once
  __shared__ double cvs[NW][N];
  __shared__ double red[32];
  __shared__ double corner;  // a(k−1, k−1) before the last reflection
  __shared__ __align__(8) unsigned long long mbar[2];
  __shared__ int gave_up;
  const StepBoundDesc D = list[blockIdx.x / C];
  const int k = D.k, ke = k + (k & 1);
  const int rank = C > 1 ? (int)cluster_rank() : 0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double *d = bsm, *e = d + ke;
  // (product, next column) of every row, by the reflection's parity
  double2* ex[2] = {reinterpret_cast<double2*>(e + ke), reinterpret_cast<double2*>(e + 3 * ke)};
  // Row t of this warp is row(t) of the matrix; lane l holds columns l, l + 32, ….
  auto row = [&](int t) { return rank + C * (warp + NW * t); };
  double a[R][Q];
  double v[Q], w[Q], col[Q];     // by columns: the last reflection, column j
  double rv[R], rw[R], rcol[R];  // the same by rows
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int c = lane + 32 * q;
    v[q] = w[q] = 0.0;
    col[q] = c < k ? 0.5 * (D.G[c] + D.G[(size_t)c * k]) : 0.0;  // column 0
  }
  // G is symmetrised as it is read: G and Gᵀ differ in rounding only.
#pragma unroll
  for (int t = 0; t < R; ++t) {
    const int r = row(t);
    rv[t] = rw[t] = 0.0;
    rcol[t] = r < k ? 0.5 * (D.G[r] + D.G[(size_t)r * k]) : 0.0;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int c = lane + 32 * q;
      const double x = r < k && c < k ? 0.5 * (D.G[r + (size_t)c * k] + D.G[c + (size_t)r * k]) : 0.0;
      a[t][q] = x;
    }
  }
  // Lane l sends row l mod N, to CTA l/N, l/N + 32/N, ….
  constexpr int GR = 32 / N, SEND = (C + GR - 1) / GR;
  const int st = lane & (N - 1), sr = st < R ? row(st) : k;
  unsigned to[SEND][2], tobar[SEND][2], bar[2];
  if (C > 1) {
    if (threadIdx.x == 0) {
      for (int i = 0; i < 2; ++i)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"((unsigned)__cvta_generic_to_shared(&mbar[i])));
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      gave_up = 0;
    }
    for (int i = 0; i < 2; ++i) {
      bar[i] = (unsigned)__cvta_generic_to_shared(&mbar[i]);
      for (int u = 0; u < SEND; ++u) {
        const unsigned rk = (lane / N + GR * u) % C;
        to[u][i] = in_cluster(ex[i] + min(sr, k - 1), rk);
        tobar[u][i] = in_cluster(&mbar[i], rk);
      }
    }
    cluster_sync();
  }
  // A CTA's buffers are free for reflection j + 2 once all its warps have sent j + 1; in
  // a small matrix of a mixed list some warps have no row to send.
  const bool lockstep = C > 1 && k < NW * C;
  for (int j = 0; j + 2 < k; ++j) {
    const int q1 = (j + 1) >> 5, l1 = (j + 1) & 31, b = j & 1;
    double ss = 0.0, x0 = 0.0;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int c = lane + 32 * q;
      const double x = c > j + 1 ? col[q] : 0.0;
      ss = fma(x, x, ss);
      if (q == q1) x0 = col[q];
      if (warp == 0 && c == j) d[j] = col[q];
    }
    x0 = __shfl_sync(0xffffffffu, x0, l1);
    ss = warp_sum(ss);
    // H = I − τ·u·uᵀ, u = (x0 − β, the column below); columns below 1e-145 are dropped
    // (only eigenvalues below −1 matter).  A NaN goes on, and the norm test finds it.
    const bool live = !(ss < 1e-290);
    double beta = x0, tau = 0.0, u0 = 0.0;
    if (live) {
      const double n2 = fma(x0, x0, ss), norm = n2 * rsqrt(n2);
      beta = x0 >= 0.0 ? -norm : norm;
      u0 = x0 - beta;
      tau = 1.0 / fma(norm, fabs(x0), n2);  // 2/uᵀu
    }
    if (threadIdx.x == 0) e[j] = beta;
    double vn[Q], rn[R];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int c = lane + 32 * q;
      vn[q] = c == j + 1 ? u0 : c > j + 1 && live ? col[q] : 0.0;
    }
#pragma unroll
    for (int t = 0; t < R; ++t) rn[t] = row(t) == j + 1 ? u0 : row(t) > j + 1 && live ? rcol[t] : 0.0;
    // A ← A − v·wᵀ − w·vᵀ (the previous reflection), p = A·vn.  Rows up to j are done with
    // and come along (a branch a row costs more).
    double sum[N], odd[R];
#pragma unroll
    for (int t = 0; t < N; ++t) sum[t] = 0.0;
#pragma unroll
    for (int t = 0; t < R; ++t) odd[t] = 0.0;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      if (q < q1) continue;
      const int c = lane + 32 * q;
      double x[R];
#pragma unroll
      for (int t = 0; t < R; ++t)
        x[t] = a[t][q];
#pragma unroll
      for (int t = 0; t < R; ++t) {
        x[t] = fma(-rw[t], v[q], fma(-rv[t], w[q], x[t]));
        a[t][q] = x[t];
        double& acc = q & 1 ? odd[t] : sum[t];
        acc = fma(x[t], vn[q], acc);
      }
      if (q == q1 && lane == l1)
#pragma unroll
        for (int t = 0; t < R; ++t) cvs[warp][t] = x[t];  // column j+1 of the rows
      if (j + 3 == k && c == k - 1)
#pragma unroll
        for (int t = 0; t < R; ++t)
          if (row(t) == k - 1) corner = x[t];
    }
#pragma unroll
    for (int t = 0; t < R; ++t) sum[t] += odd[t];
    const double pr = sum_many<N>(sum);
    __syncwarp();
    const double cv = cvs[warp][st];
    if (C > 1) {
      if (sr < k)
#pragma unroll
        for (int u = 0; u < SEND; ++u)
          if (lane / N + GR * u < C) send_pair(to[u][b], pr, cv, tobar[u][b]);
      if (threadIdx.x == 0)
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar[b]), "r"(16 * k) : "memory");
      const long long t0 = clock64();
      while (!barrier_done(bar[b], (j >> 1) & 1)) {
        if (clock64() - t0 > kBoundCycles || *(volatile int*)&gave_up) {
          gave_up = 1;
          asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(in_cluster(&gave_up, 0u)), "r"(1) : "memory");
          break;
        }
      }
      __syncwarp();
      if (lockstep) cluster_sync();
    } else {
      if (lane < N && sr < k) ex[b][sr] = make_double2(pr, cv);
      __syncthreads();
    }
    double pq[Q], s = 0.0, s2 = 0.0;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int c = lane + 32 * q;
      const double2 pc = c > j && c < k ? ex[b][c] : make_double2(0.0, 0.0);
      pq[q] = pc.x;
      col[q] = pc.y;
      if (q & 1) s2 = fma(pq[q], vn[q], s2);
      else s = fma(pq[q], vn[q], s);
    }
    s = warp_sum(s + s2);
    const double K = 0.5 * tau * tau * s, wj = tau * ex[b][j + 1].x - K * u0;
#pragma unroll
    for (int q = 0; q < Q; ++q) {  // (vn and p are 0 up to column j)
      w[q] = fma(tau, pq[q], -K * vn[q]);
      v[q] = vn[q];
      col[q] = col[q] - vn[q] * wj - u0 * w[q];  // column j+1 after this reflection
    }
#pragma unroll
    for (int t = 0; t < R; ++t) {
      const int r = row(t);
      const double2 pc = r > j && r < k ? ex[b][r] : make_double2(0.0, 0.0);
      rw[t] = fma(tau, pc.x, -K * rn[t]);
      rv[t] = rn[t];
      rcol[t] = pc.y - rn[t] * wj - u0 * rw[t];
    }
  }
  // The corner a(k−1, k−1) is with its owner; rank 0 finishes.
  if (C > 1) {
    __syncthreads();
    if (rank == (k - 1) % C && threadIdx.x == 0) {
      const unsigned to0 = in_cluster(&corner, 0u);
      asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(to0), "d"(corner) : "memory");
    }
    cluster_sync();
  }
  if (warp == 0 && rank == 0) {
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int c = lane + 32 * q;
      if (c == k - 2) d[k - 2] = col[q];
      if (c == k - 1) {
        e[k - 2] = col[q];
        d[k - 1] = corner - 2.0 * v[q] * w[q];
      }
    }
  }
  __syncthreads();
  if (rank == 0) {
    const double b = tridiagonal_bound<BT>(d, e, k, reinterpret_cast<double*>(ex[0]), red);
    if (threadIdx.x == 0) out[blockIdx.x / C] = C > 1 && gave_up ? NAN : b;
  }
  if (C > 1) cluster_sync();  // no CTA leaves while others may still reach it
}

constexpr int kRowWarps = 8, kRows = 4;  // row warps, rows of each
constexpr int kWide = 16;                // CTAs of a cluster

inline size_t bound_smem_doubles(int k) {
  return (size_t)kRowWarps * kRows * (k | 1) + 9ul * (k + (k & 1)) + 1;
}

// The same for larger orders (k ≤ 512): rows in shared memory, eight warps for them and one
// for the vectors; rolled loops.
__global__ void __launch_bounds__(32 * (kRowWarps + 1), 1) k_step_bound_wide(const StepBoundDesc* list, double* out) {
  constexpr int C = kWide, NW = kRowWarps, RPW = kRows, BT = 32 * (NW + 1);
  extern __shared__ __align__(16) double bsm[];
  __shared__ double red[32];
  __shared__ double corner;  // a(k−1, k−1) before the last reflection
  __shared__ __align__(8) unsigned long long mbar[2];
  __shared__ int gave_up;
  const StepBoundDesc D = list[blockIdx.x / C];
  const int k = D.k, lda = k | 1, ke = k + (k & 1);
  const int rank = (int)cluster_rank();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double *d = bsm, *e = d + ke;
  // (product, next column) of every row, by the reflection's parity
  double2* ex[2] = {reinterpret_cast<double2*>(e + ke), reinterpret_cast<double2*>(e + 3 * ke)};
  double* U[2] = {e + 5 * ke, e + 6 * ke};  // reflection vectors by parity, 0 up to column j
  double* W = e + 7 * ke;
  double* A = e + 8 * ke;
  // Row t of row warp q: rank + C·(q + 8t).  G is symmetrised as it is read: G and Gᵀ
  // differ in rounding only.
  for (int i = warp; i < NW * RPW; i += NW + 1) {
    const int r = rank + C * i;
    for (int c = lane; c < k; c += 32)
      A[i * lda + c] = r < k ? 0.5 * (D.G[r + (size_t)c * k] + D.G[c + (size_t)r * k]) : 0.0;
  }
  for (int c = threadIdx.x; c < k; c += BT) {
    U[1][c] = W[c] = 0.0;
    U[0][c] = 0.5 * (D.G[c] + D.G[(size_t)c * k]);  // column 0
  }
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"((unsigned)__cvta_generic_to_shared(&mbar[i])));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    gave_up = 0;
  }
  __syncthreads();
  cluster_sync();  // every CTA is ready to be written to
  // Buffers are free for reflection j + 2 once every CTA has sent its part of j + 1; in a
  // small matrix of a mixed list some have nothing to send.
  const bool lockstep = k < C;
  const unsigned bar[2] = {(unsigned)__cvta_generic_to_shared(&mbar[0]), (unsigned)__cvta_generic_to_shared(&mbar[1])};

  if (warp < NW) {  // ---- rows
    int row[RPW];
#pragma unroll
    for (int t = 0; t < RPW; ++t) row[t] = rank + C * (warp + NW * t);
    // Lane l sends row l mod 4 to the CTAs l/4 and l/4 + 8.
    constexpr int SEND = 2;
    const int st = lane & 3, sr = rank + C * (warp + NW * st);
    double* sa = A + (warp + NW * st) * lda;
    unsigned to[SEND][2], tobar[SEND][2];
    for (int i = 0; i < 2; ++i)
      for (int u = 0; u < SEND; ++u) {
        const unsigned rk = (lane / 4 + 8 * u) % C;
        to[u][i] = in_cluster(ex[i] + min(sr, k - 1), rk);
        tobar[u][i] = in_cluster(&mbar[i], rk);
      }
    for (int j = 0; j + 2 < k; ++j) {
      const int b = j & 1;
      __syncwarp();
      tile64::bar_sync(1, BT);  // the vectors of reflection j are there
      const double *u = U[b], *v = U[b ^ 1];
      double s[RPW] = {};
      // Rows t0 … t0 + NR − 1 are past column j and inside the matrix.
      int t0 = 0, t1 = 0;
#pragma unroll
      for (int t = 0; t < RPW; ++t) t0 += row[t] <= j, t1 += row[t] < k;
      auto pass = [&](auto n) {
        constexpr int NR = decltype(n)::value;
        double nv[NR], nw[NR], acc[NR];
        double* ar[NR];
#pragma unroll
        for (int t = 0; t < NR; ++t) {
          const int r = rank + C * (warp + NW * (t0 + t));
          ar[t] = A + (warp + NW * (t0 + t)) * lda;
          nv[t] = -v[r];
          nw[t] = -W[r];
          acc[t] = 0.0;
        }
        int c = ((j + 1) & ~31) + lane;
        for (; c + 32 < k; c += 64) {  // two columns a lane, all loads first
          const double u0 = u[c], v0 = v[c], w0 = W[c], u1 = u[c + 32], v1 = v[c + 32], w1 = W[c + 32];
          double x[NR], y[NR];
#pragma unroll
          for (int t = 0; t < NR; ++t) x[t] = ar[t][c], y[t] = ar[t][c + 32];
#pragma unroll
          for (int t = 0; t < NR; ++t) {
            x[t] = fma(nw[t], v0, fma(nv[t], w0, x[t]));
            y[t] = fma(nw[t], v1, fma(nv[t], w1, y[t]));
            ar[t][c] = x[t];
            ar[t][c + 32] = y[t];
            acc[t] = fma(y[t], u1, fma(x[t], u0, acc[t]));
          }
        }
        if (c < k) {
          const double u0 = u[c], v0 = v[c], w0 = W[c];
#pragma unroll
          for (int t = 0; t < NR; ++t) {
            const double x = fma(nw[t], v0, fma(nv[t], w0, ar[t][c]));
            ar[t][c] = x;
            acc[t] = fma(x, u0, acc[t]);
          }
        }
#pragma unroll
        for (int t = 0; t < NR; ++t)
#pragma unroll
          for (int q = 0; q < RPW; ++q)
            if (q == t0 + t) s[q] = acc[t];
      };
      switch (t1 - t0) {
        case 4: pass(std::integral_constant<int, 4>()); break;
        case 3: pass(std::integral_constant<int, 3>()); break;
        case 2: pass(std::integral_constant<int, 2>()); break;
        case 1: pass(std::integral_constant<int, 1>()); break;
      }
      const double p = sum_many<RPW>(s);
      __syncwarp();
      const double cv = sa[j + 1];  // the row's entry of column j + 1
      if (sr < k)
#pragma unroll
        for (int q = 0; q < SEND; ++q) send_pair(to[q][b], p, cv, tobar[q][b]);
      if (lockstep) cluster_sync();
    }
  } else {  // ---- vectors
    // Reflection j: H = I − τ·u·uᵀ, u = (x0 − β, the column below), from the sum ss of
    // the squares below x0; columns below 1e-145 are dropped (only eigenvalues below −1
    // matter).  A NaN goes on, and the norm test finds it.
    double tau = 0.0, u0 = 0.0;
    auto reflect = [&](int j, double x0, double ss) {
      double* u = U[j & 1];
      double beta = x0;
      tau = u0 = 0.0;
      if (!(ss < 1e-290)) {
        const double n2 = fma(x0, x0, ss), norm = n2 * rsqrt(n2);
        beta = x0 >= 0.0 ? -norm : norm;
        u0 = x0 - beta;
        tau = 1.0 / fma(norm, fabs(x0), n2);  // 2/uᵀu
      } else {
        for (int c = j + 2 + lane; c < k; c += 32) u[c] = 0.0;
      }
      if (lane == 0) {
        u[j + 1] = u0;
        e[j] = beta;
      }
      __syncwarp();
    };
    {
      double ss = 0.0;
      for (int c = 2 + lane; c < k; c += 32) ss = fma(U[0][c], U[0][c], ss);
      const double x0 = U[0][1];
      if (lane == 0) {
        d[0] = U[0][0];
        U[0][0] = 0.0;
      }
      reflect(0, x0, warp_sum(ss));
    }
    for (int j = 0; j + 2 < k; ++j) {
      const int b = j & 1;
      __syncwarp();
      tile64::bar_sync(1, BT);
      if (lane == 0)
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar[b]), "r"(16 * k) : "memory");
      const long long t0 = clock64();
      while (!barrier_done(bar[b], (j >> 1) & 1)) {
        if (clock64() - t0 > kBoundCycles || *(volatile int*)&gave_up) {
          gave_up = 1;
          asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(in_cluster(&gave_up, 0u)), "r"(1) : "memory");
          break;
        }
      }
      __syncwarp();
      if (lockstep) cluster_sync();
      const double* u = U[b];
      double* un = U[b ^ 1];
      const double2* q = ex[b];
      const int c0 = j & ~31;
      double s = 0.0;
#pragma unroll 4
      for (int c = c0 + lane; c < k; c += 32)
        if (c > j) s = fma(q[c].x, u[c], s);
      s = warp_sum(s);
      const double K = 0.5 * tau * tau * s, wj = tau * q[j + 1].x - K * u0, uj = u0;
      double ss = 0.0, x0 = 0.0;
#pragma unroll 4
      for (int c = c0 + lane; c < k; c += 32) {
        const double2 pc = q[c];
        const double uc = u[c];
        const double w = c > j ? fma(tau, pc.x, -K * uc) : 0.0;
        double x = pc.y - uc * wj - uj * w;  // column j + 1 after this reflection
        W[c] = w;
        if (c == j + 1) d[j + 1] = x;
        if (c == j + 2) x0 = x;
        if (c <= j + 1) x = 0.0;
        un[c] = x;
        if (c > j + 2) ss = fma(x, x, ss);
      }
      x0 = __shfl_sync(0xffffffffu, x0, (j + 2) & 31);
      ss = warp_sum(ss);
      __syncwarp();
      if (j + 3 < k) reflect(j + 1, x0, ss);
      else if (lane == 0) e[k - 2] = x0;
    }
  }
  // The corner is with its owner; rank 0 finishes.
  __syncthreads();
  if (threadIdx.x == 0 && rank == (k - 1) % C) {
    const double x = A[((k - 1) / C) * lda + k - 1];
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(in_cluster(&corner, 0u)), "d"(x) : "memory");
  }
  cluster_sync();
  __syncthreads();
  if (threadIdx.x == 0) d[k - 1] = corner - 2.0 * U[(k - 3) & 1][k - 1] * W[k - 1];
  __syncthreads();
  if (rank == 0) {
    const double b = tridiagonal_bound<BT>(d, e, k, reinterpret_cast<double*>(ex[0]), red);
    if (threadIdx.x == 0) out[blockIdx.x / C] = gave_up ? NAN : b;
  }
  cluster_sync();  // no CTA leaves while others may still reach it
}

// Clusters of 16 are not portable and need the opt-in (idempotent, per device).
template <class Kern>
void ensure_cluster16(Kern kern) {
  SDPX_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
}

struct ClusterConfig {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  template <class Kern>
  ClusterConfig(Kern kern, int clusters, int C, int threads, size_t smem, cudaStream_t st) {
    if (C > 8) ensure_cluster16(kern);
    ensure_smem(kern, smem);
    cfg.gridDim = dim3(clusters * C);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = C;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
  }
  ClusterConfig(const ClusterConfig&) = delete;
};

// The kernel for orders up to kmax, and f(kernel, CTAs of a cluster, threads, shared bytes).
// Cluster and warps by the largest order: every warp repeats the vector work, so few
// warps, and few rows in each, beat a small cluster's shorter barrier.  Cycles measured
// (cluster × warps): k = 30  63e3 (1×8), 66e3 (4×4); 61  153e3 (1×8), 131e3 (4×4), 145e3
// (8×4); 100  291e3 (4×8), 243e3 (8×4); 200  746e3 (8×8), 744e3 (8×4), 624e3 (16×4).
constexpr int kOrderLimits[] = {32, 64, 128, 224, 448};
template <int C, int NW, int Q, int R, class F>
auto with_regs(int kmax, F f) {
  static_assert(32 * Q <= R * C * NW, "every row has a place");
  return f(k_step_bound_regs<C, NW, Q, R>, C, 32 * NW, (6ul * (kmax + (kmax & 1)) + 1) * sizeof(double));
}
template <class F>
auto with_kernel(int kmax, F f) {
  if (kmax <= kOrderLimits[0]) return with_regs<1, 8, 1, 4>(kmax, f);
  if (kmax <= kOrderLimits[1]) return with_regs<4, 4, 2, 4>(kmax, f);
  if (kmax <= kOrderLimits[2]) return with_regs<8, 4, 4, 4>(kmax, f);
  if (kmax <= kOrderLimits[3]) return with_regs<16, 4, 7, 4>(kmax, f);
  return f(k_step_bound_wide, kWide, 32 * (kRowWarps + 1), bound_smem_doubles(kmax) * sizeof(double));
}

}  // namespace

// A part of a GPU may have no place for the larger clusters.
int step_bound_max_order() {
  static std::atomic<int> known[64];
  int dev = 0;
  SDPX_CUDA(cudaGetDevice(&dev));
  const bool keep = dev >= 0 && dev < 64;
  int order = keep ? known[dev].load(std::memory_order_relaxed) : 0;
  if (order) return order;
  for (int limit : kOrderLimits) {
    const bool runs = with_kernel(limit, [](auto kern, int C, int threads, size_t smem) {
      const ClusterConfig q(kern, 1, C, threads, smem, nullptr);
      int places = 0;
      const bool ok = cudaOccupancyMaxActiveClusters(&places, kern, &q.cfg) == cudaSuccess && places > 0;
      if (!ok) cudaGetLastError();
      return ok;
    });
    if (!runs) break;
    order = limit;
  }
  if (order == 0) order = 2;  // none (every order that needs the kernel is larger)
  if (keep) known[dev].store(order, std::memory_order_relaxed);
  return order;
}

void step_bounds(const StepBoundDesc* d_list, int n, int kmax, double* out, cudaStream_t st) {
  if (n <= 0) return;
  if (kmax > step_bound_max_order()) throw std::invalid_argument("step_bounds: order too large");
  with_kernel(kmax, [&](auto kern, int C, int threads, size_t smem) {
    const ClusterConfig q(kern, n, C, threads, smem, st);
    SDPX_CUDA(cudaLaunchKernelEx(&q.cfg, kern, d_list, out));
    SDPX_LAUNCH_CHECK();
  });
}

}  // namespace sdpx
