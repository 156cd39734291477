// Fraction-to-boundary bounds of M + t·dM from eigenvalues: with M = L·Lᵀ and
// G = L⁻¹·dM·L⁻ᵀ, the largest t ≤ 1 that keeps M + t·dM positive semidefinite is
// t* = −1/λ_min(G), or 1 when λ_min(G) ≥ −1 — the value that the 64-step bisection
// of Cholesky tests (`fraction_to_boundary_bound!`, src/kernels/generic.jl:350-422)
// approaches from below, up to the rounding of its tests.
//
// λ_min comes from a Householder tridiagonalisation and a Sturm-count
// multisection.  One cluster of C CTAs per matrix holds it in shared memory, rows
// dealt out cyclically.  What bounds it is the chain of k reflections, so each has
// one pass over the rows and one cluster barrier: the pass applies the previous
// reflection's rank-2 update and multiplies with this reflection's vector, and
// the barrier exchanges the product together with the next column, from which every
// CTA forms the next vector for itself.
//
// Against the bisection's 10 to 15 rounds of batched Cholesky tests (each with its
// uploads, factorizations and read-back), both sides of one iterate on the B200:
//   block orders       12        200       400 + 200
//   bisection rounds   0.45      2.0       6.3 ms
//   here               0.021     0.48      1.21 ms
// and within 4e-15 of −1/λ_min in 64 bits where the bisection is, iterates of κ = 100.
#include "step_bound.h"
#include "lambda_bound.cuh"

namespace sdpx {
namespace {

constexpr int BT = 512;  // threads

__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// A store to the same shared location of CTA `rank` of the cluster.
__device__ __forceinline__ void st_cluster(double* p, unsigned rank, double v) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(p);
  unsigned b;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(b) : "r"(a), "r"(rank));
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(b), "d"(v) : "memory");
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Σ over the CTA; one barrier (two alternating scratch rows, so no second one).
__device__ __forceinline__ double bsum(double v, double* red) {
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = 0.0;
#pragma unroll
  for (int w = 0; w < BT / 32; w += 2) {
    const double2 u = *reinterpret_cast<const double2*>(red + w);
    s += u.x + u.y;
  }
  return s;
}

__host__ __device__ inline size_t bound_smem_doubles(int k, int C) {
  const int lda = k | 1, rows = (k + C - 1) / C;
  return (size_t)rows * lda + 9ul * (k + (k & 1)) + 1;
}

// out[q] = bound of matrix q of the list (k ≥ 3).
template <int C>
__global__ void __launch_bounds__(BT, 1) k_step_bound(const StepBoundDesc* list, double* out) {
  extern __shared__ __align__(16) double bsm[];
  __shared__ __align__(16) double red[2][BT / 32];
  __shared__ double dlast;
  const StepBoundDesc Q = list[blockIdx.x / C];
  const int k = Q.k, lda = k | 1, ke = k + (k & 1);
  const int rank = C > 1 ? (int)cluster_rank() : 0;
  const int me = threadIdx.x, lane = me & 31, warp = me >> 5;
  const int nrow = (k - rank + C - 1) / C;  // rows rank, rank + C, …
  double* v = bsm;
  double *w = v + ke, *vn = w + ke, *d = vn + ke, *e = d + ke;
  double* pb[2] = {e + ke, e + 2 * ke};
  double* cb[2] = {e + 3 * ke, e + 4 * ke};
  double* A = e + 5 * ke;
  // G is symmetrised as it is read: G and Gᵀ differ in rounding only.
  for (int i = warp; i < nrow; i += BT / 32) {
    const int r = rank + C * i;
    for (int c = lane; c < k; c += 32)
      A[i * lda + c] = 0.5 * (Q.G[r + (size_t)c * k] + Q.G[c + (size_t)r * k]);
  }
  for (int i = threadIdx.x; i < k; i += BT) {
    cb[1][i] = 0.5 * (Q.G[i] + Q.G[(size_t)i * k]);  // column 0
    v[i] = w[i] = 0.0;
  }
  __syncthreads();
  if (C > 1) cluster_sync();  // every CTA runs before its shared memory is written from outside
  for (int j = 0; j + 2 < k; ++j) {
    // col: column j of the current matrix (rows ≥ j); thread i owns entry i of every vector
    const double* col = cb[(j + 1) & 1];
    double *p = pb[j & 1], *cn = cb[j & 1];
    const double ci = me > j + 1 && me < k ? col[me] : 0.0;
    const double ss = bsum(ci * ci, red[0]);
    const double x0 = col[j + 1];
    double beta = x0, tau = 0.0, scale = 0.0;
    if (ss != 0.0) {  // (NaN: goes on, and the norm test below finds it)
      const double norm = sqrt(x0 * x0 + ss);
      beta = x0 >= 0.0 ? -norm : norm;
      tau = (beta - x0) / beta;
      scale = 1.0 / (x0 - beta);
    }
    if (me > j && me < k) vn[me] = me == j + 1 ? 1.0 : ci * scale;
    if (me == 0) {
      d[j] = col[j];
      e[j] = beta;
    }
    __syncthreads();
    // rows r > j: A ← A − v·wᵀ − w·vᵀ (the previous reflection), p = A·vn
    int i0 = j + 1 > rank ? (j + 1 - rank + C - 1) / C : 0;
    for (int ib = i0 + warp * 2; ib < nrow; ib += 2 * (BT / 32)) {
      const int r0 = rank + C * ib;
      const bool two = ib + 1 < nrow;
      const int r1 = two ? r0 + C : r0;
      double *a0 = A + ib * lda, *a1 = two ? a0 + lda : a0;
      const double v0 = v[r0], w0 = w[r0], v1 = v[r1], w1 = w[r1];
      double s0 = 0.0, s1 = 0.0;
      for (int c = j + 1 + lane; c < k; c += 32) {
        const double vc = v[c], wc = w[c], nc = vn[c];
        const double x = fma(-w0, vc, fma(-v0, wc, a0[c]));
        const double y = fma(-w1, vc, fma(-v1, wc, a1[c]));
        a0[c] = x;
        if (two) a1[c] = y;
        s0 = fma(x, nc, s0);
        s1 = fma(y, nc, s1);
      }
      s0 = warp_sum(s0);
      s1 = warp_sum(s1);
      __syncwarp();
      // lanes 0 … C−1 send (p, column j+1) of row r0, lanes 16 … of r1
      const int u = lane & 15, r = lane < 16 ? r0 : r1;
      if (u < C && (lane < 16 || two)) {
        const double pv = lane < 16 ? s0 : s1, cv = lane < 16 ? a0[j + 1] : a1[j + 1];
        if (C > 1) {
          st_cluster(p + r, (unsigned)u, pv);
          st_cluster(cn + r, (unsigned)u, cv);
          if (j + 3 == k && r == k - 1) st_cluster(&dlast, (unsigned)u, lane < 16 ? a0[k - 1] : a1[k - 1]);
        } else {
          p[r] = pv;
          cn[r] = cv;
          if (j + 3 == k && r == k - 1) dlast = lane < 16 ? a0[k - 1] : a1[k - 1];
        }
      }
    }
    if (C > 1) cluster_sync();
    else __syncthreads();
    const bool mine = me > j && me < k;
    const double vi = mine ? vn[me] : 0.0, pi = mine ? p[me] : 0.0;
    const double s = bsum(pi * vi, red[1]);
    const double K = 0.5 * tau * tau * s, wj = tau * p[j + 1] - K;
    if (mine) {
      const double wi = fma(tau, pi, -K * vi);
      w[me] = wi;
      v[me] = vi;
      cn[me] = cn[me] - vi * wj - wi;  // column j+1 after this reflection
    }
  }
  __syncthreads();
  if (rank == 0) {
    const double* col = cb[(k - 1) & 1];
    if (threadIdx.x == 0) {
      d[k - 2] = col[k - 2];
      e[k - 2] = col[k - 1];
      d[k - 1] = dlast - 2.0 * v[k - 1] * w[k - 1];
    }
    __syncthreads();
    // Gershgorin bounds
    double lo = INFINITY, hi = INFINITY, nrm = 0.0;
    for (int i = threadIdx.x; i < k; i += BT) {
      const double r = (i > 0 ? fabs(e[i - 1]) : 0.0) + (i + 1 < k ? fabs(e[i]) : 0.0);
      lo = fmin(lo, d[i] - r);
      hi = fmin(hi, d[i]);
      const double n = fabs(d[i]) + r;
      nrm = n == n ? fmax(nrm, n) : INFINITY;
    }
    lo = -block_max(-lo, red[0]);
    hi = -block_max(-hi, red[0]);
    nrm = block_max(nrm, red[0]);
    if (!(nrm < 1e300)) {
      if (threadIdx.x == 0) out[blockIdx.x / C] = 0.0;  // non-finite direction: no step
    } else if (lo >= -1.0) {
      if (threadIdx.x == 0) out[blockIdx.x / C] = 1.0;
    } else {
      const double f = 1.0 / nrm;  // nrm ≥ |lo| > 1
      double *ds = pb[1], *es = cb[0];
      for (int i = threadIdx.x; i < k; i += BT) {
        ds[i] = d[i] * f;
        es[i] = i + 1 < k ? fmax(e[i] * f * (e[i] * f), 1e-36) : 0.0;
      }
      __syncthreads();
      double b = 1.0;
      // thread 0 at −1: does the full step stay inside?
      if (__syncthreads_or(threadIdx.x == 0 && minors_below(ds, es, k, -f) > 0)) {
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
        b = bound_from_below(l / f);
      }
      if (threadIdx.x == 0) out[blockIdx.x / C] = b;
    }
  }
  if (C > 1) cluster_sync();  // no CTA leaves while others may still reach it
}

// Cluster size for order k: one CTA up to 64 rows, then enough for rows to go
// round quickly, and for the matrix to fit.
int cluster_for(int k) {
  for (int C : {1, 2, 4, 8}) {
    if (k > 64 * C && C < 8) continue;
    if (bound_smem_doubles(k, C) * sizeof(double) <= 225 * 1024) return C;
  }
  return 0;
}

template <int C>
void launch(const StepBoundDesc* d_list, int n, int kmax, double* out, cudaStream_t st) {
  const size_t smem = bound_smem_doubles(kmax, C) * sizeof(double);
  ensure_smem(k_step_bound<C>, smem);
  if (C == 1) {
    k_step_bound<C><<<n, BT, smem, st>>>(d_list, out);
  } else {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(n * C);
    cfg.blockDim = dim3(BT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = C;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    SDPX_CUDA(cudaLaunchKernelEx(&cfg, k_step_bound<C>, d_list, out));
  }
  SDPX_LAUNCH_CHECK();
}

}  // namespace

bool step_bound_fits(int k) { return k >= 3 && k <= BT && cluster_for(k) != 0; }

void step_bounds(const StepBoundDesc* d_list, int n, int kmax, double* out, cudaStream_t st) {
  if (n <= 0) return;
  switch (cluster_for(kmax)) {
    case 1: return launch<1>(d_list, n, kmax, out, st);
    case 2: return launch<2>(d_list, n, kmax, out, st);
    case 4: return launch<4>(d_list, n, kmax, out, st);
    case 8: return launch<8>(d_list, n, kmax, out, st);
    default: throw std::invalid_argument("step_bounds: order too large");
  }
}

}  // namespace sdpx
