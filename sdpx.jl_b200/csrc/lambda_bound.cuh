// Fraction-to-boundary bound of I + t·G from the smallest eigenvalue of G, orders up
// to 64 (the batched engine's instances, small blocks of a single solve): Householder
// tridiagonalisation by 128 threads and a Sturm-count multisection, everything in
// shared memory.
//
// What bounds it is the chain of reflections, so each is cut to two barriers of its
// 128 threads: two threads a row apply the previous reflection's rank-2 update and
// multiply with this reflection's vector in one pass, and the two inner products of a
// reflection are formed by every warp for itself.
#pragma once
#include "tile64.cuh"

namespace sdpx {

struct LambdaScratch {
  double col[2][64], p[64], cn[64], v[64], w[64], d[64], e[64];
};

// Number of eigenvalues below x of the tridiagonal (d, e2 = squared off-diagonal,
// all scaled to norm ≤ 1): sign changes of the leading minors of T − x·I by their
// three-term recurrence, one fma a row in the chain, rescaled every eight rows (within
// which two consecutive minors grow at most 3⁸-fold and shrink to 1e-288 at worst),
// the next eight rows' entries on their way.  e2 ≥ 1e-36 keeps two consecutive minors
// from vanishing together (a change of T of 1e-18 of its norm).
__device__ __forceinline__ int minors_below(const double* d, const double* e2, int k, double x) {
  double pp = 1.0, p = d[0] - x;
  int neg = __double2hiint(p) < 0;
  int i = 1;
  constexpr int U = 8;
  double di[U], ei[U];
  if (i + U <= k) {
#pragma unroll
    for (int u = 0; u < U; ++u) di[u] = d[i + u], ei[u] = e2[i + u - 1];
  }
  for (; i + U <= k; i += U) {
    double dn[U], en[U];
    const bool more = i + 2 * U <= k;
#pragma unroll
    for (int u = 0; u < U; ++u) dn[u] = more ? d[i + U + u] : 0.0, en[u] = more ? e2[i + U + u - 1] : 0.0;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const double q = fma(di[u] - x, p, -ei[u] * pp);
      neg += (unsigned)(__double2hiint(q) ^ __double2hiint(p)) >> 31;
      pp = p;
      p = q;
    }
    const int ex = max((__double2hiint(p) >> 20) & 2047, (__double2hiint(pp) >> 20) & 2047);
    const double f = __hiloint2double(min(2046, max(1, 2046 - ex)) << 20, 0);  // ≈ 2^(1023−ex)
    p *= f;
    pp *= f;
#pragma unroll
    for (int u = 0; u < U; ++u) di[u] = dn[u], ei[u] = en[u];
  }
  for (; i < k; ++i) {
    const double q = fma(d[i] - x, p, -e2[i - 1] * pp);
    neg += (unsigned)(__double2hiint(q) ^ __double2hiint(p)) >> 31;
    pp = p;
    p = q;
  }
  return neg;
}

// The bound from a lower bound l of λ_min: from below, as the bisection's last passing
// trial is; l holds up to its last ulp and the quotient is rounded once: two ulps.
__device__ __forceinline__ double bound_from_below(double l) {
  return fmin(1.0, __longlong_as_double(__double_as_longlong(-1.0 / l) - 2));
}

// min(1, −1/λ_min) of the symmetric G (tile of leading dimension FLD, k ≤ 64, both
// triangles; overwritten), 0 when G is not finite.  Called by 128 threads (tid) that
// share named barrier `bar`; the same value in all of them.
__device__ __forceinline__ double lambda_bound_64(double* G, int k, LambdaScratch& s, int tid, int bar) {
  constexpr int LD = tile64::FLD;
  const int lane = tid & 31, r = tid >> 1, q = tid & 1;
  auto sync = [&]() {
    __syncwarp();
    tile64::bar_sync(bar, 128);
  };
  if (tid < k) {
    s.col[0][tid] = G[tid];
    s.v[tid] = s.w[tid] = 0.0;
  }
  sync();
  for (int j = 0; j + 2 < k; ++j) {
    const double* col = s.col[j & 1];  // column j of the current matrix, rows ≥ j
    double* next = s.col[(j + 1) & 1];
    const int i0 = lane, i1 = lane + 32;
    const double c0 = i0 > j + 1 && i0 < k ? col[i0] : 0.0, c1 = i1 > j + 1 && i1 < k ? col[i1] : 0.0;
    const double x0 = col[j + 1];
    const double ss = warp_sum(fma(c0, c0, c1 * c1));
    double beta = x0, tau = 0.0, scale = 0.0;
    if (ss != 0.0) {  // (NaN goes on; the norm test below finds it)
      const double norm = sqrt(fma(x0, x0, ss));
      beta = x0 >= 0.0 ? -norm : norm;
      tau = (beta - x0) / beta;
      scale = 1.0 / (x0 - beta);
    }
    if (tid == 0) {
      s.d[j] = col[j];
      s.e[j] = beta;
    }
    // rows r > j: G ← G − v·wᵀ − w·vᵀ (the previous reflection), p = G·vn
    double t0 = 0.0, t1 = 0.0;
    if (r > j && r < k) {
      const double vr = s.v[r], wr = s.w[r];
      int c = j + 1 + ((j + 1 + q) & 1);  // c ≡ q (mod 2)
      for (; c + 2 < k; c += 4) {
        const double a = fma(-wr, s.v[c], fma(-vr, s.w[c], G[c * LD + r]));
        const double b = fma(-wr, s.v[c + 2], fma(-vr, s.w[c + 2], G[(c + 2) * LD + r]));
        G[c * LD + r] = a;
        G[(c + 2) * LD + r] = b;
        if (c == j + 1) s.cn[r] = a;
        t0 = fma(a, c == j + 1 ? 1.0 : col[c] * scale, t0);
        t1 = fma(b, col[c + 2] * scale, t1);
      }
      if (c < k) {
        const double a = fma(-wr, s.v[c], fma(-vr, s.w[c], G[c * LD + r]));
        G[c * LD + r] = a;
        if (c == j + 1) s.cn[r] = a;
        t0 = fma(a, c == j + 1 ? 1.0 : col[c] * scale, t0);
      }
    }
    t0 += t1;
    t0 += __shfl_xor_sync(0xffffffffu, t0, 1);
    if (q == 0 && r > j && r < k) s.p[r] = t0;
    sync();
    const double v0 = i0 == j + 1 ? 1.0 : c0 * scale, v1 = i1 == j + 1 ? 1.0 : c1 * scale;
    const double p0 = i0 > j && i0 < k ? s.p[i0] : 0.0, p1 = i1 > j && i1 < k ? s.p[i1] : 0.0;
    const double pv = warp_sum(fma(p0, v0, p1 * v1));
    const double K = 0.5 * tau * tau * pv, wj = tau * s.p[j + 1] - K;
    if (tid < 64 && tid > j && tid < k) {  // thread i < 64 owns entry i
      const double vi = tid < 32 ? v0 : v1, pi = tid < 32 ? p0 : p1;
      const double wi = fma(tau, pi, -K * vi);
      s.w[tid] = wi;
      s.v[tid] = vi;
      next[tid] = s.cn[tid] - vi * wj - wi;  // column j+1 after this reflection
    }
    sync();
  }
  if (tid == 0) {
    const double* col = s.col[(k - 2) & 1];
    if (k >= 2) {
      s.d[k - 2] = col[k - 2];
      s.e[k - 2] = col[k - 1];
      s.d[k - 1] = G[(k - 1) * LD + k - 1] - 2.0 * s.v[k - 1] * s.w[k - 1];
    } else {
      s.d[0] = G[0];
    }
  }
  sync();
  // Gershgorin bounds, in every warp alike
  double lo = INFINITY, hi = INFINITY, nrm = 0.0;
  for (int i = lane; i < k; i += 32) {
    const double rad = (i > 0 ? fabs(s.e[i - 1]) : 0.0) + (i + 1 < k ? fabs(s.e[i]) : 0.0);
    lo = fmin(lo, s.d[i] - rad);
    hi = fmin(hi, s.d[i]);
    const double n = fabs(s.d[i]) + rad;
    nrm = n == n ? fmax(nrm, n) : INFINITY;
  }
  lo = warp_min(lo);
  hi = warp_min(hi);
  nrm = warp_max(nrm);
  if (!(nrm < 1e300)) return 0.0;
  if (lo >= -1.0) return 1.0;
  const double f = 1.0 / nrm;  // nrm ≥ |lo| > 1
  sync();
  if (tid < k) {
    s.v[tid] = s.d[tid] * f;
    s.w[tid] = tid + 1 < k ? fmax(s.e[tid] * f * (s.e[tid] * f), 1e-36) : 0.0;
  }
  sync();
  if (minors_below(s.v, s.w, k, -f) == 0) return 1.0;  // the full step stays inside
  double l = lo * f - 1e-15, h = fmin(hi * f + 1e-15, -f);
  for (int round = 0; round < 14; ++round) {
    const double step = (h - l) / 129.0;
    const bool clear = minors_below(s.v, s.w, k, l + step * (tid + 1)) == 0;
    // counts are monotone: the first m shifts have no eigenvalue below them
    const int mine = __popc(__ballot_sync(0xffffffffu, clear));
    if (lane == 0) s.p[tid >> 5] = (double)mine;
    sync();
    const int m = (int)(s.p[0] + s.p[1] + s.p[2] + s.p[3]);
    sync();
    const double nl = m > 0 ? l + step * m : l, nh = m < 128 ? l + step * (m + 1) : h;
    l = nl;
    h = nh;
    if (h - l <= 2e-16 * fabs(l)) break;
  }
  return bound_from_below(l / f);
}

}  // namespace sdpx
