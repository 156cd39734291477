// FP64 Cholesky of a few matrices in one launch, ordered by tile flags instead
// of grid barriers or kernel boundaries (potrf_flow, chol.h), and the inverses
// of the diagonal tiles of a factor.
//
// What bounds it: the pivot chain.  A 64-column panel costs 64 dependent
// square roots and reciprocals (about 150 cycles each with the products that
// follow) whatever the GPU's width, and the flops of the orders used here (blocks
// and trials of a few hundred, m ≤ 3000 for the Schur and normal matrices) are
// small beside it.  So one CTA
// per matrix runs the chain alone — factor tile (j,j), solve tile (j+1,j)
// against it, update tile (j+1,j+1) with that, all from shared memory and
// registers — and the other CTAs of the matrix keep every other tile up to date
// (left-looking: a CTA holds its tile in registers over all panels), so the
// chain never waits for a whole panel.  Tiles are published with a
// release store of a flag each and read after an acquire load.
//
// The arithmetic of every element is that of the panel-by-panel factorization:
// per 64-wide panel its products summed from zero in increasing column order
// and subtracted once, inside a panel subtracted one by one, columns scaled by
// the reciprocal pivot (LAPACK's dpotf2).
//
// Eight warps of a CTA compute; warp w owns rows 8w … 8w+7 of a 64×64 tile (a
// strip; as DMMA accumulators lane 4g+t holds row g, columns 8f+2t and 8f+2t+1 of
// fragment f).  In the chain's CTA four more warps do the global side: they store
// and publish finished tiles and fetch the next two, so that a store's fence
// (about 1 µs) and a load's latency are not in the chain.  The chain's loops are
// rolled and work from shared memory: unrolled over a strip in registers the factor
// of a tile took 24.5 k cycles instead of 18 k, most of it fetching instructions.
#include "chol.h"
#include "tile64.cuh"

namespace sdpx {
using namespace tile64;
namespace {

constexpr int FIO = 128;      // threads of the chain's global side
constexpr int kTile = FB * FLD;
constexpr size_t kFlowSmem = sizeof(double) * 3 * kTile;
constexpr unsigned kSpinLimit = 1u << 22;  // polls of ≥ 0.3 µs: over a second

// Named barriers (0 is __syncthreads): 1–4 the block factor, then
enum { kBarCompute = 5, kBarIo, kBarFactored, kBarSolved, kBarUpdated, kBarLoaded, kBarStored, kBarTasks };

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(unsigned* p, unsigned v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// Barrier of the computing threads that also returns whether ok held in all.  (All of them
// execute it whatever thread 0 did before, as with __syncthreads.)
__device__ __forceinline__ bool compute_and(int ok) {
  int r;
  asm volatile(
      "{\n.reg .pred p, q;\nsetp.ne.s32 p, %1, 0;\nbar.red.and.pred q, %2, %3, p;\nselp.s32 %0, 1, 0, q;\n}"
      : "=r"(r)
      : "r"(ok), "n"((int)kBarCompute), "n"((int)FT)
      : "memory");
  return r != 0;
}
__device__ __forceinline__ void compute_sync() { bar_sync(kBarCompute, FT); }

// Flag words of one matrix of nt tile rows: ready[i·nt + j] (tile final),
// c1[j] (tile (j+1,j) updated by the panels before j), c2[j] (tile (j,j) updated
// by the panels before j−1), then the failure and the timeout.  Epoch 0, which no launch
// has: the matrix has one CTA and no flags.
struct Flags {
  unsigned *ready, *c1, *c2, *stop;
  unsigned epoch;  // the value that marks
  int nt;
  __device__ Flags(unsigned* base, int n, unsigned ep)
      : ready(base), c1(base + n * n), c2(c1 + n), stop(c2 + n), epoch(ep), nt(n) {}
  __device__ bool alone() const { return epoch == 0; }
  __device__ unsigned* tile(int i, int j) const { return ready + i * nt + j; }
  __device__ bool set(const unsigned* f) const { return ld_acquire(f) == epoch; }
  __device__ void mark(unsigned* f) const { st_release(f, epoch); }
};

// One thread waits for a and b; false when the matrix failed or a wait timed out.
__device__ __forceinline__ bool poll_flags(const Flags& F, const unsigned* a, const unsigned* b) {
  unsigned spins = 0;
  while (!F.set(a) || !F.set(b)) {
    if (F.set(F.stop) || F.set(F.stop + 1)) return false;
    if (++spins > kSpinLimit) {
      atomicExch(F.stop + 1, F.epoch);
      return false;
    }
  }
  return true;
}

// Copies of the h×w tile at (r0, c0) between global memory and shared T by NTH
// threads, this one being `tid`; coalesced down the columns, zeros outside the
// tile.  Loads go to L2: another SM may have written the tile after this SM last
// read its lines.  lower: rows ≥ columns only (a diagonal tile's upper part
// belongs to zero_upper_part).
template <int NTH>
__device__ __forceinline__ void load_tile(double* T, const MatDesc<double>& M, int r0, int c0, int h, int w,
                                          int tid) {
  const int r = tid & 63, cb = tid >> 6;
  const double* p = M.a + (size_t)c0 * M.ld + r0 + r;
  constexpr int PER = FB * FB / NTH, BATCH = 16;
#pragma unroll 1
  for (int k0 = 0; k0 < PER; k0 += BATCH) {
    double v[BATCH];
#pragma unroll
    for (int k = 0; k < BATCH; ++k) {
      const int c = cb + (k0 + k) * (NTH / 64);
      v[k] = (r < h && c < w) ? __ldcg(p + (size_t)c * M.ld) : 0.0;
    }
#pragma unroll
    for (int k = 0; k < BATCH; ++k) T[(cb + (k0 + k) * (NTH / 64)) * FLD + r] = v[k];
  }
}
template <int NTH>
__device__ __forceinline__ void store_tile(const double* T, const MatDesc<double>& M, int r0, int c0, int h,
                                           int w, bool lower, int tid) {
  const int r = tid & 63, cb = tid >> 6;
  double* p = M.a + (size_t)c0 * M.ld + r0 + r;
#pragma unroll 8
  for (int k = 0; k < FB * FB / NTH; ++k) {
    const int c = cb + k * (NTH / 64);
    if (r < h && c < w && (!lower || r >= c)) __stcg(p + (size_t)c * M.ld, T[c * FLD + r]);
  }
}

// x −= (rows of La)·(rows of Lb)ᵀ over one 64-wide panel, the products summed from
// zero first.
__device__ __forceinline__ void strip_update(double (&x)[8][2], const double* La, const double* Lb) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, r = (threadIdx.x >> 5) * 8 + g;
  double acc[8][2] = {};
#pragma unroll 2
  for (int kk = 0; kk < FB; kk += 4) {
    const double av = La[(kk + t) * FLD + r];
    const double* lb = Lb + (kk + t) * FLD + g;
#pragma unroll
    for (int f = 0; f < 8; ++f) mma8(acc[f][0], acc[f][1], av, lb[8 * f]);
  }
#pragma unroll
  for (int f = 0; f < 8; ++f) {
    x[f][0] -= acc[f][0];
    x[f][1] -= acc[f][1];
  }
}

// Y −= X·Xᵀ on the lower 8×8 blocks, the products summed from zero first.  Warps w
// and w+4 share a quarter of the SM: strips w and 7−w give each quarter 9 blocks,
// two of a strip's blocks at a time to cover the pipe's latency.
__device__ __forceinline__ void lower_update(double* Y, const double* X) {
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int s = wp < 4 ? wp : 11 - wp;
  double av[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) av[k] = X[(4 * k + t) * FLD + 8 * s + g];
#pragma unroll 1
  for (int f = 0; f <= s; f += 2) {
    const double* lb = X + t * FLD + 8 * f + g;
    double acc[2][2] = {};
#pragma unroll
    for (int k = 0; k < 16; ++k) {  // (f = s: the second block is not used)
      mma8(acc[0][0], acc[0][1], av[k], lb[4 * k * FLD]);
      mma8(acc[1][0], acc[1][1], av[k], lb[4 * k * FLD + 8]);
    }
#pragma unroll
    for (int u = 0; u < 2; ++u)
      if (f + u <= s) {
        double* y = Y + (8 * (f + u) + 2 * t) * FLD + 8 * s + g;
        y[0] -= acc[u][0];
        y[FLD] -= acc[u][1];
      }
  }
}

// A tile of 64 columns (h of its rows in range) through registers: all loads
// issued before the first shared store.
struct TileRegs {
  double v[FB * FB / FT];
  __device__ __forceinline__ void load(const MatDesc<double>& M, int r0, int c0, int h) {
    const int r = threadIdx.x & 63, cb = threadIdx.x >> 6;
    const double* p = M.a + (size_t)(c0 + cb) * M.ld + r0 + r;
#pragma unroll
    for (int k = 0; k < FB * FB / FT; ++k) v[k] = r < h ? __ldcg(p + (size_t)(4 * k) * M.ld) : 0.0;
  }
  __device__ __forceinline__ void store(double* S) const {
    const int r = threadIdx.x & 63, cb = threadIdx.x >> 6;
#pragma unroll
    for (int k = 0; k < FB * FB / FT; ++k) S[(cb + 4 * k) * FLD + r] = v[k];
  }
};

// x ← the strip of tile (i, q) updated by panels 0 … np−1 (q ≤ i).  The next
// panel's tiles are loaded while this panel's products run, when they are there.  alone:
// they are, the CTA's own barriers order them.
__device__ __forceinline__ bool update_tile(double (&x)[8][2], const MatDesc<double>& M, const Flags& F,
                                            int i, int q, int np, double* La, double* Lb) {
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, t = lane & 3;
  const int h = min(FB, M.n - i * FB), hq = min(FB, M.n - q * FB);
  const int r = 8 * wp + (lane >> 2);
  const double* p0 = M.a + (size_t)(q * FB) * M.ld + i * FB + r;
#pragma unroll
  for (int f = 0; f < 8; ++f)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int c = 8 * f + 2 * t + e;
      x[f][e] = (r < h && c < hq) ? __ldcg(p0 + (size_t)c * M.ld) : 0.0;
    }
  TileRegs ra, rb;
  const bool alone = F.alone();
  bool loaded = false;
  for (int p = 0; p < np; ++p) {
    if (!loaded) {
      if (!alone) {
        int ok = 1;
        if (threadIdx.x == 0) ok = poll_flags(F, F.tile(i, p), F.tile(q, p));
        if (!compute_and(ok)) return false;
      }
      ra.load(M, i * FB, p * FB, h);
      if (i != q) rb.load(M, q * FB, p * FB, hq);
    }
    compute_sync();  // the previous panel's reads of La and Lb are done
    ra.store(La);
    if (i != q) rb.store(Lb);
    if (alone) {
      loaded = p + 1 < np;
      compute_sync();
    } else {
      int there = 1;
      if (threadIdx.x == 0)
        there = p + 1 < np && F.set(F.tile(i, p + 1)) && F.set(F.tile(q, p + 1));
      loaded = compute_and(there);
    }
    if (loaded) {
      ra.load(M, i * FB, (p + 1) * FB, h);
      if (i != q) rb.load(M, q * FB, (p + 1) * FB, hq);
    }
    strip_update(x, La, i != q ? Lb : La);
  }
  return true;
}

// Tasks of panel j besides the chain, in the order in which they can run:
// tile (j+1,j+1) by the panels before j, tile (j+1,j) by the panels before j,
// tiles (i,j), i ≥ j+2, finished.  Each depends on earlier tasks and on the
// chain alone, so CTAs that take them in this order never wait in a cycle.
__host__ __device__ inline int flow_tasks(int nt, int j) {
  if (j + 1 >= nt) return 0;
  return (j > 0 ? 2 : 0) + (nt - j - 2);
}

// (M and F by value: by reference they would live in local memory and be read again
// after every store.)
__device__ __noinline__ bool run_task(const MatDesc<double> M, const Flags F, int j, int u, double* La,
                                      double* Lb, double* inv) {
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const bool partial = j > 0 && u < 2;
  const int i = partial ? j + 1 : j + 2 + u - (j > 0 ? 2 : 0), q = partial && u == 0 ? j + 1 : j;
  const int h = min(FB, M.n - i * FB), w = min(FB, M.n - q * FB);
  double x[8][2];
  if (!update_tile(x, M, F, i, q, j, La, Lb)) return false;
  if (!partial) {
    int ok = 1;
    if (!F.alone() && threadIdx.x == 0) ok = poll_flags(F, F.tile(j, j), F.tile(j, j));
    if (!compute_and(ok)) return false;  // (also: La and Lb are free)
    load_tile<FT>(La, M, j * FB, j * FB, FB, FB, threadIdx.x);
  } else {
    compute_sync();
  }
#pragma unroll
  for (int f = 0; f < 8; ++f)
#pragma unroll
    for (int e = 0; e < 2; ++e) Lb[(8 * f + 2 * t + e) * FLD + 8 * wp + g] = x[f][e];
  compute_sync();
  if (!partial) {
    if (threadIdx.x < FB) inv[threadIdx.x] = 1.0 / La[threadIdx.x * FLD + threadIdx.x];
    compute_sync();
    solve_strip(Lb, La, inv);
    compute_sync();
  }
  store_tile<FT>(Lb, M, i * FB, q * FB, h, w, i == q, threadIdx.x);
  if (!F.alone()) __threadfence();
  compute_sync();
  if (!F.alone() && threadIdx.x == 0) F.mark(!partial ? F.tile(i, j) : u == 0 ? F.c2 + i : F.c1 + j);
  return true;
}

// The chain of one matrix: the computing threads' side.  Buffers: the factored
// tile and the one that becomes the next alternate between T[0] and T[1], tile
// (j+1,j) is in X.  alone: the matrix has no other CTA, so the tasks of each
// panel run here too (in the buffers of the tiles not yet fetched), without flags.
struct ChainShared {
  double inv[FB], tinv[FB];
  int fail, err;
};

__device__ __forceinline__ void chain_compute(const MatDesc<double> M, const Flags F, bool alone, double* T0, double* T1,
                              double* X, ChainShared& cs, int* info, double* dmin, double* dmax) {
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int nt = F.nt;
  double lo = INFINITY, hi = 0.0;  // thread c < 64: pivots of column c of every tile
  int failed = 0;
  load_tile<FT>(T0, M, 0, 0, min(FB, M.n), min(FB, M.n), threadIdx.x);
  compute_sync();
  for (int j = 0; j < nt; ++j) {
    double *D = j & 1 ? T1 : T0, *Y = j & 1 ? T0 : T1;
    const int w = min(FB, M.n - j * FB), nb = (w + 7) >> 3;
    if (w & 7) {  // identity beyond the matrix in its last strip
      const int r = 8 * (nb - 1) + g;
      if (wp < 8 && r >= w)
        for (int c = 2 * t + (wp & 1) + 8 * (wp >> 1); c < FB; c += 32) D[c * FLD + r] = r == c ? 1.0 : 0.0;
      compute_sync();
    }
    factor_tile(D, cs.inv, nb, &cs.fail);
    compute_sync();
    const int fail = cs.fail;
    bar_arrive(kBarFactored, FT + FIO);
    if (fail != kNoFail) {
      failed = j * FB + fail + 1;
      if (!alone && j < nt - 1) bar_sync(kBarLoaded, FT + FIO);  // the fetch under way
      break;
    }
    if ((int)threadIdx.x < w) {
      const double v = D[threadIdx.x * FLD + threadIdx.x];
      lo = fmin(lo, v);
      hi = fmax(hi, v);
    }
    if (j == nt - 1) break;
    if (alone) {
      bar_sync(kBarStored, FT + FIO);  // tile (j,j) is in global memory
      for (int u = 0; u < flow_tasks(nt, j); ++u) run_task(M, F, j, u, X, Y, cs.tinv);
      bar_arrive(kBarTasks, FT + FIO);
    }
    bar_sync(kBarLoaded, FT + FIO);
    if (cs.err) break;
    solve_strip(X, D, cs.inv);
    compute_sync();
    bar_arrive(kBarSolved, FT + FIO);
    lower_update(Y, X);
    compute_sync();
    bar_arrive(kBarUpdated, FT + FIO);
  }
  // Min and max |L_cc| over the factored tiles.
  if (threadIdx.x < FB) {
    lo = warp_min(lo);
    hi = warp_max(hi);
    if (lane == 0) cs.tinv[wp] = lo, cs.tinv[2 + wp] = hi;
  }
  compute_sync();
  if (threadIdx.x == 0) {
    *info = cs.err ? -1 : failed;
    *dmin = fmin(cs.tinv[0], cs.tinv[1]);
    *dmax = fmax(cs.tinv[2], cs.tinv[3]);
  }
}

// The global side of the chain (FIO threads, tid counted from 0).
__device__ __forceinline__ void chain_io(const MatDesc<double> M, const Flags F, bool alone, double* T0, double* T1,
                         double* X, ChainShared& cs, int tid) {
  const int nt = F.nt;
  auto fetch = [&](int j) {  // tiles (j+1,j) and (j+1,j+1)
    const int h = min(FB, M.n - (j + 1) * FB);
    load_tile<FIO>(X, M, (j + 1) * FB, j * FB, h, FB, tid);
    load_tile<FIO>(j & 1 ? T0 : T1, M, (j + 1) * FB, (j + 1) * FB, h, h, tid);
    bar_arrive(kBarLoaded, FT + FIO);
  };
  auto publish = [&](unsigned* f) {
    __threadfence();
    bar_sync(kBarIo, FIO);
    if (tid == 0) F.mark(f);
  };
  if (nt > 1 && !alone) fetch(0);
  for (int j = 0; j < nt; ++j) {
    const int w = min(FB, M.n - j * FB), h = min(FB, M.n - (j + 1) * FB);
    bar_sync(kBarFactored, FT + FIO);
    if (cs.fail != kNoFail) {
      if (tid == 0) F.mark(F.stop);
      return;
    }
    store_tile<FIO>(j & 1 ? T1 : T0, M, j * FB, j * FB, w, w, true, tid);
    if (j == nt - 1) return;
    publish(F.tile(j, j));
    if (alone) {
      bar_sync(kBarIo, FIO);  // the flag is set
      bar_arrive(kBarStored, FT + FIO);
      bar_sync(kBarTasks, FT + FIO);
      fetch(j);
    }
    bar_sync(kBarSolved, FT + FIO);
    store_tile<FIO>(X, M, (j + 1) * FB, j * FB, h, FB, false, tid);
    publish(F.tile(j + 1, j));
    bar_sync(kBarUpdated, FT + FIO);  // X and tile (j,j)'s buffer are free
    if (j + 2 < nt && !alone) {
      if (tid == 0 && !poll_flags(F, F.c1 + j + 1, F.c2 + j + 2)) cs.err = 1;
      bar_sync(kBarIo, FIO);
      if (cs.err) {
        bar_sync(kBarFactored, FT + FIO);
        bar_arrive(kBarLoaded, FT + FIO);
        return;
      }
      fetch(j + 1);
    }
  }
}

// Strict upper triangle: a warp per column.
__device__ void zero_upper_part(const MatDesc<double>& M, int part, int parts, int nwarps) {
  const int lane = threadIdx.x & 31;
  for (int c = part * nwarps + (threadIdx.x >> 5); c < M.n; c += parts * nwarps)
    for (int r = lane; r < c; r += 32) M.a[(size_t)c * M.ld + r] = 0.0;
}

struct FlowMats {
  MatDesc<double> m[kFlowInline];
};

// gsize CTAs per matrix; CTA 0 of a group runs the chain.  Groups take the
// matrices in turn when there are more matrices than groups.
__global__ void __launch_bounds__(FT + FIO, 1)
    k_potrf_flow(const __grid_constant__ FlowMats few, const MatDesc<double>* mats, int nmat, int gsize,
                 int ngroups, unsigned* flags, int words, unsigned epoch, int* info, double* dmin,
                 double* dmax, int zero_upper) {
  extern __shared__ __align__(16) double fsm[];
  double *T0 = fsm, *T1 = fsm + kTile, *X = fsm + 2 * kTile;
  __shared__ ChainShared cs;
  const int grp = blockIdx.x / gsize, me = blockIdx.x % gsize;
  for (int b = grp; b < nmat; b += ngroups) {
    const MatDesc<double> M = nmat <= kFlowInline ? few.m[b] : mats[b];
    const int nt = (M.n + FB - 1) / FB;
    const Flags F(flags + (size_t)b * words, nt, gsize == 1 ? 0u : epoch);
    __syncthreads();
    if (me == 0) {
      if (threadIdx.x == 0) cs.fail = kNoFail, cs.err = 0;
      __syncthreads();
      if (threadIdx.x < FT) chain_compute(M, F, gsize == 1, T0, T1, X, cs, info + b, dmin + b, dmax + b);
      else chain_io(M, F, gsize == 1, T0, T1, X, cs, (int)threadIdx.x - FT);
      __syncthreads();
    } else if (threadIdx.x < FT) {
      int first = me - 1;  // this CTA's next task, counted over the panels
      bool ok = true;
      for (int j = 0; ok && j < nt; ++j) {
        const int n = flow_tasks(nt, j);
        while (ok && first < n) {
          ok = run_task(M, F, j, first, T0, T1, cs.tinv);
          first += gsize - 1;
        }
        first -= n;
      }
    }
    if (zero_upper) zero_upper_part(M, me, gsize, (FT + FIO) / 32);
  }
}

// Tile s of L (lower, w of its rows in range) inverted: X = L⁻ᵀ in shared X, from the
// strips' solves of X·Lᵀ = I, so that W = Xᵀ.  49 → 6 µs a call against one thread per
// column, whose chain was 64 rows of up to 63 dependent products and a division each.
__device__ __forceinline__ void invert_tile(const double* L, long long ld, int s0, int w, double* D, double* X,
                                            double* inv) {
  for (int e = threadIdx.x; e < FB * FB; e += FT) {
    const int r = e & 63, c = e >> 6;
    D[c * FLD + r] = (r < w && c <= r) ? L[(size_t)(s0 + c) * ld + s0 + r] : (r == c ? 1.0 : 0.0);
    X[c * FLD + r] = r == c ? 1.0 : 0.0;
  }
  __syncthreads();
  if (threadIdx.x < FB) inv[threadIdx.x] = 1.0 / D[threadIdx.x * FLD + threadIdx.x];
  __syncthreads();
  solve_strip(X, D, inv);
  __syncthreads();
}

// Dinv[s] = (tile s of L)⁻¹, 64×64 column-major, zeros above the diagonal and outside.
__global__ void __launch_bounds__(FT) k_tile_inverse(const double* L, long long ld, int n, double* Dinv) {
  extern __shared__ __align__(16) double fsm[];
  __shared__ double inv[FB];
  const int s0 = blockIdx.x * FB, w = min(FB, n - s0);
  invert_tile(L, ld, s0, w, fsm, fsm + kTile, inv);
  double* out = Dinv + (size_t)blockIdx.x * FB * FB;
  for (int e = threadIdx.x; e < FB * FB; e += FT) {
    const int c = e & 63, r = e >> 6;  // W[c][r] = X[r][c]
    out[e] = r <= c && c < w ? fsm[kTile + c * FLD + r] : 0.0;
  }
}

// The diagonal tiles of W_b = L_b⁻¹ (lower parts).
__global__ void __launch_bounds__(FT) k_tile_inverse_list(const __grid_constant__ TrinvList q) {
  extern __shared__ __align__(16) double fsm[];
  __shared__ double inv[FB];
  const int n = q.n[blockIdx.y], s0 = blockIdx.x * FB, w = min(FB, n - s0);
  if (w <= 0) return;
  invert_tile(q.L[blockIdx.y], n, s0, w, fsm, fsm + kTile, inv);
  double* W = q.W[blockIdx.y];
  for (int e = threadIdx.x; e < FB * FB; e += FT) {
    const int c = e & 63, r = e >> 6;
    if (r <= c && c < w) W[(size_t)(s0 + r) * n + s0 + c] = fsm[kTile + c * FLD + r];
  }
}

}  // namespace

size_t potrf_flow_flag_words(int nmat, int nmax) {
  const size_t nt = ceil_div(nmax, FB);
  return (size_t)nmat * (nt * nt + 2 * nt + 2);
}

int potrf_flow_group(int nmat, int nmax, int sms) {
  const int nt = ceil_div(nmax, FB);
  int tasks = 0;
  for (int j = 0; j < nt; ++j) tasks += flow_tasks(nt, j);
  return std::max(1, std::min(sms / nmat, 1 + tasks));
}

// One CTA per SM fits (104 KB of shared memory, 168 registers); a group is as large
// as the tasks of the largest matrix can use.  Measured on the B200, one matrix, ms
// (before: panels in shared memory below 459, one cooperative launch with grid
// barriers above; the factors are identical bit for bit, but for a column whose pivot
// is the one exception of sqrt_rcp):
//   n       64     128    320    512    1030   2000   3000
//   before  0.039  0.087  0.252  0.434  0.989  1.848  3.084
//   now     0.022  0.044  0.102  0.164  0.352  0.657  1.004
// A panel takes about 20 µs of it: 9 µs for the 64 pivots, 4 µs for tile (j+1,j),
// 2 µs for tile (j+1,j+1); the rest is the way round through the other CTAs (tile
// (j,j) out, row j+2 solved, tiles (j+2,j+1) and (j+2,j+2) updated and back).
void potrf_flow(const MatDesc<double>* mats, MatDesc<double>* d_mats, int nmat, int nmax, int* info,
                double* dmin, double* dmax, FlowFlags& flags, int sms, cudaStream_t st, bool zero_upper) {
  if (nmat <= 0 || nmax <= 0) return;
  ensure_smem(k_potrf_flow, kFlowSmem);
  const int nt = ceil_div(nmax, FB);
  int words = nt * nt + 2 * nt + 2, gsize = potrf_flow_group(nmat, nmax, sms);
  int ngroups = std::min(nmat, sms / gsize), zu = zero_upper ? 1 : 0;
  FlowMats few{};
  if (nmat <= kFlowInline) std::copy(mats, mats + nmat, few.m);
  else SDPX_CUDA(cudaMemcpyAsync(d_mats, mats, sizeof(*mats) * nmat, cudaMemcpyHostToDevice, st));
  flags.next(nmat, nmax, st);
  unsigned* fw = flags.words.p;
  unsigned ep = flags.epoch;
  if (gsize == 1) {  // no CTA waits for another
    k_potrf_flow<<<ngroups, FT + FIO, kFlowSmem, st>>>(few, d_mats, nmat, gsize, ngroups, fw, words, ep, info,
                                                       dmin, dmax, zu);
  } else {
    void* args[] = {&few, &d_mats, &nmat, &gsize, &ngroups, &fw, &words, &ep, &info, &dmin, &dmax, &zu};
    SDPX_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<void*>(k_potrf_flow), dim3(ngroups * gsize),
                                          dim3(FT + FIO), args, kFlowSmem, st));
  }
  SDPX_LAUNCH_CHECK();
}

void factor_diag_inverses(const double* L, long long ld, int n, double* Dinv, cudaStream_t st) {
  const size_t smem = sizeof(double) * 2 * kTile;
  ensure_smem(k_tile_inverse, smem);
  k_tile_inverse<<<ceil_div(n, FB), FT, smem, st>>>(L, ld, n, Dinv);
  SDPX_LAUNCH_CHECK();
}

void invert_diag_tiles(const TrinvList& q, cudaStream_t st) {
  int nmax = 0;
  for (int b = 0; b < q.count; ++b) nmax = std::max(nmax, q.n[b]);
  if (nmax == 0) return;
  const size_t smem = sizeof(double) * 2 * kTile;
  ensure_smem(k_tile_inverse_list, smem);
  k_tile_inverse_list<<<dim3(ceil_div(nmax, FB), q.count), FT, smem, st>>>(q);
  SDPX_LAUNCH_CHECK();
}

}  // namespace sdpx
