// Batched Cholesky / triangular kernels (chol.cu).
#pragma once
#include <algorithm>

#include "common.cuh"
#include "dbuf.h"

namespace sdpx {

template <class T>
struct MatDesc {
  T* a;     // column-major n×n, leading dimension ld
  int n;
  int ld;
};

// Tile flags of potrf_flow, for the launches of one stream.  Each launch marks with an
// epoch of its own, so the words are cleared only when allocated or when the count wraps.
size_t potrf_flow_flag_words(int nmat, int nmax);
struct FlowFlags {
  DBuf<unsigned> words;
  unsigned epoch = 0;
  void next(int nmat, int nmax, cudaStream_t st) {
    const size_t need = potrf_flow_flag_words(nmat, nmax);
    if (words.n < need) {
      words.alloc(2 * need);
      epoch = 0;
    }
    if (++epoch <= 1) {
      words.zero(st);
      epoch = 1;
    }
  }
};

// CTAs that potrf_flow gives each of nmat matrices, the largest of order nmax.
int potrf_flow_group(int nmat, int nmax, int sms);

// Lower Cholesky in place of nmat matrices (host array `mats`, largest order nmax), one
// launch (potrf_flow.cu): a CTA per matrix runs the pivot chain, sms/nmat − 1 others its
// remaining tiles, ordered by tile flags.  info[b] = 0 on success, else the 1-based index
// of the first non-positive pivot (the no-throw contract of SDPX's `kchol!`,
// src/kernels/generic.jl:133-155), or −1 when a wait for a tile gave up (about a second).
// dmin/dmax receive min/max |L_ii|; the three may be pinned host memory, readable once
// the stream is synchronised.  The strict upper triangle is zeroed unless zero_upper is
// false (positive-definiteness tests that only read info/dmin/dmax).  d_mats takes the
// descriptors of more than kFlowInline matrices (fewer travel with the launch).
constexpr int kFlowInline = 16;
void potrf_flow(const MatDesc<double>* mats, MatDesc<double>* d_mats, int nmat, int nmax, int* info,
                double* dmin, double* dmax, FlowFlags& flags, int sms, cudaStream_t st,
                bool zero_upper = true);

// Inverses of the 64×64 diagonal tiles of a lower factor L (n×n): Dinv[s]
// (64×64, column-major).
void factor_diag_inverses(const double* L, long long ld, int n, double* Dinv, cudaStream_t st);

// rhs ← (L Lᵀ)⁻¹ rhs, one launch (cooperative for n > 64).  `work`
// (cholesky_solve_work(n) doubles) and `err` must not be shared by concurrent calls;
// *err (zero on entry, else nothing waits) becomes 1 and rhs NaN when a wait gave up.
inline size_t cholesky_solve_work(int n) { return 2 * (size_t)ceil_div(n, 64) * 64; }
void cholesky_solve(const double* L, long long ld, int n, const double* Dinv, double* rhs, double* work,
                    int* err, int sms, cudaStream_t st);

// Lower factors to invert together: W_b = L_b⁻¹ (n_b×n_b, column-major, ld n_b), tmp_b
// n_b×n_b scratch.  The strict upper triangle of W must be zero on entry and is not
// written.
constexpr int kTrinvMax = 16;
struct TrinvList {
  int count = 0;
  int n[kTrinvMax];
  const double* L[kTrinvMax];
  double *W[kTrinvMax], *tmp[kTrinvMax];
};
void invert_diag_tiles(const TrinvList& q, cudaStream_t st);  // the 64×64 diagonal tiles alone
// By recursive doubling over 64×64 tiles, every step one launch for the whole list.
void trinv(const TrinvList& q, cudaStream_t st);

}  // namespace sdpx
