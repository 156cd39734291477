// Host launchers of the memory-bound kernels (vec_kernels.cu).
#pragma once
#include <algorithm>

#include "common.cuh"

namespace sdpx {

struct TrialDesc {
  const double* X;
  const double* dX;
  double* out;
  double t;
  int k;
};
// (`list` in host memory; d_list takes more than kTrialInline entries.)
constexpr int kTrialInline = 16;
void make_trials_list(const TrialDesc* list, TrialDesc* d_list, int n, int kmax, cudaStream_t st);

void gemv_n(const double* A, long long K, int m, const double* x, double* out, double* part,
            int chunks, cudaStream_t st);
void gemv_t(const double* A, long long K, int m, const double* z, double alpha, const double* base,
            double beta, double* out, cudaStream_t st);
// The same products as compensated (Dot2) sums rounded once, for the
// residuals: out = 𝒜x − X − C (X, C may be null; part holds 2·chunks·K
// doubles) and out = alpha·𝒜ᵀz + beta·base.
void gemv_n_acc(const double* A, long long K, int m, const double* x, const double* X,
                const double* C, double* out, double* part, int chunks, cudaStream_t st);
void gemv_n_sym_acc(const double* Ap, long long Kt, int m, const double* x, const long long* lo,
                    const long long* up, const double* X, const double* C, double* out,
                    double* part, int chunks, cudaStream_t st);
void gemv_t_acc(const double* A, long long K, int m, const double* z, double alpha,
                const double* base, double beta, double* out, cudaStream_t st);
// Lower-triangle copy of the constraint matrix (Kt kept rows per column):
// pack_rows gathers it, gemv_n_sym writes Ap·x to both stacked positions
// lo[q] and up[q] of every kept row, fold_sym folds a stacked vector onto the
// kept rows (z[lo] + z[up] off the diagonal) for Apᵀ·zf = 𝒜ᵀz.
void pack_rows(const double* A, long long K, int m, const long long* rows, long long Kt, double* Ap,
               cudaStream_t st);
void gemv_n_sym(const double* Ap, long long Kt, int m, const double* x, const long long* lo,
                const long long* up, double* out, double* part, int chunks, cudaStream_t st);
void fold_sym(long long Kt, const double* z, const long long* lo, const long long* up, double* zf,
              cudaStream_t st);
void axpbypcz(long long n, double a, const double* x, double b, const double* y, double c,
              const double* z, double* out, cudaStream_t st);
void combine(long long n, double* x, double t, const double* d, cudaStream_t st);
void scale(long long n, double* x, double f, cudaStream_t st);
// Several vectors set to zero by one launch.
constexpr int kZeroMax = 32;
struct ZeroList {
  int n = 0;
  double* p[kZeroMax];
  long long len[kZeroMax];
};
void zero_list(const ZeroList& q, cudaStream_t st);
void absmax(long long n, const double* x, double* out, cudaStream_t st);
// out[e] = max|x_e| of every entry (NaN counts as +inf), one launch; `out` may be pinned
// host memory.  `work` is zero between launches and belongs to one stream.
constexpr int kNormMax = 8;
struct NormWork {
  double v[kNormMax];
  unsigned done;
};
struct NormList {
  int n = 0, first[kNormMax + 1] = {0};  // blocks of an entry: [first[e], first[e+1])
  long long len[kNormMax];
  const double* x[kNormMax];
  double* out[kNormMax];
  void add(long long len_, const double* x_, double* out_);  // entries of length 0 are dropped
};
void absmax_list(const NormList& q, NormWork* work, cudaStream_t st);
// Chunks of the segments of a dot product: chunk q covers rows [start, end) of segment
// seg; segment s owns the chunks [first[s], first[s+1]).
struct SegChunk {
  long long start, end;
  int seg;
};
constexpr int kSegChunk = 2048;
// out[s] = Σ over segment s; `out` may be pinned host memory, `done` is zero between
// launches, `part` holds a value per chunk.
void seg_dot(const SegChunk* d_chunks, int nchunk, const int* d_first, int nseg, const double* x,
             const double* dx, double tx, const double* y, const double* dy, double ty, double* part,
             unsigned* done, double* out, cudaStream_t st);
void block_trace(const long long* d_off, const int* d_k, int nseg, const double* M, double* out,
                 cudaStream_t st);
void add_diag(const long long* d_off, const int* d_k, int nseg, int kmax, double* M,
              const double* d_shifts, double uniform, cudaStream_t st);
// The same with the shifts in host memory; d_tmp takes those of more than kShiftInline
// segments.
constexpr int kShiftInline = 16;
void add_diag_host(const long long* d_off, const int* d_k, int nseg, int kmax, double* M,
                   const double* shifts, double* d_tmp, cudaStream_t st);
void symmetrize(const long long* d_off, const int* d_k, int nseg, int kmax, double* M,
                cudaStream_t st);
void gershgorin(const long long* d_off, const int* d_k, int nseg, int kmax, const double* M,
                double* d_cand, const long long* d_cand_off, double* d_scale, int* d_nonfinite,
                cudaStream_t st);
void diag_residual_R(int nd, long long od, const double* X, const double* Y, const double* mu_user,
                     const int* user, int use_affine, double* R, cudaStream_t st);
void diag_factor(int nd, long long od, const double* X, const double* Y, double* LX, double* MY,
                 int* fail, cudaStream_t st);
void diag_rhs_Z(int nd, long long od, const double* P, const double* Y, const double* R,
                const double* LX, double* Z, cudaStream_t st);
void diag_dY(int nd, long long od, const double* R, const double* dX, const double* Y,
             const double* LX, double* dY, cudaStream_t st);
void diag_corrector_R(int nd, long long od, const double* X, const double* Y, const double* dX,
                      const double* dY, const double* target_user, const int* user, double* R,
                      cudaStream_t st);
void diag_panel(long long K, int m, int nd, long long od, const double* A, const double* LX,
                const double* MY, double* Pc, cudaStream_t st);
constexpr int kDiagSteps = 16;
struct DiagSteps {
  int n = 0;
  double t[kDiagSteps];
};
// (fail may be pinned host memory; zero on entry.)
void diag_trial(int nd, long long od, const double* X, const double* dX, const DiagSteps& q, int margin, int* fail,
                cudaStream_t st);
void diag_ftb(int nd, long long od, const double* X, const double* dX, double* d_out,
              cudaStream_t st);
void gather(long long n, const long long* map, const double* src, double* dst, cudaStream_t st);
void scatter(long long n, const long long* map, const double* src, double* dst, cudaStream_t st);
void mirror_lower(int m, double* S, cudaStream_t st);
// (err_out, pinned host memory, receives *err where err is not null.)
void copy_reg(int m, const double* S, double* Sf, double reg, cudaStream_t st, const int* err = nullptr,
              int* err_out = nullptr);
// (d0, d1) = (s0, s1)
void copy_pair(long long n, const double* s0, double* d0, const double* s1, double* d1, cudaStream_t st);
// dst[map[e]] = a·x[e] + b·y[e]
void scatter_axpby(long long n, const long long* map, double a, const double* x, double b, const double* y,
                   double* dst, cudaStream_t st);
void symv_full(int m, const double* S, const double* x, double alpha, const double* b, double beta,
               double* y, cudaStream_t st);
void ruiz_rowmax_dense(const double* A, const double* C, long long K, int m, long long off, int k, int np,
                       const double* F, int rows, const int* active, double* rn, cudaStream_t st);
void ruiz_rowmax_diag(const double* A, const double* C, long long K, int m, long long od, int nd, int np,
                      const double* F, int rows, const int* active, double* rn, cudaStream_t st);
void ruiz_update(int it, int nb, const int* d_k, const int* d_row0, int nd, double* rn, double* F, double* E,
                 int* active, int* used, int* any, cudaStream_t st);
void ruiz_weights(int nb, const int* d_k, const long long* d_off, const int* d_row0, int kmax, int nd,
                  long long od, long long K, int np, const double* F, int rows, double* w, cudaStream_t st);
void colmax(const double* A, const double* w, int np, long long K, int m, double* out, cudaStream_t st);
void scale_store(double* A, double* A0, long long K, int m, const double* w, int np, const double* s,
                 cudaStream_t st);

}  // namespace sdpx
