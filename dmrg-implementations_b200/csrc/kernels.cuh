// Launchers for the Krylov, SVD and data-movement kernels.
#pragma once

#include "common.cuh"

namespace dmrg2 {

constexpr int KRYLOV_CAP = 128;   // hard cap on Krylov vectors per Lanczos pass
constexpr int VEC_THREADS = 256;

// Device-resident state of one Lanczos solve (one per engine).
struct LanczosDev {
  double alpha[KRYLOV_CAP];
  double beta[KRYLOV_CAP];
  double coef[2 * (KRYLOV_CAP + 1)];   // projection coefficients of the current pass (re, im)
  double ritz[KRYLOV_CAP];             // Ritz coefficients (real: T is real symmetric)
  double nrm2;                         // squared norm produced by the last reduction
  double e_prev, e_cur;
  double tol;
  int done;                            // 1 once converged / broken down / Krylov space full
  int gave_up;                         // a block's bounded wait at a grid barrier ran out: no result
  int converged;
  int n_iter;                          // size of the tridiagonal matrix
  int randomized;
  int kmax;
  int j;                               // Krylov index of the device-looped solve's current step
  int guard;                           // loop bodies run so far (bounds the device loop)
  unsigned long long t_mark;           // %globaltimer when the current matvec was issued
  unsigned long long mv_ns;            // matvec time accumulated by the device-looped solve
  unsigned bar[8];                     // grid barrier counters of the fused step, start and Ritz kernels
};

// What the host needs of a finished solve, in page-locked host memory (the last kernel of
// the solve writes it; valid once the stream has run it).
struct LanczosHost {
  double e_cur;
  unsigned long long mv_ns;
  int done, converged, n_iter, guard;
  int gave_up;  // cleared by the host before a solve, only ever set by its kernels
};

// Reduction scratch shared by the vector kernels.
struct RedScratch {
  double* part = nullptr;   // [nblk][ncoef*2]
  unsigned* counter = nullptr;
  int nblk = 0;
  int step_blocks = 0;      // blocks a cooperative Lanczos kernel may have (0: none is launched)
};

constexpr int STEP_BLOCKS = 148;  // blocks of a cooperative Lanczos step at most (one per SM)
int vec_blocks(ll n);
// blocks' worth of partial sums (2 (KRYLOV_CAP + 2) each) RedScratch::part holds for vectors
// of up to n elements: the streaming passes', or the fused step's two sets
int red_blocks(ll n);

// w <- H v is done by the caller; these kernels implement one Lanczos step.
// start: nrm(theta) -> (random fill if ~0) -> v0 = theta/|theta| (also into cur when given);
// seed_host, when given, is page-locked host memory that holds the seed (read only where the
// random fill is needed)
template <typename T>
void lz_start(T* theta, T* v0, ll n, LanczosDev* st, RedScratch& r, unsigned seed, double tol,
              int kmax, cudaStream_t s, T* cur = nullptr, const unsigned* seed_host = nullptr);
// Krylov step nv (w = H v_(nv-1)): w orthogonalised against v_0 .. v_(nv-1), alpha, beta and the
// stop rule, v_nv = w / |w| into V when nv < kmax, and the done flag into host_done
// (page-locked; valid once the stream has run the step). One launch where the vectors fit
// the fused kernel, the streaming passes (which overwrite w) beyond.
template <typename T>
void lz_step(T* V, int nv, ll n, T* w, LanczosDev* st, RedScratch& r, int kmax, int* host_done, cudaStream_t s);
// The same step with the Krylov index read on the device (st->j), for a loop that runs
// without the host: v_(j+1) also into cur (the matvec's fixed input); it ends one body of
// the device loop, advancing st->j and setting the loop condition of h to "not done and
// fewer than kmax bodies run".
template <typename T>
void lz_step_dev(T* V, ll n, T* w, T* cur, LanczosDev* st, RedScratch& r, int kmax, cudaGraphConditionalHandle h,
                 cudaStream_t s);
// Ritz vector out = sum_i ritz_i V_i, normalised, and the solve's report into host.
template <typename T>
void lz_ritz(const T* V, ll n, T* out, LanczosDev* st, RedScratch& r, LanczosHost* host, cudaStream_t s);

// Test hook: this many deferred solves from now (0: none) one is made to fail, as by a barrier that gave up.
std::atomic<int>& lz_fail_countdown();
void lz_fail(LanczosDev* st, LanczosHost* host, cudaStream_t s);

// ---------------------------------------------------------------- SVD
struct JacobiCtl {
  unsigned bar_count;
  unsigned bar_gen;
  int err;
  int sweeps;
  int rotated[64];
};

struct SvdOut {
  int k;            // kept rank
  int nonzero;
  double trunc_err; // sum of discarded sigma^2
  double sigma_max;
  double sigma_max2;
  double fro2;
  int jacobi_sweeps;
  int jacobi_err;
  int ns_done;      // eigenvector block already orthonormal (Newton-Schulz steps skipped)
  int ns_near;      // one Newton-Schulz step makes it so (a bound on every entry it leaves is below the tolerance)
};

template <typename T>
void svd_jacobi(T* X, T* Q, int nvec, ll len, JacobiCtl* ctl, int max_sweeps, double tol,
                const double* fro2_dev, cudaStream_t s);  // fro2_dev: |X|_F^2 on device, or null for 1
template <typename T>
void svd_sort_truncate(const T* X, int nvec, ll len, double* sigma, int* perm, SvdOut* out,
                       int chi_max, double cutoff, bool relative_cutoff, const JacobiCtl* ctl,
                       cudaStream_t s);
// gather: left (rows x k) and right (k x cols) factors from X (rotated vectors) / Q.
//   mode 0 ('R'): vectors were rows of theta: left = conj(Q^T) cols, right = X rows
//   mode 1 ('L'): vectors were columns:       left = X^T,            right = conj(Q) rows
template <typename T>
void svd_gather(const T* X, const T* Q, const int* perm, int nvec, ll len, int k, int mode,
                T* left, T* right, cudaStream_t s);

// boundary merge of the parallel sweep: the k kept singular values in sorted order,
// v <- 1 / max(v, floor), and out = diag(v) in (or diag(1/v) in) for a rows x cols block
void gather_sigma(const double* sigma, const int* perm, int k, double* out, cudaStream_t s);
void inv_clip(double* v, int k, double floor, cudaStream_t s);
template <typename T>
void row_scale(const T* in, const double* v, int rows, ll cols, T* out, bool invert, cudaStream_t s);

// ---------------------------------------------------------------- eigen path (eig.cu)
template <typename T>
void hetrd_cluster(T* G, int n, ll ld, double* d, double* e, T* tau, cudaStream_t s);
void tridiag_eigvals(const double* d, const double* e, int n, int K, double* lam, cudaStream_t s);
// gtol_rel: the group tolerance (relative to lam[0]) that group_mgs will use on the result
void tridiag_eigvecs(const double* d, const double* e, int n, int K, const double* lam,
                     const SvdOut* tr, double* Z, double* scratch, double gtol_rel, cudaStream_t s);
void group_mgs(double* Z, int n, int K, const double* lam, const SvdOut* tr, double gtol_rel,
               cudaStream_t s);
// compact-WY triangles of the reflector blocks that apply_q uses for (n, K); apply_q builds
// them itself unless wy_ready says they were built already (e.g. on a side stream)
template <typename T>
void wy_build(const T* R, ll ld, const T* tau, int n, int K, T* Tb, cudaStream_t s);
template <typename T>
void apply_q(const T* R, ll ld, const T* tau, int n, const double* Z, int K, const SvdOut* tr, T* Zg,
             T* Tb, cudaStream_t s, bool wy_ready = false);
// sets out->ns_done and out->ns_near from S = Z^T Z (K x K); part: 64 doubles
void ns_check(const double* S, int K, SvdOut* out, double tol, double* part, unsigned* counter,
              cudaStream_t s);
// Up to `iters` Newton-Schulz steps of Z (n x K) in one launch, with ns_check's flag; false, with
// nothing launched, for blocks beyond 128 x 64
bool ns_small(double* Z, int n, int K, SvdOut* out, double tol, int iters, cudaStream_t s);
// k from the eigenvalues: min(chi_max, K, #lam above max(cutoff^2 (x lam_max if relative),
// floor_rel lam_max)); eigenvalues at or below floor_rel lam_max are rounding noise
constexpr double EIG_NOISE_FLOOR = 16.0 * 2.2e-16;
void eig_truncate(const double* d, const double* lam, int n, int K, int chi_max, double cutoff,
                  bool relative, SvdOut* out, cudaStream_t s, double floor_rel = EIG_NOISE_FLOOR);
template <typename T>
void copy_cols_conj(const T* in, ll ldi, int rows, int k, T* out, cudaStream_t s);
template <typename T>
void transpose_conj(const T* in, ll ldi, int rows, int k, T* out, cudaStream_t s, const int* skip = nullptr);

// ---------------------------------------------------------------- warm-started split
// What the host needs of a split, in page-locked host memory.
struct SplitHost {
  double theta2, kept2;  // |theta|^2, |kept factor|^2
  int failed;            // an orthonormalisation gave up or the polish did not converge
};
// status <- 0, *out <- {k}
void split_begin(int* status, SvdOut* out, int k, cudaStream_t s);
// |theta|^2 and |kept|^2, and the split's report into host (one launch; the last block of the
// grid sums the partials in block order and writes the report)
template <typename T>
void split_finish(const T* theta, ll nt, const T* kept, ll nk, const int* status, const SvdOut* out, SplitHost* host,
                  RedScratch& r, cudaStream_t s);

// left <- l (nl elements) and right <- r (nr), unless *skip
template <typename T>
void split_commit(const T* l, T* left, ll nl, const T* r, T* right, ll nr, const int* skip, cudaStream_t s);

// ---------------------------------------------------------------- misc
template <typename T>
void transpose(const T* in, T* out, ll rows, ll cols, cudaStream_t s);  // out[c][r] = in[r][c]
template <typename T>
void set_identity(T* Q, int n, cudaStream_t s);
template <typename T>
void scale_inplace(T* x, ll n, const double* inv_scale_dev, cudaStream_t s);
template <typename T>
void norm2(const T* x, ll n, double* out_dev, RedScratch& r, cudaStream_t s);
template <typename T>
void trace_real(const T* M, int n, ll ld, double* out_re, double* out_im, cudaStream_t s);
// flag = 1 when the n x n matrix P equals the identity to tol (max |P - 1|)
template <typename T>
void identity_check(const T* P, int n, double tol, int* flag, cudaStream_t s);

}  // namespace dmrg2
