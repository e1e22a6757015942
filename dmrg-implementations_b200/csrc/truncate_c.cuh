// Warm-started subspace split of complex two-site tensors.
//
// The same power half-steps, modes and acceptance as the real split (wst_split in
// truncate.cuh), with complex DMMA GEMMs for the products with theta. Each
// orthonormalisation runs on the real embedding of the complex column block, with the
// column pairs (y_j, i y_j) interleaved (embed_pairs / extract_pairs). On it, unit
// columns, the Gram matrix, the tiled Cholesky factor and the row solve amount to complex
// Gram-Schmidt: each y_j is orthogonalised against a span closed under multiplication by
// i. So the even columns of the result are a complex-orthonormal basis, triangular in the
// columns as the real split requires. The final Newton-Schulz polish also runs on the
// embedding: for a matrix of that structure each step is the embedding of the complex
// step.
//
//   'R': U1 = tri(theta B^H) [+ V1 = tri(theta^H U1), U2 = tri(theta V1)], left = U,
//        right = U^H theta;
//   'L': V1 = tri(theta^H A) [+ U1 = tri(theta V1), V2 = tri(theta^H U1)], right = V^H,
//        left = theta V.
// theta B^H is formed as the transpose of conj(B) theta^T, because the GEMM conjugates
// only its first operand.
#pragma once

#include "rsvd.cuh"
#include "truncate.cuh"

namespace dmrg2 {

struct WstWorkC {
  zc* Ya = nullptr;      // qmax x kmax
  zc* Yb = nullptr;
  double* Z1 = nullptr;  // real embeddings: (2 qmax) x (2 kmax) each
  double* Z2 = nullptr;
  double* S = nullptr;   // Gram matrix, then its tiled factor (np x np, np = chol_padded(2 kmax))
  double* dscale = nullptr;  // 1 / norm of each embedded column
  double* part = nullptr;
  unsigned* counter = nullptr;
  int* status = nullptr;
  SvdOut* out = nullptr;
  SplitHost* h_rep = nullptr;  // pinned: the split's report
  int qmax = 0, kmax = 0;
  size_t bytes = 0;
  std::vector<void*> owned;

  void* alloc(size_t b) {
    void* p = dev_alloc(std::max<size_t>(b, 16));
    owned.push_back(p);
    bytes += b;
    return p;
  }
  void init(int qmax_, int kmax_) {
    qmax = std::max(qmax_, 1);
    kmax = std::max(std::min(kmax_, CHOL_MAX / 2), 1);
    const size_t qk = (size_t)qmax * kmax;
    Ya = (zc*)alloc(sizeof(zc) * qk);
    Yb = (zc*)alloc(sizeof(zc) * qk);
    Z1 = (double*)alloc(sizeof(double) * 4 * qk);
    Z2 = (double*)alloc(sizeof(double) * 4 * qk);
    const size_t np = (size_t)chol_padded(2 * kmax);
    S = (double*)alloc(sizeof(double) * np * np);
    dscale = (double*)alloc(sizeof(double) * 2 * (size_t)kmax);
    part = (double*)alloc(sizeof(double) * 64);
    counter = (unsigned*)alloc(sizeof(unsigned) * 4);
    status = (int*)alloc(sizeof(int) * 4);
    out = (SvdOut*)alloc(sizeof(SvdOut));
    DMRG2_CUDA(cudaMemset(counter, 0, sizeof(unsigned) * 4));
    h_rep = (SplitHost*)host_pinned(sizeof(SplitHost));
  }
  void release() {
    for (void* p : owned) dev_free(p);
    owned.clear();
    if (h_rep) host_unpin(h_rep);
    h_rep = nullptr;
  }
};

// device bytes WstWorkC::init(qmax, kmax) allocates
inline size_t wstc_bytes(ll qmax, ll kmax) {
  qmax = std::max<ll>(qmax, 1);
  kmax = std::max<ll>(std::min<ll>(kmax, CHOL_MAX / 2), 1);
  const ll qk = qmax * kmax;
  const ll np = chol_padded((int)(2 * kmax));
  return sizeof(zc) * (size_t)(2 * qk) +
         sizeof(double) * (size_t)(8 * qk + np * np + 2 * kmax + 64) +
         sizeof(unsigned) * 4 + sizeof(int) * 4 + sizeof(SvdOut);
}

// Warm-started split of complex theta (m x nt) at kept rank k; `warm` is B (k x nt) for
// 'R', A (m x k) for 'L'. Writes left (m x k) and right (k x nt) and returns true, or
// returns false (left / right undefined) when the warm start was not good enough. The
// host waits once; ev_end, when given, is recorded after the split's kernels. skip and solved: see wst_split
// (left and right are written directly, by kernels that return where skip is set).
inline bool wst_split_c(WstWorkC& W, RedScratch& red, const zc* theta, int m, int nt, char dir, int k,
                        const zc* warm, zc* left, zc* right, double& trunc_err, cudaStream_t s,
                        WstMode mode = WST_FULL, cudaEvent_t ev_end = nullptr, const int* skip = nullptr,
                        const std::function<void()>& solved = nullptr) {
  if (k > W.kmax || m > W.qmax || nt > W.qmax) throw std::runtime_error("wst_split_c: workspace too small");
  if (2 * std::max(m, nt) > 32 * COLNORM_MAX_CHUNKS) return false;  // longer columns take the exact split
  split_begin(W.status, W.out, k, s);
  // complex C (M x N) = op(A) op(B): ta / ca transpose / conjugate A, tb transposes B
  auto mulz = [&](bool ta, bool ca, const zc* A, ll lda, int M, int N, int Kd, const zc* B, ll ldb, bool tb,
                  zc* C, ll ldc, const int* no_write = nullptr) {
    Gemm<zc> g;
    g.ta = ta; g.ca = ca; g.tb = tb;
    g.M = M; g.N = N; g.K = Kd;
    g.A = A; g.lda = lda;
    g.B = B; g.ldb = ldb;
    g.C = C; g.ldc = ldc;
    g.skip = no_write;
    launch_gemm(g, s);
  };
  // real C = alpha op(A) op(B) + beta C on the embeddings
  auto mulr = [&](bool ta, const double* A, ll lda, int M, int N, int Kd, const double* B, ll ldb, double* C,
                  ll ldc, double alpha, double beta, const int* skip, const double* Cin = nullptr) {
    Gemm<double> g;
    g.ta = ta;
    g.M = M; g.N = N; g.K = Kd;
    g.A = A; g.lda = lda;
    g.B = B; g.ldb = ldb;
    g.C = C; g.ldc = ldc;
    g.alpha = alpha; g.beta = beta;
    g.skip = skip;
    g.Cin = Cin;
    launch_gemm(g, s);
  };
  const int k2 = 2 * k;
  const int ldS = chol_padded(k2);
  // Z (rows x k) -> dst: complex CholeskyQR on the embedding (unit columns, Gram matrix,
  // tiled Cholesky factor, row solve), then the even columns
  auto tri = [&](const zc* Z, ll rows, zc* dst) {
    embed_pairs(Z, rows, k, W.Z1, s);
    mulr(true, W.Z1, k2, k2, k2, (int)(2 * rows), W.Z1, k2, W.S, ldS, 1.0, 0.0, nullptr);
    chol_tiles(W.S, k2, ldS, W.S, ldS, W.status, 1e-10, 0.0, s, W.dscale);
    trsm_rows(W.Z1, 2 * rows, k2, W.S, ldS, W.Z2, W.status, s, W.dscale);
    extract_pairs(W.Z2, rows, k, dst, s);
  };
  // one Newton-Schulz step on the embedding of Z (rows x k) unless it is orthonormal already, result
  // into dst; a split whose bound on the step's result (ns_check) is above the tolerance reports a failure
  auto polish = [&](const zc* Z, ll rows, zc* dst, const int* skip_dst) {
    const ll r2 = 2 * rows;
    embed_pairs(Z, rows, k, W.Z1, s);
    mulr(true, W.Z1, k2, k2, k2, (int)r2, W.Z1, k2, W.S, k2, 1.0, 0.0, nullptr);
    ns_check(W.S, k2, W.out, 4e-16 * (double)r2, W.part, W.counter, s);
    mulr(false, W.Z1, k2, (int)r2, k2, k2, W.S, k2, W.Z2, k2, -0.5, 1.5, &W.out->ns_done, W.Z1);
    extract_pairs(W.Z2, rows, k, dst, s, skip_dst);
  };
  const zc* kept = nullptr;
  ll nkept = 0;
  if (dir == 'R') {
    if (mode != WST_RESUME) {
      mulz(false, true, warm, nt, k, m, nt, theta, nt, true, W.Yb, m);  // conj(B) theta^T (k x m)
      transpose<zc>(W.Yb, W.Ya, (ll)k, (ll)m, s);                          // theta B^H (m x k)
      tri(W.Ya, m, W.Yb);                                                  // U1
    } else {
      DMRG2_CUDA(cudaMemcpyAsync(W.Yb, left, sizeof(zc) * (size_t)m * k, cudaMemcpyDeviceToDevice, s));  // U1
    }
    if (mode != WST_SHORT) {
      mulz(true, true, theta, nt, nt, k, m, W.Yb, k, false, W.Ya, k);  // theta^H U1
      tri(W.Ya, nt, W.Yb);                                             // V1
      mulz(false, false, theta, nt, m, k, nt, W.Yb, k, false, W.Ya, k);  // theta V1
      tri(W.Ya, m, W.Yb);                                                // U2
    }
    polish(W.Yb, m, left, skip);
    mulz(true, true, left, k, k, nt, m, theta, nt, false, right, nt, skip);  // right = U^H theta
    kept = right;
    nkept = (ll)k * nt;
  } else {
    if (mode != WST_RESUME) {
      mulz(true, true, theta, nt, nt, k, m, warm, k, false, W.Ya, k);  // theta^H A
      tri(W.Ya, nt, W.Yb);                                             // V1
    } else {
      DMRG2_CUDA(cudaMemcpyAsync(W.Yb, W.Ya, sizeof(zc) * (size_t)nt * k, cudaMemcpyDeviceToDevice, s));
    }
    if (mode != WST_SHORT) {
      mulz(false, false, theta, nt, m, k, nt, W.Yb, k, false, W.Ya, k);  // theta V1
      tri(W.Ya, m, W.Yb);                                                // U1
      mulz(true, true, theta, nt, nt, k, m, W.Yb, k, false, W.Ya, k);    // theta^H U1
      tri(W.Ya, nt, W.Yb);                                               // V2
    }
    polish(W.Yb, nt, W.Ya, nullptr);                                     // V in Ya
    transpose_conj<zc>(W.Ya, k, nt, k, right, s, skip);                  // right = V^H
    mulz(false, false, theta, nt, m, k, nt, W.Ya, k, false, left, k, skip);  // left = theta V
    kept = left;
    nkept = (ll)m * k;
  }
  split_finish(theta, (ll)m * nt, kept, nkept, W.status, W.out, W.h_rep, red, s);
  if (ev_end) DMRG2_CUDA(cudaEventRecord(ev_end, s));
  DMRG2_CUDA(cudaStreamSynchronize(s));
  if (solved) solved();
  const SplitHost& rep = *W.h_rep;
  if (rep.failed || !std::isfinite(rep.theta2) || !std::isfinite(rep.kept2)) return false;
  trunc_err = std::max(rep.theta2 - rep.kept2, 0.0);
  return true;
}

}  // namespace dmrg2
