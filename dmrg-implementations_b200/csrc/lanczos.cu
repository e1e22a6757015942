// Device-resident Lanczos with full reorthogonalisation.
//
// Replaces the reference's Lanczos loop (gpu-rocm/dmrg2-gpu/src/dmrg2_gpu_impl.h:971-1160):
// the BLAS-1/2 calls (dot, axpy, two reorthogonalisation GEMVs, nrm2, scal) and
// the per-iteration scalar kernels become three fused streaming kernels per
// iteration that read every Krylov vector with coalesced loads, reduce with
// warp shuffles, and finalise in the last block to arrive (no host sync). The
// last block of the third kernel also solves the tridiagonal eigenproblem for
// its lowest eigenvalue (multisection on the leading minors), applies the |dE| stop
// rule and, once done, computes the Ritz coefficients by inverse iteration, so
// the host never copies alpha/beta back. Vectors that fit the fused step kernel's
// shared memory (every n below about 1.8M doubles) take one launch per Krylov step
// instead (lz_step_kernel).
#include <cooperative_groups.h>

#include <algorithm>

#include "gemm.cuh"
#include "kernels.cuh"

namespace dmrg2 {

static constexpr int MAX_CHUNK = 2048;

int red_blocks(ll n) { return std::max(vec_blocks(n), 2 * STEP_BLOCKS); }

int vec_blocks(ll n) {
  ll nb = (n + VEC_THREADS - 1) / VEC_THREADS;
  if (nb > 592) nb = 592;
  if (nb < 1) nb = 1;
  ll ch = (n + nb - 1) / nb;
  if (ch > MAX_CHUNK) nb = (n + MAX_CHUNK - 1) / MAX_CHUNK;
  return (int)nb;
}

__device__ inline double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ inline double block_sum(double v, double* sh) {
  v = warp_sum(v);
  int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) sh[w] = v;
  __syncthreads();
  double r = 0.0;
  if (threadIdx.x < 32) {
    r = (threadIdx.x < (blockDim.x >> 5)) ? sh[threadIdx.x] : 0.0;
    r = warp_sum(r);
  }
  __syncthreads();
  if (threadIdx.x == 0) sh[0] = r;
  __syncthreads();
  r = sh[0];
  __syncthreads();
  return r;
}

__device__ inline bool arrive_last(unsigned* counter, unsigned nblk) {
  __shared__ int am_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) am_last = (atomicAdd(counter, 1u) == nblk - 1) ? 1 : 0;
  __syncthreads();
  if (am_last) __threadfence();
  return am_last != 0;
}

// ----------------------------------------------------------------------------
// tridiagonal helpers (block-wide / single thread)
// ----------------------------------------------------------------------------
// Lowest eigenvalue of the symmetric tridiagonal (a, b) of order k <= KRYLOV_CAP, a and b in
// shared memory; hint is the lowest eigenvalue of the leading block of order k - 1 (unused for
// k = 1). One warp; every lane gets the result. sa, sb: KRYLOV_CAP + 8 doubles of shared memory each.
//
// Multisection with two trial points per lane. x lies below the lowest eigenvalue exactly
// when every leading principal minor of T - x is positive, so a trial is the minors'
// recurrence p_i = (a_i - x) p_(i-1) - b_(i-1)^2 p_(i-2) and one sign test per step: one
// multiply and one fused multiply-add on the dependent chain, no division. T is scaled by a
// power of two to entries of at most 1 and the pair (p_i, p_(i-1)) is rescaled by a power of
// two before it can underflow, so the signs are those of the unscaled recurrence. One warp with
// two chains a lane just hides the chain's latency; a block of 512 trial points instead is
// bound by the FP64 pipe (12,300 cycles at k = 10, 23,100 at k = 25). The trial points
// are ordered, so the count of positive ones is the position of the eigenvalue.
// Bracket: interlacing gives lambda_k <= hint, Weyl's bound
// lambda_k >= min(hint, a_k) - |b_(k-1)|; the slack covers the rounding in hint.
__device__ double tridiag_lowest(const double* a, const double* b, int k, double hint, double* sa, double* sb) {
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  if (k == 1) return a[0];
  double mx = 0.0, lo = 1e300, hi = 1e300;
  bool bad = false;  // a NaN or infinity (fmax and fmin would drop a NaN)
  for (int i = lane; i < k; i += 32) {
    bad = bad || !isfinite(a[i]) || (i < k - 1 && !isfinite(b[i]));
    const double l = i > 0 ? fabs(b[i - 1]) : 0.0, r = i < k - 1 ? fabs(b[i]) : 0.0;
    mx = fmax(mx, fabs(a[i]) + l + r);
    lo = fmin(lo, a[i] - l - r);
    hi = fmin(hi, a[i]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    mx = fmax(mx, __shfl_xor_sync(FULL, mx, o));
    lo = fmin(lo, __shfl_xor_sync(FULL, lo, o));
    hi = fmin(hi, __shfl_xor_sync(FULL, hi, o));
  }
  if (__any_sync(FULL, bad)) return nan("");
  if (!(mx > 0.0)) return 0.0;
  if (isfinite(hint) && fabs(hint) < 1e299) {
    lo = fmax(lo, fmin(hint, a[k - 1]) - fabs(b[k - 2]));
    hi = fmin(hi, hint);
  }
  int e = 0;
  frexp(mx, &e);
  // (sb[i] belongs to step i; steps beyond k - 1 up to a whole group of 8 keep every sign: the
  // trial points are below 4 after the scaling)
  const int kp = ((k + 6) / 8) * 8 + 1;
  for (int i = lane; i < kp; i += 32) {
    sa[i] = i < k ? ldexp(a[i], -e) : 8.0;
    const double bi = (i > 0 && i < k) ? ldexp(b[i - 1], -e) : 0.0;
    sb[i] = -bi * bi;
  }
  lo = ldexp(lo, -e) - 4e-15;
  hi = ldexp(hi, -e) + 4e-15;
  __syncwarp();
  for (int round = 0; round < 16; ++round) {
    const double step = (hi - lo) * (1.0 / 65.0);
    const double x0 = fma(step, (double)(lane + 1), lo), x1 = fma(step, (double)(lane + 33), lo);
    double m0 = 1.0, m1 = 1.0, p0 = sa[0] - x0, p1 = sa[0] - x1;
    bool pos0 = p0 > 0.0, pos1 = p1 > 0.0;
    for (int i0 = 1; i0 < kp; i0 += 8) {
      double ai[8], bi[8];  // loaded ahead of the chain
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        ai[u] = sa[i0 + u];
        bi[u] = sb[i0 + u];
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const double q0 = fma(ai[u] - x0, p0, bi[u] * m0), q1 = fma(ai[u] - x1, p1, bi[u] * m1);
        m0 = p0; p0 = q0;
        m1 = p1; p1 = q1;
        pos0 = pos0 && (p0 > 0.0);
        pos1 = pos1 && (p1 > 0.0);
      }
      if (fmax(fabs(p0), fabs(m0)) < 0x1p-300) { p0 *= 0x1p+300; m0 *= 0x1p+300; }
      if (fmax(fabs(p1), fabs(m1)) < 0x1p-300) { p1 *= 0x1p+300; m1 *= 0x1p+300; }
    }
    const int n = __popc(__ballot_sync(FULL, pos0)) + __popc(__ballot_sync(FULL, pos1));
    const double l2 = n > 0 ? fma(step, (double)n, lo) : lo;
    if (n < 64) hi = fma(step, (double)(n + 1), lo);
    lo = l2;
    if (hi - lo <= 4e-16 * fmax(fabs(lo), fabs(hi)) + 1e-300) break;
  }
  return ldexp(0.5 * (lo + hi), e);
}

// Eigenvector of the tridiagonal (a, b) for eigenvalue lam by inverse iteration
// with partial pivoting (single thread; k <= KRYLOV_CAP).
__device__ void tridiag_vector(const double* a, const double* b, int k, double lam, double* y,
                               double* work) {
  double* u0 = work;
  double* u1 = work + KRYLOV_CAP;
  double* u2 = work + 2 * KRYLOV_CAP;
  double* l = work + 3 * KRYLOV_CAP;
  double* sw = work + 4 * KRYLOV_CAP;
  double scale = 0.0;
  for (int i = 0; i < k; ++i) scale = fmax(scale, fabs(a[i]) + (i < k - 1 ? fabs(b[i]) : 0.0));
  const double tiny = 1e-15 * fmax(scale, 1e-300);
  for (int i = 0; i < k; ++i) {
    u0[i] = a[i] - lam;
    u1[i] = (i < k - 1) ? b[i] : 0.0;
    u2[i] = 0.0;
  }
  for (int i = 0; i < k - 1; ++i) {
    double s = b[i];
    if (fabs(u0[i]) >= fabs(s)) {
      if (u0[i] == 0.0) u0[i] = tiny;
      double m = s / u0[i];
      u0[i + 1] -= m * u1[i];
      l[i] = m;
      sw[i] = 0.0;
    } else {
      double m = u0[i] / s;
      double old_u1i = u1[i];
      u0[i] = s;
      u1[i] = u0[i + 1];
      u2[i] = u1[i + 1];
      u0[i + 1] = old_u1i - m * u1[i];
      u1[i + 1] = -m * u2[i];
      l[i] = m;
      sw[i] = 1.0;
    }
  }
  if (u0[k - 1] == 0.0) u0[k - 1] = tiny;
  for (int i = 0; i < k; ++i) y[i] = 1.0;
  for (int it = 0; it < 3; ++it) {
    for (int i = 0; i < k - 1; ++i) {
      if (sw[i] != 0.0) { double t = y[i]; y[i] = y[i + 1]; y[i + 1] = t; }
      y[i + 1] -= l[i] * y[i];
    }
    for (int i = k - 1; i >= 0; --i) {
      double v = y[i];
      if (i + 1 < k) v -= u1[i] * y[i + 1];
      if (i + 2 < k) v -= u2[i] * y[i + 2];
      double d = u0[i];
      if (fabs(d) < tiny) d = (d < 0 ? -tiny : tiny);
      y[i] = v / d;
    }
    double nrm = 0.0;
    for (int i = 0; i < k; ++i) nrm += y[i] * y[i];
    nrm = sqrt(nrm);
    if (!(nrm > 0.0) || !isfinite(nrm)) {
      for (int i = 0; i < k; ++i) y[i] = (i == 0) ? 1.0 : 0.0;
      break;
    }
    for (int i = 0; i < k; ++i) y[i] /= nrm;
  }
}

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// The end of a Krylov step (the first warp of a block): the lowest Ritz value of the k-step
// matrix (a, b) (shared memory), the stop rule and, once done, the Ritz coefficients. Returns
// whether the solve is done.
struct StepState {
  double a[KRYLOV_CAP], b[KRYLOV_CAP], y[KRYLOV_CAP], work[5 * KRYLOV_CAP];
};
__device__ bool lz_finish_step(LanczosDev* st, StepState& sh, int k, int kmax, double e_prev, double tol) {
  const double lam = tridiag_lowest(sh.a, sh.b, k, e_prev, sh.work, sh.work + 2 * KRYLOV_CAP);
  const bool conv = (k >= 3) && (fabs(lam - e_prev) < tol);
  const bool brk = sh.b[k - 1] < 1e-14;
  const bool done = conv || brk || k >= kmax;
  __syncwarp();  // the work area is free again
  if (threadIdx.x == 0) {
    st->e_cur = lam;
    st->e_prev = lam;
    if (done) {
      st->converged = (conv || brk) ? 1 : 0;
      st->n_iter = k;
      tridiag_vector(sh.a, sh.b, k, lam, sh.y, sh.work);
      for (int i = 0; i < k; ++i) st->ritz[i] = sh.y[i];
      __threadfence();
      st->done = 1;
    }
  }
  return done;
}

// ----------------------------------------------------------------------------
// one Krylov step in one launch
// ----------------------------------------------------------------------------
// A step's vectors live in the L2 (2.1 MB each at chi = 256), so the passes above are bound
// by their latency: three launches, each with a grid-wide last-block reduction that the next
// one waits for, then a normalisation and a loop kernel. Here one grid keeps its slice of w in
// shared memory through the whole step and meets at two barriers:
//   coef0 = V^H w | w -= V coef0, coef1 = V^H w, |w|^2 | w -= V coef1, v_(j+1) = w / |w|
// (the same classical Gram-Schmidt, applied twice). The norm after the second projection
// follows from the one before it, |w'|^2 - |coef1|^2 (V is orthonormal to rounding, coef1 is
// the rounding left by the first projection, a few eps |H|; the difference is relatively good to
// eps (1 + |coef1|^2 / beta^2), and beta is above 1e-14 or the solve ends, so |H| would have to
// reach 1e5 before a beta of pure rounding noise lost half its digits), so no third barrier is
// needed, and block 0
// solves the tridiagonal problem while the others finish their slices. Every block sums the
// partial products itself, in the same fixed order.
// The barrier: up to LS_CLUSTER blocks are one thread-block cluster (hardware barrier);
// beyond, a cooperative launch of one block per SM with a counter barrier (bounded), except
// where Jacobi kernels of other streams would keep it waiting (cooperative_step_blocks).
// The staged basis is read four times a step, so a slice costs one pass over the L2.
// Per step at chi = 256 (n = 262,144, 3 Krylov vectors) 31 us in five launches before and
// 15 us now; in a 12-site chain at chi = 64 (n <= 16,384) 33 us before, 16 us now.
constexpr int LS_THREADS = 512;
constexpr int LS_WARPS = LS_THREADS / 32;
constexpr int LS_CLUSTER = 16;
constexpr int LS_PUSH = 32;                    // values exchanged through the cluster's shared memory at most
constexpr size_t LS_SMEM_W = 96 * 1024;        // slice of w per block at most
// w and the staged basis per block: one block per SM of the cooperative grid; a cluster leaves room
// for a second block, since the clusters of concurrent solves share the SMs
constexpr size_t LS_SMEM_GRID = 176 * 1024, LS_SMEM_CLUSTER = 72 * 1024;
constexpr long long LS_SPIN = 1ll << 22;       // barrier polls before a block gives up (seconds)
constexpr long long LS_SPIN_TEST = 1ll << 14;  // the same under the unsignalled-wait test hook

struct StepGrid {
  int blocks = 0;  // 0: the vector does not fit, the streaming passes run
  int chunk = 0;
  bool cluster = false;
};

template <typename T>
static StepGrid step_grid(ll n, int coop) {
  // slices of 512 elements (one per thread) until 16 blocks are reached, which a cluster holds up
  // to 2048 elements each; then one block per SM (`coop` of them at most)
  StepGrid g;
  const ll cl_max = 2048 / (ll)(sizeof(T) / sizeof(double));
  ll nb = (n + LS_THREADS - 1) / LS_THREADS;
  g.cluster = n <= LS_CLUSTER * cl_max;
  const ll cap = g.cluster ? LS_CLUSTER : std::min(coop, STEP_BLOCKS);
  if (cap < 1) return g;
  if (nb > cap) nb = cap;
  const ll ch = ((n + nb - 1) / nb + 1) & ~1ll;  // even: 16-byte slices
  if (ch * (ll)sizeof(T) > (ll)LS_SMEM_W) return g;
  g.blocks = (int)nb;
  g.chunk = (int)ch;
  return g;
}

__device__ __forceinline__ unsigned ld_acquire_gpu(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// all blocks of the grid meet; false when this block's bounded wait ran out (unsignalled: the test
// hook, the last block waits for one more than there are). The caller records it in st->gave_up: a
// single block that went on without the others has wrong sums, whoever it is.
template <bool CL>
__device__ __forceinline__ bool step_barrier(unsigned* bar, int unsignalled) {
  if constexpr (CL) {
    cooperative_groups::this_cluster().sync();
    return true;
  } else {
    __syncthreads();
    bool ok = true;
    if (threadIdx.x == 0) {
      const bool hook = unsignalled && blockIdx.x == gridDim.x - 1;
      const unsigned need = gridDim.x + (hook ? 1u : 0u);
      const long long spin = hook ? LS_SPIN_TEST : LS_SPIN;
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
      long long it = 0;
      while (ld_acquire_gpu(bar) < need && ++it < spin) {
      }
      ok = it < spin;
    }
    return __syncthreads_and(ok ? 1 : 0) != 0;
  }
}

// warp sums of eight values per lane, out[0 .. cnt-1]: the sums share their shuffles (nine instead
// of forty; the value index follows lane bits 4, 3 and 2)
__device__ __forceinline__ void warp_sum8(double (&v)[8], int lane, double* out, int cnt) {
  const bool h = lane & 16, g = lane & 8, f = lane & 4;
  double a[4], b[2];
#pragma unroll
  for (int i = 0; i < 4; ++i) a[i] = (h ? v[4 + i] : v[i]) + __shfl_xor_sync(0xffffffffu, h ? v[i] : v[4 + i], 16);
#pragma unroll
  for (int i = 0; i < 2; ++i) b[i] = (g ? a[2 + i] : a[i]) + __shfl_xor_sync(0xffffffffu, g ? a[i] : a[2 + i], 8);
  double c = (f ? b[1] : b[0]) + __shfl_xor_sync(0xffffffffu, f ? b[0] : b[1], 4);
  c += __shfl_xor_sync(0xffffffffu, c, 2);
  c += __shfl_xor_sync(0xffffffffu, c, 1);
  const int idx = (h ? 4 : 0) + (g ? 2 : 0) + (f ? 1 : 0);
  if ((lane & 3) == 0 && idx < cnt) out[idx] = c;
}

// A block's slice of the Krylov basis: the first nc vectors staged in shared memory (they are
// read four times in a step), the others read from the L2.
template <typename T>
struct BasisSlice {
  const T* sm;  // [nc][chunk]
  int nc, chunk;
  const T* g;   // vector i at g + i n
  ll n;
};

// <v_i, ws> for u < m vectors from i0 (stride ld), this thread's elements, into acc
template <typename T, int U, bool FULL>
__device__ __forceinline__ void dots_group(const T* v0, ll ld, int m, const T* ws, int len, double (&acc)[8]) {
  constexpr bool CPLX = ST<T>::cplx;
#pragma unroll 2
  for (int x = threadIdx.x; x < len; x += LS_THREADS) {
    const T wv = ws[x];
    T v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = (FULL || u < m) ? v0[u * ld + x] : ST<T>::zero();
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const T p = ST<T>::cmul(v[u], wv);
      if constexpr (CPLX) {
        acc[2 * u] += p.re;
        acc[2 * u + 1] += p.im;
      } else {
        acc[u] += p;
      }
    }
  }
}

// per-warp sums of <v_i, ws>, i < nv (c = i, or 2 i and 2 i + 1 for complex data), into
// wsum[warp][c]
template <typename T>
__device__ __forceinline__ void slice_dots(const BasisSlice<T>& V, int nv, const T* ws, int len, double* wsum,
                                           int wpitch) {
  constexpr bool CPLX = ST<T>::cplx;
  constexpr int U = CPLX ? 4 : 8;  // the vectors of one eight-value reduction
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int i0 = 0; i0 < nv;) {
    double acc[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    const bool in_sm = i0 < V.nc;
    const int m = min(U, (in_sm ? V.nc : nv) - i0);
    if (in_sm) {
      const T* v0 = V.sm + i0 * V.chunk;
      if (m == U) dots_group<T, U, true>(v0, V.chunk, m, ws, len, acc);
      else dots_group<T, U, false>(v0, V.chunk, m, ws, len, acc);
    } else {
      const T* v0 = V.g + (ll)i0 * V.n;
      if (m == U) dots_group<T, U, true>(v0, V.n, m, ws, len, acc);
      else dots_group<T, U, false>(v0, V.n, m, ws, len, acc);
    }
    warp_sum8(acc, lane, wsum + warp * wpitch + (CPLX ? 2 * i0 : i0), CPLX ? 2 * m : m);
    i0 += m;
  }
}

// ws -= sum_i c_i v_i on this thread's elements; returns its share of |ws|^2
template <typename T>
__device__ __forceinline__ double slice_update(const BasisSlice<T>& V, int nv, T* ws, int len, const double* c) {
  constexpr bool CPLX = ST<T>::cplx;
  auto coef = [&](int i) {
    if constexpr (CPLX) return mkz(c[2 * i], c[2 * i + 1]);
    else return c[i];
  };
  double ww = 0.0;
  for (int x = threadIdx.x; x < len; x += LS_THREADS) {
    T v = ws[x];
    int i = 0;
#pragma unroll 4
    for (; i < V.nc; ++i) v = v - ST<T>::mul(coef(i), V.sm[i * V.chunk + x]);
#pragma unroll 8
    for (; i < nv; ++i) v = v - ST<T>::mul(coef(i), V.g[(ll)i * V.n + x]);
    ws[x] = v;
    ww += ST<T>::abs2(v);
  }
  return ww;
}

// The grid's sums of `ncoef` values from each block's per-warp sums, into dst (shared memory,
// every block, the same order everywhere). A cluster with few values pushes them into every
// block's shared memory (xch: LS_CLUSTER x ncoef there) ahead of the hardware barrier; otherwise they
// go through part[c][block] and the grid barrier. Returns false when a bounded wait ran out.
template <bool CL>
__device__ __forceinline__ bool exchange_sums(const double* wsum, int wpitch, int ncoef, double* part, unsigned* bar,
                                              double* xch, double* dst, int unsignalled) {
  const int tid = threadIdx.x, lane = tid & 31, nblk = gridDim.x;
  const bool push = CL && ncoef <= LS_PUSH;
  __syncthreads();
  for (int c = tid; c < ncoef; c += LS_THREADS) {
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < LS_WARPS; ++w) s += wsum[w * wpitch + c];
    if (push) {
      cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
      for (int b = 0; b < nblk; ++b) cl.map_shared_rank(xch, b)[blockIdx.x * ncoef + c] = s;
    } else {
      part[(ll)c * nblk + blockIdx.x] = s;
    }
  }
  const bool ok = step_barrier<CL>(bar, unsignalled);
  if (push) {
    for (int c = tid; c < ncoef; c += LS_THREADS) {
      double s = 0.0;
      for (int b = 0; b < nblk; ++b) s += xch[b * ncoef + c];
      dst[c] = s;
    }
  } else {
    for (int c = tid >> 5; c < ncoef; c += LS_WARPS) {
      double s = 0.0;
      for (int b = lane; b < nblk; b += 32) s += __ldcg(part + (ll)c * nblk + b);
      s = warp_sum(s);
      if (lane == 0) dst[c] = s;
    }
  }
  __syncthreads();
  return ok;
}

// asynchronous copy of `count` elements from global to shared memory (committed by the caller);
// vec: both are 16-byte aligned
template <typename T>
__device__ __forceinline__ void copy_async(T* dst, const T* src, int count, bool vec) {
  if (vec && sizeof(T) == 8) {
    for (int x = 2 * threadIdx.x; x + 1 < count; x += 2 * LS_THREADS) cp_async_16(dst + x, src + x, true);
    if ((count & 1) && threadIdx.x == 0) cp_async_8(dst + count - 1, src + count - 1, true);
  } else {
    for (int x = threadIdx.x; x < count; x += LS_THREADS) {
      if constexpr (sizeof(T) == 16) cp_async_16(dst + x, src + x, true);
      else cp_async_8(dst + x, src + x, true);
    }
  }
}

// loop != 0: the device-looped solve (the Krylov index is st->j, cur gets v_(j+1), the matvec's
// time since st->t_mark is added to st->mv_ns, and block 0 advances the index and sets the
// loop condition of handle h); else nv = j + 1 is given and host_done, when given, gets the
// done flag (page-locked host memory). ncache: vectors of the basis staged in shared memory.
template <typename T, bool CL>
__global__ void __launch_bounds__(LS_THREADS, 1)
    lz_step_kernel(T* V, int nv, ll n, const T* w, T* cur, LanczosDev* st, double* part, int kmax, int chunk,
                   int ncache, int loop, cudaGraphConditionalHandle h, volatile int* host_done, int unsignalled) {
  extern __shared__ __align__(16) unsigned char ls_smem[];
  __shared__ StepState sh;
  __shared__ double csum[2 * KRYLOV_CAP + 1];
  __shared__ double xch[CL ? 2 * LS_CLUSTER * LS_PUSH : 1];
  constexpr int CV = ST<T>::cplx ? 2 : 1;
  const int tid = threadIdx.x;
  const bool lead = blockIdx.x == 0;
  pdl_wait();
  // one thread per block reads the state (every warp of 148 blocks reading these words took 2.6 us:
  // they are one L2 line), all fields in one round trip
  __shared__ int s_j, s_guard, s_done;
  __shared__ double s_eprev, s_tol;
  if (tid == 0) {
    s_done = *((volatile int*)&st->done) | *((volatile int*)&st->gave_up);
    s_j = *((volatile int*)&st->j);
    s_guard = *((volatile int*)&st->guard);
    s_eprev = *((volatile double*)&st->e_prev);
    s_tol = *((volatile double*)&st->tol);
  }
  __syncthreads();
  const int j = s_j, guard = s_guard;
  // set by an earlier launch, so the same for every block (or by a block of this one that gave up
  // waiting for this block: the solve is lost either way)
  if (s_done) {
    if (lead && tid == 0) {
      if (host_done) *host_done = 1;
      if (loop) cudaGraphSetConditional(h, 0u);
    }
    return;
  }
  if (loop) {
    nv = j + 1;
    if (lead && tid == 0) st->mv_ns += global_ns() - st->t_mark;
  }
  const int nc = CV * nv, wpitch = nc + 1;
  const ll x0 = (ll)blockIdx.x * chunk;
  const int len = (int)max((ll)0, min((ll)chunk, n - x0));
  T* ws = reinterpret_cast<T*>(ls_smem);
  T* vs = ws + chunk;                                                // [ncache][chunk]
  double* wsum = reinterpret_cast<double*>(vs + (ll)ncache * chunk);  // LS_WARPS x wpitch
  const BasisSlice<T> B{vs, min(nv, ncache), chunk, V + x0, n};
  {
    const bool vec = ((n | chunk) & 1) == 0;  // slices and vectors start on 16 bytes
    copy_async(ws, w + x0, len, vec);
    for (int i = 0; i < B.nc; ++i) copy_async(vs + i * chunk, V + (ll)i * n + x0, len, vec);
    cp_async_commit();
  }
  if (lead)
    for (int i = tid; i < nv - 1; i += LS_THREADS) {
      sh.a[i] = st->alpha[i];
      sh.b[i] = st->beta[i];
    }
  if (lead && tid == 0 && !CL) {  // before anyone passes the first barrier
    volatile unsigned* bar = st->bar;
    bar[1] = bar[2] = bar[3] = 0u;  // the last step's, and the start's
  }
  if (CL) cooperative_groups::this_cluster().sync();  // the peers run: their shared memory may be written
  cp_async_wait<0>();
  __syncthreads();
  slice_dots<T>(B, nv, ws, len, wsum, wpitch);
  bool ok = exchange_sums<CL>(wsum, wpitch, nc, part, &st->bar[0], xch, csum, unsignalled);
  const double a0 = csum[CV * (nv - 1)];
  {
    const double ww = warp_sum(slice_update<T>(B, nv, ws, len, csum));
    slice_dots<T>(B, nv, ws, len, wsum, wpitch);
    if ((tid & 31) == 0) wsum[(tid >> 5) * wpitch + nc] = ww;
  }
  ok = exchange_sums<CL>(wsum, wpitch, nc + 1, part + (ll)nc * gridDim.x, &st->bar[1],
                         xch + (CL ? LS_CLUSTER * LS_PUSH : 0), csum, unsignalled) && ok;
  if (!ok && tid == 0) *((volatile int*)&st->gave_up) = 1;
  double c2 = 0.0;
  for (int c = 0; c < nc; ++c) c2 += csum[c] * csum[c];
  const double nrm2 = fmax(csum[nc] - c2, 0.0);
  if (nv < kmax) {
    slice_update<T>(B, nv, ws, len, csum);
    const double inv = nrm2 > 0.0 ? 1.0 / sqrt(nrm2) : 0.0;
    T* vn = V + (ll)nv * n + x0;
    for (int x = tid; x < len; x += LS_THREADS) {
      const T v = ST<T>::scale(inv, ws[x]);
      vn[x] = v;
      if (cur) cur[x0 + x] = v;
    }
  }
  if (!lead || tid >= 32) return;
  const double beta = sqrt(nrm2);
  if (tid == 0) {
    sh.a[nv - 1] = st->alpha[nv - 1] = a0 + csum[CV * (nv - 1)];
    sh.b[nv - 1] = st->beta[nv - 1] = beta;
    st->nrm2 = nrm2;
    if (!CL) *((volatile unsigned*)&st->bar[0]) = 0u;  // everyone is past the first barrier
    if (!ok) {  // a barrier gave up: end the solve without a result
      st->n_iter = 0;
      st->done = 1;
    }
  }
  __syncwarp();
  const bool done = ok ? lz_finish_step(st, sh, nv, kmax, s_eprev, s_tol) : true;
  if (tid == 0) {
    if (host_done) *host_done = done ? 1 : 0;
    if (loop) {
      st->guard = guard + 1;
      if (!done) st->j = j + 1;
      st->t_mark = global_ns();
      cudaGraphSetConditional(h, (!done && guard + 1 < kmax) ? 1u : 0u);
    }
  }
}

__device__ inline double hash_uniform(unsigned long long x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  x ^= x >> 31;
  return (double)(x >> 11) * (1.0 / 9007199254740992.0) * 2.0 - 1.0;
}

// start of a solve: |theta|^2 (theta replaced by a seeded random vector where it is ~0 or not a
// number), the solver state, v_0 = theta / |theta| into V and cur
template <typename T, bool CL>
__global__ void __launch_bounds__(LS_THREADS, 1)
    lz_start_kernel(T* theta, T* v0, T* cur, ll n, LanczosDev* st, double* part, unsigned seed,
                    const unsigned* seed_host, double tol, int kmax, int chunk, int unsignalled) {
  __shared__ double wsum[LS_WARPS], xch_s[2][LS_CLUSTER], tot;
  const int tid = threadIdx.x;
  const bool lead = blockIdx.x == 0;
  pdl_wait();
  if (CL) cooperative_groups::this_cluster().sync();  // the peers run: their shared memory may be written
  const ll x0 = (ll)blockIdx.x * chunk;
  const int len = (int)max((ll)0, min((ll)chunk, n - x0));
  auto norm = [&](double* p, unsigned* bar, double* xch) {
    double ww = 0.0;
    for (int x = tid; x < len; x += LS_THREADS) ww += ST<T>::abs2(theta[x0 + x]);
    ww = warp_sum(ww);
    if ((tid & 31) == 0) wsum[tid >> 5] = ww;
    return exchange_sums<CL>(wsum, 1, 1, p, bar, xch, &tot, unsignalled);
  };
  if (lead && tid == 0 && !CL) *((volatile unsigned*)&st->bar[4]) = 0u;  // the last solve's
  bool ok = norm(part, &st->bar[2], xch_s[0]);
  const bool tiny = !(tot >= 1e-28);
  if (tiny) {
    if (seed_host) seed = *((volatile const unsigned*)seed_host);
    for (int e = tid; e < len; e += LS_THREADS) {
      const ll x = x0 + e;
      const double r = hash_uniform(((unsigned long long)seed << 32) ^ (unsigned long long)(2 * x));
      const double i = ST<T>::cplx ? hash_uniform(((unsigned long long)seed << 32) ^ (2 * x + 1)) : 0.0;
      theta[x] = ST<T>::make(r, i);
    }
    __syncthreads();  // tot is read by every thread before the second sum replaces it
    ok = norm(part + gridDim.x, &st->bar[3], xch_s[1]) && ok;
  }
  const double inv = 1.0 / sqrt(tot);
  for (int x = tid; x < len; x += LS_THREADS) {
    const T v = ST<T>::scale(inv, theta[x0 + x]);
    v0[x0 + x] = v;
    if (cur) cur[x0 + x] = v;
  }
  if (!ok && tid == 0) *((volatile int*)&st->gave_up) = 1;
  if (lead && tid == 0) {
    st->nrm2 = tot;
    st->randomized = tiny ? 1 : 0;
    st->done = ok ? 0 : 1;
    st->converged = 0;
    st->n_iter = 0;
    st->e_prev = 1e300;
    st->e_cur = 0.0;
    st->tol = tol;
    st->kmax = kmax;
    st->j = 0;
    st->guard = 0;
    st->t_mark = global_ns();
    st->mv_ns = 0ull;
  }
}

__device__ __forceinline__ void lz_report(const LanczosDev* st, LanczosHost* host) {
  volatile LanczosHost* h = host;
  h->e_cur = st->e_cur;
  h->mv_ns = st->mv_ns;
  h->done = st->done;
  h->converged = st->converged;
  h->n_iter = st->n_iter;
  h->guard = st->guard;
  if (st->gave_up) h->gave_up = 1;
}
__global__ void lz_report_kernel(const LanczosDev* st, LanczosHost* host) { lz_report(st, host); }

// end of a solve: out = sum_i ritz_i v_i, normalised, and the report to the host
template <typename T, bool CL>
__global__ void __launch_bounds__(LS_THREADS, 1)
    lz_ritz_norm_kernel(const T* V, ll n, T* out, LanczosDev* st, double* part, LanczosHost* host, int chunk,
                        int unsignalled) {
  extern __shared__ __align__(16) unsigned char ls_smem[];
  __shared__ double r[KRYLOV_CAP], wsum[LS_WARPS], xch[LS_CLUSTER], tot;
  const int tid = threadIdx.x;
  pdl_wait();
  const int k = st->n_iter;
  if (CL) cooperative_groups::this_cluster().sync();  // the peers run: their shared memory may be written
  if (blockIdx.x == gridDim.x - 1 && tid == 0) lz_report(st, host);
  T* ws = reinterpret_cast<T*>(ls_smem);
  const ll x0 = (ll)blockIdx.x * chunk;
  const int len = (int)max((ll)0, min((ll)chunk, n - x0));
  for (int i = tid; i < k; i += LS_THREADS) r[i] = st->ritz[i];
  __syncthreads();
  double ww = 0.0;
  for (int x = tid; x < len; x += LS_THREADS) {
    T acc = ST<T>::zero();
#pragma unroll 4
    for (int i = 0; i < k; ++i) acc = acc + ST<T>::scale(r[i], V[(ll)i * n + x0 + x]);
    ws[x] = acc;
    ww += ST<T>::abs2(acc);
  }
  ww = warp_sum(ww);
  if ((tid & 31) == 0) wsum[tid >> 5] = ww;
  if (!exchange_sums<CL>(wsum, 1, 1, part, &st->bar[4], xch, &tot, unsignalled) && tid == 0) {
    *((volatile int*)&st->gave_up) = 1;
    *((volatile int*)&host->gave_up) = 1;
  }
  const double inv = tot > 0.0 ? 1.0 / sqrt(tot) : 0.0;
  for (int x = tid; x < len; x += LS_THREADS) out[x0 + x] = ST<T>::scale(inv, ws[x]);
  if (blockIdx.x == 0 && tid == 0) st->nrm2 = tot;
}

// ----------------------------------------------------------------------------
// the fused streaming kernel
//   PHASE 0: coef_i = <v_i, w>              (i < nv), nrm2 = |w|^2; alpha_j = Re coef_j
//   PHASE 1: w -= sum coef_i v_i; coef_i = <v_i, w>; alpha_j += Re coef_j
//   PHASE 2: w -= sum coef_i v_i; beta_j = |w|; convergence check
// nv < 0: the device-looped solve; nv = st->j + 1, and PHASE 0 (the first kernel after
// the matvec) adds the matvec's time since st->t_mark to st->mv_ns
// ----------------------------------------------------------------------------
template <typename T, int PHASE>
__global__ void __launch_bounds__(VEC_THREADS)
    lz_pass_kernel(const T* __restrict__ V, int nv, ll n, T* __restrict__ w, LanczosDev* st,
                   double* part, unsigned* counter, int kmax) {
  if (*((volatile int*)&st->done)) return;
  if (nv < 0) {
    if (PHASE == 0 && blockIdx.x == 0 && threadIdx.x == 0) st->mv_ns += global_ns() - st->t_mark;
    nv = st->j + 1;
  }
  constexpr bool CPLX = ST<T>::cplx;
  constexpr int NW = VEC_THREADS / 32;
  __shared__ T ws[MAX_CHUNK];
  __shared__ double csh[2 * (KRYLOV_CAP + 1)];
  __shared__ double red[32];
  const int nblk = gridDim.x;
  const ll ch = (n + nblk - 1) / nblk;
  const ll x0 = (ll)blockIdx.x * ch;
  const ll x1 = (x0 + ch < n) ? x0 + ch : n;
  const int len = (x1 > x0) ? (int)(x1 - x0) : 0;
  const int ncoef = (PHASE == 2) ? 0 : nv;

  if (PHASE >= 1) {
    for (int i = threadIdx.x; i < 2 * nv; i += blockDim.x) csh[i] = st->coef[i];
    __syncthreads();
  }
  double ww = 0.0;
  for (int x = threadIdx.x; x < len; x += blockDim.x) {
    T v = w[x0 + x];
    if (PHASE >= 1) {
      for (int i = 0; i < nv; ++i) {
        T c = ST<T>::make(csh[2 * i], csh[2 * i + 1]);
        v = v - ST<T>::mul(c, V[(ll)i * n + x0 + x]);
      }
      w[x0 + x] = v;
    }
    ws[x] = v;
    ww += ST<T>::abs2(v);
  }
  __syncthreads();
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = wid; i < ncoef; i += NW) {
    const T* vi = V + (ll)i * n + x0;
    double sr = 0.0, si = 0.0;
    for (int x = lane; x < len; x += 32) {
      T p = ST<T>::cmul(vi[x], ws[x]);
      sr += ST<T>::re(p);
      if (CPLX) si += ST<T>::im(p);
    }
    sr = warp_sum(sr);
    if (CPLX) si = warp_sum(si);
    if (lane == 0) {  // partials are coefficient-major: part[idx][block]
      part[(ll)(2 * i) * nblk + blockIdx.x] = sr;
      part[(ll)(2 * i + 1) * nblk + blockIdx.x] = si;
    }
  }
  ww = block_sum(ww, red);
  if (threadIdx.x == 0) part[(ll)(2 * nv) * nblk + blockIdx.x] = ww;

  if (!arrive_last(counter, nblk)) return;

  // ---- finalize (last block): deterministic fixed-order sums, one warp per coefficient
  //      (lane l adds blocks l, l+32, ... in order, then a fixed shuffle tree)
  for (int c = wid; c < 2 * ncoef + 1; c += NW) {
    const int idx = (c == 2 * ncoef) ? 2 * nv : c;
    const double* pc = part + (ll)idx * nblk;
    double s = 0.0;
    for (int b = lane; b < nblk; b += 32) s += pc[b];
    s = warp_sum(s);
    if (lane == 0) {
      if (c == 2 * ncoef) st->nrm2 = s;
      else st->coef[c] = s;
    }
  }
  __syncthreads();
  __threadfence_block();
  const int j = nv - 1;
  if (PHASE == 0) {
    if (threadIdx.x == 0) st->alpha[j] = st->coef[2 * j];
  } else if (PHASE == 1) {
    if (threadIdx.x == 0) st->alpha[j] += st->coef[2 * j];
  } else {
    __shared__ StepState sh;
    if (threadIdx.x == 0) st->beta[j] = sqrt(fmax(st->nrm2, 0.0));
    __syncthreads();
    for (int i = threadIdx.x; i <= j; i += blockDim.x) {
      sh.a[i] = st->alpha[i];
      sh.b[i] = st->beta[i];
    }
    __syncthreads();
    if (threadIdx.x < 32) lz_finish_step(st, sh, j + 1, kmax, st->e_prev, st->tol);
  }
  if (threadIdx.x == 0) *counter = 0u;
}

template <typename T>
__global__ void lz_normalize_kernel(T* __restrict__ vnext, const T* __restrict__ w, ll n,
                                    LanczosDev* st) {
  if (*((volatile int*)&st->done)) return;
  double inv = 1.0 / sqrt(st->nrm2);
  for (ll x = (ll)blockIdx.x * blockDim.x + threadIdx.x; x < n; x += (ll)gridDim.x * blockDim.x)
    vnext[x] = ST<T>::scale(inv, w[x]);
}

// device-looped form: v_(j+1) = w / |w| into V[j + 1] and into cur, j = st->j
template <typename T>
__global__ void lz_normalize_dev_kernel(T* __restrict__ V, T* __restrict__ cur, const T* __restrict__ w,
                                        ll n, LanczosDev* st) {
  if (*((volatile int*)&st->done)) return;
  const int j1 = st->j + 1;
  if (j1 >= st->kmax) return;
  double inv = 1.0 / sqrt(st->nrm2);
  T* vnext = V + (ll)j1 * n;
  for (ll x = (ll)blockIdx.x * blockDim.x + threadIdx.x; x < n; x += (ll)gridDim.x * blockDim.x) {
    const T v = ST<T>::scale(inv, w[x]);
    vnext[x] = v;
    cur[x] = v;
  }
}

// last node of the device loop's body (one thread)
__global__ void lz_loop_next_kernel(LanczosDev* st, cudaGraphConditionalHandle h, int kmax) {
  const int g = st->guard + 1;
  st->guard = g;
  const int done = *((volatile int*)&st->done);
  if (!done) st->j += 1;
  st->t_mark = global_ns();
  cudaGraphSetConditional(h, (!done && g < kmax) ? 1u : 0u);
}

// |x|^2 into st->nrm2 (or out), last-block finalize
template <typename T>
__global__ void norm2_kernel(const T* __restrict__ x, ll n, double* out, double* part,
                             unsigned* counter) {
  __shared__ double red[32];
  double s = 0.0;
  for (ll i = (ll)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (ll)gridDim.x * blockDim.x)
    s += ST<T>::abs2(x[i]);
  s = block_sum(s, red);
  if (threadIdx.x == 0) part[blockIdx.x] = s;
  if (!arrive_last(counter, gridDim.x)) return;
  if (threadIdx.x < 32) {  // fixed order: lane l adds blocks l, l+32, ..., then a shuffle tree
    double t = 0.0;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += 32) t += part[b];
    t = warp_sum(t);
    if (threadIdx.x == 0) {
      *out = t;
      *counter = 0u;
    }
  }
}

// reset solver state; if |theta| is ~0, replace theta by a seeded random vector
template <typename T>
__global__ void lz_reset_kernel(T* theta, ll n, LanczosDev* st, unsigned seed, double tol, int kmax,
                                const unsigned* seed_host) {
  const bool tiny = !(st->nrm2 >= 1e-28);
  if (tiny) {
    if (seed_host) seed = *((volatile const unsigned*)seed_host);
    for (ll x = (ll)blockIdx.x * blockDim.x + threadIdx.x; x < n; x += (ll)gridDim.x * blockDim.x) {
      double r = hash_uniform(((unsigned long long)seed << 32) ^ (unsigned long long)(2 * x));
      double i = ST<T>::cplx ? hash_uniform(((unsigned long long)seed << 32) ^ (2 * x + 1)) : 0.0;
      theta[x] = ST<T>::make(r, i);
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    st->randomized = tiny ? 1 : 0;
    st->done = 0;
    st->converged = 0;
    st->n_iter = 0;
    st->e_prev = 1e300;
    st->e_cur = 0.0;
    st->tol = tol;
    st->kmax = kmax;
    st->j = 0;
    st->guard = 0;
    st->t_mark = 0ull;
    st->mv_ns = 0ull;
  }
}

template <typename T>
__global__ void lz_v0_kernel(const T* __restrict__ theta, T* __restrict__ v0, ll n, LanczosDev* st,
                             T* __restrict__ cur) {
  double inv = 1.0 / sqrt(st->nrm2);
  for (ll x = (ll)blockIdx.x * blockDim.x + threadIdx.x; x < n; x += (ll)gridDim.x * blockDim.x) {
    const T v = ST<T>::scale(inv, theta[x]);
    v0[x] = v;
    if (cur) cur[x] = v;
  }
  if (cur && blockIdx.x == 0 && threadIdx.x == 0) st->t_mark = global_ns();
}

template <typename T>
__global__ void lz_ritz_kernel(const T* __restrict__ V, ll n, T* __restrict__ out,
                               const LanczosDev* st) {
  __shared__ double r[KRYLOV_CAP];
  const int k = st->n_iter;
  for (int i = threadIdx.x; i < k; i += blockDim.x) r[i] = st->ritz[i];
  __syncthreads();
  for (ll x = (ll)blockIdx.x * blockDim.x + threadIdx.x; x < n; x += (ll)gridDim.x * blockDim.x) {
    T acc = ST<T>::zero();
    for (int i = 0; i < k; ++i) acc = acc + ST<T>::scale(r[i], V[(ll)i * n + x]);
    out[x] = acc;
  }
}

template <typename T>
__global__ void scale_by_inv_sqrt_kernel(T* x, ll n, const double* nrm2) {
  double s = *nrm2;
  double inv = (s > 0.0) ? 1.0 / sqrt(s) : 0.0;
  for (ll i = (ll)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (ll)gridDim.x * blockDim.x)
    x[i] = ST<T>::scale(inv, x[i]);
}

static int grid_for(ll n) {
  ll g = (n + VEC_THREADS - 1) / VEC_THREADS;
  if (g > 148 * 8) g = 148 * 8;
  if (g < 1) g = 1;
  return (int)g;
}

namespace {
// launches a kernel of the fused step on grid g: one cluster, or cooperatively
template <typename K, typename... A>
void launch_step(K kernel, std::atomic<unsigned long long>& attr, std::atomic<unsigned long long>& attr_c,
                 const StepGrid& g, size_t smem, cudaStream_t s, A... args) {
  // (g.cluster is the same in every launch of one kernel instantiation)
  const size_t smem_max = (g.cluster ? LS_SMEM_CLUSTER : LS_SMEM_GRID) + sizeof(double) * LS_WARPS * (2 * KRYLOV_CAP + 1);
  set_smem_attr_once(attr, (const void*)kernel, (int)smem_max);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(g.blocks);
  cfg.blockDim = dim3(LS_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  at[1] = pdl_attribute();
  cfg.numAttrs = 1;
  if (g.cluster) {
    cfg.numAttrs = 2;  // (not with the cooperative launch)
    func_attr_once(attr_c, (const void*)kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = g.blocks;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
  } else {
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
  }
  cfg.attrs = at;
  DMRG2_CUDA(cudaLaunchKernelEx(&cfg, kernel, args...));
  DMRG2_CHECK_LAUNCH();
}

template <typename T, bool CL>
void step_launch(const StepGrid& g, T* V, int nv, ll n, const T* w, T* cur, LanczosDev* st, RedScratch& r, int kmax,
                 int loop, cudaGraphConditionalHandle h, int* host_done, cudaStream_t s) {
  static std::atomic<unsigned long long> attr{0}, attr_c{0};
  const int nvm = loop ? kmax : nv, nc = (ST<T>::cplx ? 2 : 1) * nvm;
  const size_t row = sizeof(T) * (size_t)g.chunk, cap = g.cluster ? LS_SMEM_CLUSTER : LS_SMEM_GRID;
  const int ncache = cap > row ? (int)std::min<size_t>((cap - row) / row, (size_t)nvm) : 0;
  const size_t smem = row * (size_t)(1 + ncache) + sizeof(double) * (size_t)LS_WARPS * (nc + 1);
  launch_step(lz_step_kernel<T, CL>, attr, attr_c, g, smem, s, V, nv, n, w, cur, st, r.part, kmax, g.chunk,
              ncache, loop, h, (volatile int*)host_done, test_unsignalled_wait("step") ? 1 : 0);
}
template <typename T, bool CL>
void start_launch(const StepGrid& g, T* theta, T* v0, T* cur, ll n, LanczosDev* st, RedScratch& r, unsigned seed,
                  const unsigned* seed_host, double tol, int kmax, cudaStream_t s) {
  static std::atomic<unsigned long long> attr{0}, attr_c{0};
  launch_step(lz_start_kernel<T, CL>, attr, attr_c, g, 0, s, theta, v0, cur, n, st, r.part, seed, seed_host, tol, kmax,
              g.chunk, test_unsignalled_wait("start") ? 1 : 0);
}
template <typename T, bool CL>
void ritz_launch(const StepGrid& g, const T* V, ll n, T* out, LanczosDev* st, RedScratch& r, LanczosHost* host,
                 cudaStream_t s) {
  static std::atomic<unsigned long long> attr{0}, attr_c{0};
  launch_step(lz_ritz_norm_kernel<T, CL>, attr, attr_c, g, sizeof(T) * (size_t)g.chunk, s, V, n, out, st, r.part,
              host, g.chunk, test_unsignalled_wait("ritz") ? 1 : 0);
}
}  // namespace

template <typename T>
void norm2(const T* x, ll n, double* out_dev, RedScratch& r, cudaStream_t s) {
  int g = grid_for(n);
  if (g > r.nblk) g = r.nblk;
  norm2_kernel<T><<<g, VEC_THREADS, 0, s>>>(x, n, out_dev, r.part, r.counter);
  DMRG2_CHECK_LAUNCH();
}

template <typename T>
void lz_start(T* theta, T* v0, ll n, LanczosDev* st, RedScratch& r, unsigned seed, double tol,
              int kmax, cudaStream_t s, T* cur, const unsigned* seed_host) {
  const StepGrid g = step_grid<T>(n, r.step_blocks);
  if (g.blocks && g.cluster) return start_launch<T, true>(g, theta, v0, cur, n, st, r, seed, seed_host, tol, kmax, s);
  if (g.blocks) return start_launch<T, false>(g, theta, v0, cur, n, st, r, seed, seed_host, tol, kmax, s);
  norm2<T>(theta, n, &st->nrm2, r, s);
  lz_reset_kernel<T><<<grid_for(n), VEC_THREADS, 0, s>>>(theta, n, st, seed, tol, kmax, seed_host);
  DMRG2_CHECK_LAUNCH();
  norm2<T>(theta, n, &st->nrm2, r, s);
  lz_v0_kernel<T><<<grid_for(n), VEC_THREADS, 0, s>>>(theta, v0, n, st, cur);
  DMRG2_CHECK_LAUNCH();
}

namespace {
// the streaming passes, for vectors beyond the fused step (nv < 0: read from st->j)
template <typename T>
void step_passes(T* V, int nv, ll n, T* w, LanczosDev* st, RedScratch& r, int kmax, cudaStream_t s) {
  lz_pass_kernel<T, 0><<<vec_blocks(n), VEC_THREADS, 0, s>>>(V, nv, n, w, st, r.part, r.counter, 0);
  DMRG2_CHECK_LAUNCH();
  lz_pass_kernel<T, 1><<<vec_blocks(n), VEC_THREADS, 0, s>>>(V, nv, n, w, st, r.part, r.counter, 0);
  DMRG2_CHECK_LAUNCH();
  lz_pass_kernel<T, 2><<<vec_blocks(n), VEC_THREADS, 0, s>>>(V, nv, n, w, st, r.part, r.counter, kmax);
  DMRG2_CHECK_LAUNCH();
}
}  // namespace

template <typename T>
void lz_step(T* V, int nv, ll n, T* w, LanczosDev* st, RedScratch& r, int kmax, int* host_done, cudaStream_t s) {
  const StepGrid g = step_grid<T>(n, r.step_blocks);
  if (g.blocks && g.cluster)
    return step_launch<T, true>(g, V, nv, n, w, nullptr, st, r, kmax, 0, cudaGraphConditionalHandle{}, host_done, s);
  if (g.blocks)
    return step_launch<T, false>(g, V, nv, n, w, nullptr, st, r, kmax, 0, cudaGraphConditionalHandle{}, host_done, s);
  step_passes<T>(V, nv, n, w, st, r, kmax, s);
  if (nv < kmax) {
    lz_normalize_kernel<T><<<grid_for(n), VEC_THREADS, 0, s>>>(V + (ll)nv * n, w, n, st);
    DMRG2_CHECK_LAUNCH();
  }
  DMRG2_CUDA(cudaMemcpyAsync(host_done, &st->done, sizeof(int), cudaMemcpyDeviceToHost, s));
}

template <typename T>
void lz_step_dev(T* V, ll n, T* w, T* cur, LanczosDev* st, RedScratch& r, int kmax, cudaGraphConditionalHandle h,
                 cudaStream_t s) {
  const StepGrid g = step_grid<T>(n, r.step_blocks);
  if (g.blocks && g.cluster) return step_launch<T, true>(g, V, 0, n, w, cur, st, r, kmax, 1, h, nullptr, s);
  if (g.blocks) return step_launch<T, false>(g, V, 0, n, w, cur, st, r, kmax, 1, h, nullptr, s);
  step_passes<T>(V, -1, n, w, st, r, kmax, s);
  lz_normalize_dev_kernel<T><<<grid_for(n), VEC_THREADS, 0, s>>>(V, cur, w, n, st);
  DMRG2_CHECK_LAUNCH();
  lz_loop_next_kernel<<<1, 1, 0, s>>>(st, h, kmax);
  DMRG2_CHECK_LAUNCH();
}

template <typename T>
void lz_ritz(const T* V, ll n, T* out, LanczosDev* st, RedScratch& r, LanczosHost* host, cudaStream_t s) {
  const StepGrid g = step_grid<T>(n, r.step_blocks);
  if (g.blocks && g.cluster) return ritz_launch<T, true>(g, V, n, out, st, r, host, s);
  if (g.blocks) return ritz_launch<T, false>(g, V, n, out, st, r, host, s);
  lz_ritz_kernel<T><<<grid_for(n), VEC_THREADS, 0, s>>>(V, n, out, st);
  DMRG2_CHECK_LAUNCH();
  norm2<T>(out, n, &st->nrm2, r, s);
  scale_by_inv_sqrt_kernel<T><<<grid_for(n), VEC_THREADS, 0, s>>>(out, n, &st->nrm2);
  DMRG2_CHECK_LAUNCH();
  lz_report_kernel<<<1, 1, 0, s>>>(st, host);
  DMRG2_CHECK_LAUNCH();
}

// The end of a warm-started split. As two norm kernels and three copies to the host this took
// about 20 us of a bond (five latency-bound operations); the last block's report to
// page-locked memory needs no copy.
template <typename T>
__global__ void __launch_bounds__(512)
    split_finish_kernel(const T* __restrict__ theta, ll nt, const T* __restrict__ kept, ll nk,
                        const int* status, const SvdOut* out, SplitHost* host, double* part, unsigned* counter) {
  __shared__ double red[32];
  const ll step = (ll)gridDim.x * blockDim.x, t0 = (ll)blockIdx.x * blockDim.x + threadIdx.x;
  double a = 0.0, b = 0.0;
#pragma unroll 4
  for (ll i = t0; i < nt; i += step) a += ST<T>::abs2(theta[i]);
#pragma unroll 4
  for (ll i = t0; i < nk; i += step) b += ST<T>::abs2(kept[i]);
  a = block_sum(a, red);
  b = block_sum(b, red);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = a;
    part[gridDim.x + blockIdx.x] = b;
  }
  if (!arrive_last(counter, gridDim.x)) return;
  if (threadIdx.x < 32) {  // fixed order: lane l adds blocks l, l+32, ..., then a shuffle tree
    double s = 0.0, t = 0.0;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += 32) {
      s += __ldcg(part + i);
      t += __ldcg(part + gridDim.x + i);
    }
    s = warp_sum(s);
    t = warp_sum(t);
    if (threadIdx.x == 0) {
      volatile SplitHost* h = host;
      h->theta2 = s;
      h->kept2 = t;
      h->failed = (*status || !(out->ns_done || out->ns_near)) ? 1 : 0;
      *counter = 0u;
    }
  }
}

__global__ void split_begin_kernel(int* status, SvdOut* out, int k) {
  SvdOut o{};
  o.k = k;
  *out = o;
  *status = 0;
}

void split_begin(int* status, SvdOut* out, int k, cudaStream_t s) {
  split_begin_kernel<<<1, 1, 0, s>>>(status, out, k);
  DMRG2_CHECK_LAUNCH();
}

template <typename T>
void split_finish(const T* theta, ll nt, const T* kept, ll nk, const int* status, const SvdOut* out, SplitHost* host,
                  RedScratch& r, cudaStream_t s) {
  // four elements of theta per thread, at most one block per SM (the sums of their partials are
  // the serial end of the kernel)
  const int g = (int)std::max<ll>(1, std::min<ll>(std::min(STEP_BLOCKS, r.nblk / 2), (nt + 2047) / 2048));
  split_finish_kernel<T><<<g, 512, 0, s>>>(theta, nt, kept, nk, status, out, host, r.part, r.counter);
  DMRG2_CHECK_LAUNCH();
}

template <typename T>
__global__ void __launch_bounds__(256)
    split_commit_kernel(const T* __restrict__ l, T* __restrict__ left, ll nl, const T* __restrict__ r,
                        T* __restrict__ right, ll nr, const int* skip) {
  if (skip && *((volatile const int*)skip)) return;
  const ll step = (ll)gridDim.x * blockDim.x, t0 = (ll)blockIdx.x * blockDim.x + threadIdx.x;
#pragma unroll 4
  for (ll i = t0; i < nl; i += step) left[i] = l[i];
#pragma unroll 4
  for (ll i = t0; i < nr; i += step) right[i] = r[i];
}

template <typename T>
void split_commit(const T* l, T* left, ll nl, const T* r, T* right, ll nr, const int* skip, cudaStream_t s) {
  const int g = (int)std::min<ll>(4 * STEP_BLOCKS, std::max<ll>(1, (std::max(nl, nr) + 511) / 512));
  split_commit_kernel<T><<<g, 256, 0, s>>>(l, left, nl, r, right, nr, skip);
  DMRG2_CHECK_LAUNCH();
}

std::atomic<int>& lz_fail_countdown() {
  static std::atomic<int> n{0};
  return n;
}
__global__ void lz_fail_kernel(LanczosDev* st, LanczosHost* host) {
  st->gave_up = 1;
  *((volatile int*)&host->gave_up) = 1;
}
void lz_fail(LanczosDev* st, LanczosHost* host, cudaStream_t s) {
  lz_fail_kernel<<<1, 1, 0, s>>>(st, host);
  DMRG2_CHECK_LAUNCH();
}

template <typename T>
void scale_inplace(T* x, ll n, const double* nrm2_dev, cudaStream_t s) {
  scale_by_inv_sqrt_kernel<T><<<grid_for(n), VEC_THREADS, 0, s>>>(x, n, nrm2_dev);
  DMRG2_CHECK_LAUNCH();
}

#define INST(T)                                                                                   \
  template void lz_start<T>(T*, T*, ll, LanczosDev*, RedScratch&, unsigned, double, int,      \
                            cudaStream_t, T*, const unsigned*);                                   \
  template void lz_step<T>(T*, int, ll, T*, LanczosDev*, RedScratch&, int, int*, cudaStream_t);   \
  template void lz_step_dev<T>(T*, ll, T*, T*, LanczosDev*, RedScratch&, int,                     \
                               cudaGraphConditionalHandle, cudaStream_t);                         \
  template void lz_ritz<T>(const T*, ll, T*, LanczosDev*, RedScratch&, LanczosHost*, cudaStream_t); \
  template void split_finish<T>(const T*, ll, const T*, ll, const int*, const SvdOut*, SplitHost*, \
                                RedScratch&, cudaStream_t);                                       \
  template void split_commit<T>(const T*, T*, ll, const T*, T*, ll, const int*, cudaStream_t);        \
  template void norm2<T>(const T*, ll, double*, RedScratch&, cudaStream_t);                       \
  template void scale_inplace<T>(T*, ll, const double*, cudaStream_t);
INST(double)
INST(zc)
#undef INST

}  // namespace dmrg2
