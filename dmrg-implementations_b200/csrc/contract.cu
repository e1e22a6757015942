#include "contract.cuh"
#include "heff_small.cuh"

#include <algorithm>
#include <cstring>
#include <stdexcept>

namespace dmrg2 {

// Y[a][o][e] = sum_k W[o][k] X[a][k][e] for Kin, Kout <= KM (the two-site MPO
// mixing of H_eff step 2 when D d^2 is small): one thread per (a, e), the Kin
// inputs in registers, W in shared memory. Bandwidth-bound: X read once, Y
// written once.
template <typename T, int KM>
__global__ void __launch_bounds__(128)
    mpo_mix_kernel(const T* __restrict__ X, const T* __restrict__ W, T* __restrict__ Y, int Kin,
                   int Kout, int cR, ll sX, ll sY, const int* skip) {
  pdl_wait();
  if (skip && *((volatile const int*)skip)) return;
  __shared__ T Ws[KM * KM];
  for (int i = threadIdx.x; i < KM * KM; i += blockDim.x) {
    const int o = i / KM, k = i % KM;
    Ws[i] = (o < Kout && k < Kin) ? W[(ll)o * Kin + k] : ST<T>::zero();
  }
  __syncthreads();
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= cR) return;
  const ll a = blockIdx.y;
  const T* xa = X + a * sX + e;
  T* ya = Y + a * sY + e;
  T xin[KM];
#pragma unroll
  for (int k = 0; k < KM; ++k) xin[k] = (k < Kin) ? xa[(ll)k * cR] : ST<T>::zero();
  for (int o = 0; o < Kout; ++o) {
    T acc = ST<T>::zero();
#pragma unroll
    for (int k = 0; k < KM; ++k) acc = acc + ST<T>::mul(Ws[o * KM + k], xin[k]);
    ya[(ll)o * cR] = acc;
  }
}

// The same mixing with W in its nonzero form (row starts, ascending columns, values), for up to
// MIX_WIDE_K inputs: a CTA takes one a and 32 columns e, stages all Kin inputs of them in shared
// memory, and its warps walk the rows of W; each output sums only its row's nonzeros, in the order
// of the dense loop above. Bandwidth-bound on L2: X read once, Y written once, and no work for
// W's zeros, which as a dense product on the tensor cores cost 28% of a Josephson matvec's flops
// (187 of 10,000 entries are nonzero there). Real data, us at cL = cR = 96 / 180 / 256, dense above
// / here: 20 x 20, 30 nonzeros (XXZ, D = 5) 5.3 / 6.9 / 8.7 and 3.4 / 4.9 / 7.3; 32 x 32, 48 nonzeros
// (J1-J2, D = 8) 7.2 / 9.7 / 12.2 and 4.2 / 6.6 / 10.0; with 409 of 1024 entries nonzero (128 x 128)
// they meet at 7.3, where the engine's rule (at most half) stops using it. A form with one thread
// per column and its inputs in shared memory took 5.8 / 6.2 / 7.0 and 8.1 / 8.5 / 9.6.
constexpr int MIX_WIDE_NT = 256;
constexpr int MIX_WIDE_NNZ = 768;  // nonzeros staged in shared memory (more are read through L1)
template <typename T>
__global__ void __launch_bounds__(MIX_WIDE_NT)
    mpo_mix_nonzero_kernel(const T* __restrict__ X, const T* __restrict__ val, const int* __restrict__ rowp,
                        T* __restrict__ Y, int Kin, int Kout, int cR, ll sX, ll sY, const int* skip) {
  pdl_wait();
  if (skip && *((volatile const int*)skip)) return;
  extern __shared__ __align__(16) unsigned char mix_smem[];
  T* xs = reinterpret_cast<T*>(mix_smem);  // [Kin][32]
  __shared__ T vs[MIX_WIDE_NNZ];
  __shared__ int cs[MIX_WIDE_NNZ], rp[MIX_WIDE_K + 1];
  constexpr int W = MIX_WIDE_NT / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int e = blockIdx.x * 32 + lane;
  const bool in = e < cR;
  const T* xa = X + blockIdx.y * sX + e;
  T* ya = Y + blockIdx.y * sY + e;
  const int* col = rowp + Kout + 1;
  unsigned top = 0;  // largest exponent field among this thread's inputs
#pragma unroll 8
  for (int k = warp; k < Kin; k += W) {
    const T x = in ? xa[(ll)k * cR] : ST<T>::zero();
    top = max(top, ST<T>::exponent_bits(x));
    xs[k * 32 + lane] = x;
  }
  for (int i = threadIdx.x; i <= Kout; i += MIX_WIDE_NT) rp[i] = rowp[i];
  // (the slots behind the last nonzero exist: the block holds Kin Kout of them)
  const int st = min(MIX_WIDE_NNZ, Kin * Kout);
  for (int i = threadIdx.x; i < st; i += MIX_WIDE_NT) {
    cs[i] = col[i] * 32;
    vs[i] = val[i];
  }
  // An infinity or a NaN among the inputs: zero entries count too, as in the dense product.
  if (__syncthreads_or(top >= 0x7ff00000u)) {
    for (int o = warp; o < Kout; o += W) {
      const int j1 = rp[o + 1];
      T acc = ST<T>::zero();
      for (int k = 0, j = rp[o]; k < Kin; ++k) {
        const bool nz = j < j1 && col[j] == k;
        acc = acc + ST<T>::mul(nz ? val[j] : ST<T>::zero(), xs[k * 32 + lane]);
        j += nz;
      }
      if (in) ya[(ll)o * cR] = acc;
    }
    return;
  }
  const bool staged = rp[Kout] <= MIX_WIDE_NNZ;
  for (int o = warp; o < Kout; o += W) {
    const int j0 = rp[o], j1 = rp[o + 1];
    T acc = ST<T>::zero();
    if (staged) {
      for (int j = j0; j < j1; ++j) acc = acc + ST<T>::mul(vs[j], xs[cs[j] + lane]);
    } else {
#pragma unroll 4
      for (int j = j0; j < j1; ++j) acc = acc + ST<T>::mul(val[j], xs[col[j] * 32 + lane]);
    }
    if (in) ya[(ll)o * cR] = acc;
  }
}

template <typename T>
int wwt_sparse_block(std::vector<T>& w, int Kin, int Kout) {
  const ll kk = (ll)Kin * Kout;
  if ((ll)w.size() != kk) throw std::invalid_argument("wwt_sparse_block: dense matrix of the wrong size");
  std::vector<T> val((size_t)kk, ST<T>::zero());
  std::vector<int> ints((size_t)(Kout + 1 + kk), 0);
  int nnz = 0;
  for (int o = 0; o < Kout; ++o) {
    ints[(size_t)o] = nnz;
    for (int k = 0; k < Kin; ++k) {
      const T v = w[(size_t)o * Kin + k];
      if (ST<T>::nonzero(v)) {
        val[(size_t)nnz] = v;
        ints[(size_t)(Kout + 1 + nnz)] = k;
        ++nnz;
      }
    }
  }
  ints[(size_t)Kout] = nnz;
  const ll total = wwt_block_elems(Kin, Kout, sizeof(T));
  w.resize((size_t)total, ST<T>::zero());
  std::copy(val.begin(), val.end(), w.begin() + kk);
  std::memcpy(w.data() + 2 * kk, ints.data(), sizeof(int) * ints.size());
  return nnz;
}

// step 2 of the matvec: Y[a] = W X[a] for every a (MPO mixing, FP64); X[a] is Kin x cR,
// Y[a] is Kout x cR; wsp: W's nonzero form (wwt_sparse_block), or null
template <typename T>
static void mix_rows(const T* X, const T* W, T* Y, int cL, int cR, int Kin, int Kout, const int* skip,
                     cudaStream_t s, const T* wsp = nullptr) {
  if (wsp && Kin <= MIX_WIDE_K && Kout <= MIX_WIDE_K && cL <= 65535) {
    const ll kk = (ll)Kin * Kout;
    static std::atomic<unsigned long long> attr{0};
    set_smem_attr_once(attr, (const void*)mpo_mix_nonzero_kernel<T>, (int)(sizeof(T) * MIX_WIDE_K * 32));
    dim3 grid(ceil_div(cR, 32), cL);
    launch_pdl(mpo_mix_nonzero_kernel<T>, grid, MIX_WIDE_NT, sizeof(T) * (size_t)Kin * 32, s, X, wsp,
               (const int*)(wsp + kk), Y, Kin, Kout, cR, (ll)Kin * cR, (ll)Kout * cR, skip);
  } else if (Kin <= 32 && Kout <= 32 && cL <= 65535) {
    dim3 grid(ceil_div(cR, 128), cL);
    launch_pdl(mpo_mix_kernel<T, 32>, grid, 128, 0, s, X, W, Y, Kin, Kout, cR, (ll)Kin * cR, (ll)Kout * cR, skip);
  } else {
    Gemm<T> g;
    g.M = Kout; g.N = cR; g.K = Kin;
    g.A = W; g.lda = Kin; g.sA1 = 0;
    g.B = X; g.ldb = cR; g.sB1 = (ll)Kin * cR;
    g.C = Y; g.ldc = cR; g.sC1 = (ll)Kout * cR;
    g.nb1 = cL; g.skip = skip;
    launch_gemm(g, s);
  }
}

template <typename T>
void heff_apply_split(const T* Lenv, const T* Renv, const T* WWt, const T* in, T* out, T* X, T* Y, int cL,
                      int cR, int d, int Dl, int Dr, SplitScratch& ws, const int* skip, cudaStream_t s) {
  const ll dd = (ll)d * d;
  const T one = ST<T>::one(), zero = ST<T>::zero();
  // step 1: X[a][w][.] = L[a][w][:] theta, Dl batches sharing theta
  gemm_bf16x3<T>(0, 0, cL, (int)(dd * cR), cL, one, Lenv, (ll)Dl * cL, cL, in, dd * cR, 0, zero, X,
                 (ll)Dl * dd * cR, dd * cR, Dl, ws, s, skip);
  mix_rows(X, WWt, Y, cL, cR, (int)(Dl * dd), (int)(dd * Dr), skip, s);
  // step 3: out[(a,p,q)][f] = sum_(n,e) Y[(a,p,q)][(n,e)] R[f][(n,e)]
  gemm_bf16x3<T>(0, 1, (int)(cL * dd), cR, Dr * cR, one, Y, (ll)Dr * cR, 0, Renv, (ll)Dr * cR, 0, zero, out, cR,
                 0, 1, ws, s, skip);
}

template <typename T>
void heff_apply(const T* Lenv, const T* Renv, const T* WWt, const T* in, T* out, T* X, T* Y, int cL,
                int cR, int d, int Dl, int Dr, const int* skip, cudaStream_t s, const T* wsp, const int* dense) {
  const ll dd = (ll)d * d;
  if (heff_small(Lenv, Renv, WWt, in, out, cL, cR, (int)dd, Dl, Dr, skip, s)) return;
  {
    Gemm<T> g;
    g.M = cL * Dl; g.N = (int)(dd * cR); g.K = cL;  // rows (a, w)
    g.A = Lenv; g.lda = cL;
    g.B = in; g.ldb = dd * cR;
    g.C = X; g.ldc = dd * cR;
    g.skip = skip;
    launch_gemm(g, s);
  }
  if (wsp && dense) {  // which form serves is known on the device only; the other one returns at once
    mix_rows(X, WWt, Y, cL, cR, (int)(Dl * dd), (int)(dd * Dr), dense, s, wsp);
    mix_rows<T>(X, WWt, Y, cL, cR, (int)(Dl * dd), (int)(dd * Dr), dense + 1, s);
  } else {
    mix_rows(X, WWt, Y, cL, cR, (int)(Dl * dd), (int)(dd * Dr), skip, s, wsp);
  }
  {
    Gemm<T> g;
    g.tb = true;
    g.M = (int)(cL * dd); g.N = cR; g.K = Dr * cR;
    g.A = Y; g.lda = (ll)Dr * cR;
    g.B = Renv; g.ldb = (ll)Dr * cR;
    g.C = out; g.ldc = cR;
    g.skip = skip;
    launch_gemm(g, s);
  }
}

template <typename T>
void heff1_apply(const T* Lenv, const T* Renv, const T* WmixL, const T* in, T* out, T* X, T* Y, int cL, int cR,
                 int d, int Dl, int Dr, const int* skip, cudaStream_t s) {
  if (heff_small(Lenv, Renv, WmixL, in, out, cL, cR, d, Dl, Dr, skip, s)) return;
  {
    Gemm<T> g;  // X[a][w][(s,e)] = sum_c L[a][w][c] A[c][(s,e)]
    g.M = cL * Dl; g.N = d * cR; g.K = cL;
    g.A = Lenv; g.lda = cL;
    g.B = in; g.ldb = (ll)d * cR;
    g.C = X; g.ldc = (ll)d * cR;
    g.skip = skip;
    launch_gemm(g, s);
  }
  mix_rows(X, WmixL, Y, cL, cR, Dl * d, d * Dr, skip, s);  // Y[a][(t,w')][e]
  {
    Gemm<T> g;  // out[(a,t)][f] = sum_(w',e) Y[(a,t)][(w',e)] R[f][(w',e)]
    g.tb = true;
    g.M = cL * d; g.N = cR; g.K = Dr * cR;
    g.A = Y; g.lda = (ll)Dr * cR;
    g.B = Renv; g.ldb = (ll)Dr * cR;
    g.C = out; g.ldc = cR;
    g.skip = skip;
    launch_gemm(g, s);
  }
}

double heff1_flops(int cL, int cR, int d, int Dl, int Dr, bool cplx) {
  const double f = 2.0 * Dl * cL * ((double)d * cR) * cL + 2.0 * cL * ((double)d * Dr) * cR * ((double)Dl * d) +
                   2.0 * ((double)cL * d) * cR * ((double)Dr * cR);
  return cplx ? 4.0 * f : f;
}

double heff_flops(int cL, int cR, int d, int Dl, int Dr, bool cplx) {
  double dd = (double)d * d;
  double f = 2.0 * Dl * cL * (dd * cR) * cL + 2.0 * cL * (dd * Dr) * cR * (Dl * dd) +
             2.0 * (cL * dd) * cR * ((double)Dr * cR);
  return cplx ? 4.0 * f : f;
}

double env_flops(int ci, int co, int d, int Dl, int Dr, bool cplx) {
  double f = 2.0 * ((double)ci * Dl) * ((double)d * co) * ci + 2.0 * ci * ((double)d * Dr) * co * (Dl * d) +
             2.0 * co * ((double)Dr * co) * ((double)ci * d);
  return cplx ? 4.0 * f : f;
}

template <typename T>
void env_left(const T* Lenv, const T* A, const T* WmixL, T* Lnew, T* X, T* Y, int cL, int cO, int d,
              int Dl, int Dr, cudaStream_t s) {
  {
    Gemm<T> g;
    g.M = cL * Dl; g.N = d * cO; g.K = cL;
    g.A = Lenv; g.lda = cL;
    g.B = A; g.ldb = (ll)d * cO;
    g.C = X; g.ldc = (ll)d * cO;
    launch_gemm(g, s);
  }
  // Y[a] = WmixL X[a] for every a: the MPO mixing, a (d Dr) x (Dl d) matrix (a batched GEMM
  // of tiny matrices wastes most of each tensor-core tile: 13 us at chi = 256 against ~5)
  mix_rows(X, WmixL, Y, cL, cO, Dl * d, d * Dr, nullptr, s);
  {
    Gemm<T> g;
    g.ta = true; g.ca = true;
    g.M = cO; g.N = Dr * cO; g.K = cL * d;
    g.A = A; g.lda = cO;
    g.B = Y; g.ldb = (ll)Dr * cO;
    g.C = Lnew; g.ldc = (ll)Dr * cO;
    launch_gemm(g, s);
  }
}

template <typename T>
void env_right(const T* Renv, const T* B, const T* WmixR, T* Rnew, T* X, T* Y, int cI, int cO,
               int d, int Dl, int Dr, cudaStream_t s) {
  {
    Gemm<T> g;
    g.tb = true;
    g.M = cI * Dr; g.N = cO; g.K = cI;
    g.A = Renv; g.lda = cI; g.sA1 = 0;
    g.B = B; g.ldb = (ll)d * cI; g.sB1 = cI;
    g.C = X; g.ldc = (ll)d * cO; g.sC1 = cO;
    g.nb1 = d;
    launch_gemm(g, s);
  }
  // Y[s][a] = WmixR[s] X[a] for every a and physical index s (MPO mixing, Dl x (Dr d))
  for (int sp = 0; sp < d; ++sp)
    mix_rows(X, WmixR + (ll)sp * Dl * Dr * d, Y + (ll)sp * cI * Dl * cO, cI, cO, Dr * d, Dl, nullptr, s);
  {
    Gemm<T> g;
    g.ca = true;
    g.M = cO; g.N = Dl * cO; g.K = d * cI;
    g.A = B; g.lda = (ll)d * cI;
    g.B = Y; g.ldb = (ll)Dl * cO;
    g.C = Rnew; g.ldc = (ll)Dl * cO;
    launch_gemm(g, s);
  }
}

template <typename T>
void theta_form(const T* A, const T* B, T* theta, int cL, int cM, int cR, int d, cudaStream_t s) {
  Gemm<T> g;
  g.M = cL * d; g.N = d * cR; g.K = cM;
  g.A = A; g.lda = cM;
  g.B = B; g.ldb = (ll)d * cR;
  g.C = theta; g.ldc = (ll)d * cR;
  launch_gemm(g, s);
}

template <typename T>
void build_wwt(const T* WL, const T* WR, int Dl, int Dm, int Dr, int d, std::vector<T>& out) {
  // WWt[(p,q,n)][(w,s,r)] = sum_m WL[w][m][s][p] WR[m][n][r][q]
  const int rows = d * d * Dr, cols = Dl * d * d;
  out.assign((size_t)rows * cols, ST<T>::zero());
  for (int p = 0; p < d; ++p)
    for (int q = 0; q < d; ++q)
      for (int n = 0; n < Dr; ++n)
        for (int w = 0; w < Dl; ++w)
          for (int s = 0; s < d; ++s)
            for (int r = 0; r < d; ++r) {
              T acc = ST<T>::zero();
              for (int m = 0; m < Dm; ++m) {
                T a = WL[(((size_t)w * Dm + m) * d + s) * d + p];
                T b = WR[(((size_t)m * Dr + n) * d + r) * d + q];
                acc = acc + ST<T>::mul(a, b);
              }
              size_t row = ((size_t)p * d + q) * Dr + n;
              size_t col = ((size_t)w * d + s) * d + r;
              out[row * cols + col] = acc;
            }
}

template <typename T>
void build_wmix_left(const T* W, int Dl, int Dr, int d, std::vector<T>& out) {
  // WmixL[(t,w')][(w,s)] = W[w][w'][s][t]
  const int rows = d * Dr, cols = Dl * d;
  out.assign((size_t)rows * cols, ST<T>::zero());
  for (int t = 0; t < d; ++t)
    for (int wp = 0; wp < Dr; ++wp)
      for (int w = 0; w < Dl; ++w)
        for (int s = 0; s < d; ++s)
          out[((size_t)t * Dr + wp) * cols + (size_t)w * d + s] = W[(((size_t)w * Dr + wp) * d + s) * d + t];
}

template <typename T>
void build_wmix_right(const T* W, int Dl, int Dr, int d, std::vector<T>& out) {
  // WmixR[t][w'][(w,s)] = W[w'][w][s][t]   (w' left index in Dl, w right index in Dr)
  const int cols = Dr * d;
  out.assign((size_t)d * Dl * cols, ST<T>::zero());
  for (int t = 0; t < d; ++t)
    for (int wp = 0; wp < Dl; ++wp)
      for (int w = 0; w < Dr; ++w)
        for (int s = 0; s < d; ++s)
          out[((size_t)t * Dl + wp) * cols + (size_t)w * d + s] = W[(((size_t)wp * Dr + w) * d + s) * d + t];
}

#define INST(T)                                                                                 \
  template void heff_apply<T>(const T*, const T*, const T*, const T*, T*, T*, T*, int, int, int, \
                              int, int, const int*, cudaStream_t, const T*, const int*);         \
  template int wwt_sparse_block<T>(std::vector<T>&, int, int);                                  \
  template void heff1_apply<T>(const T*, const T*, const T*, const T*, T*, T*, T*, int, int, int,  \
                               int, int, const int*, cudaStream_t);                              \
  template void heff_apply_split<T>(const T*, const T*, const T*, const T*, T*, T*, T*, int, int,   \
                                    int, int, int, SplitScratch&, const int*, cudaStream_t);     \
  template void env_left<T>(const T*, const T*, const T*, T*, T*, T*, int, int, int, int, int,  \
                            cudaStream_t);                                                       \
  template void env_right<T>(const T*, const T*, const T*, T*, T*, T*, int, int, int, int, int, \
                             cudaStream_t);                                                      \
  template void theta_form<T>(const T*, const T*, T*, int, int, int, int, cudaStream_t);        \
  template void build_wwt<T>(const T*, const T*, int, int, int, int, std::vector<T>&);          \
  template void build_wmix_left<T>(const T*, int, int, int, std::vector<T>&);                   \
  template void build_wmix_right<T>(const T*, int, int, int, std::vector<T>&);
INST(double)
INST(zc)
#undef INST

}  // namespace dmrg2
