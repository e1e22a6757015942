// H_eff in one launch, for bonds whose three contractions are too short to fill the GPU.
//
//   out[a][p][q][f] = sum_{c,w,s,r,n,e} L[a][w][c] theta[c][s][r][e] WW[(p,q,n)][(w,s,r)] R[f][n][e]
//
// Nothing couples two values of a before the result, so a cluster of C CTAs takes a block of
// Ta rows a through all three steps with the intermediates in shared memory:
//   1  X[(a,w)][(s,r,e)] = sum_c L theta     CTA q computes the columns e of its C-th part
//   2  Y[(a,p,q)][(n,e)] = WW X              on the same columns
//   3  out[(a,p,q)][f]   = sum_(n,e) Y R     CTA q sums over its part of e, for every f; the C
//                                            partial results meet through distributed shared
//                                            memory, each CTA adding a C-th of the columns f
// Ta is chosen so that the rows (a, w) fill one 16-row tensor-core tile; theta and R go from
// the L2 to the DMMA fragments without a detour (each CTA reads its part of them once), so the
// traffic is ceil(cL / Ta) (theta + R) and the kernel stops paying where that exceeds what the
// tiled GEMMs move (heff_small_fits). With few column tiles the warps split the contracted
// index and the partial tiles are added in slice order. Bound by latency: one round of L2 loads
// per step, two cluster barriers.
#include <cooperative_groups.h>

#include "gemm.cuh"
#include "heff_small.cuh"

namespace cg = cooperative_groups;

namespace dmrg2 {

namespace {

constexpr int HS_THREADS = 256;
constexpr int HS_WARPS = HS_THREADS / 32;
constexpr int HS_KMAX = 32;                    // largest d^2 D: a row of WW is one warp's read
constexpr size_t HS_SMEM_MAX = 200 * 1024;

struct HsPlan {
  int Ta = 0, C = 0;      // rows a per cluster, CTAs per cluster (0: not this path)
  int El = 0;             // columns e (and f) per CTA, a multiple of 8
  int ks1 = 1, ks3 = 1;   // slices of the contracted index in steps 1 and 3
  int pA = 0, pX = 0, pY = 0;  // shared-memory row pitches (elements)
  int MT3 = 0;            // 16-row tiles of step 3
  size_t smem = 0;
};

__host__ __device__ inline int hs_pitch(int k) { return ((k + 7) / 8) * 8 + 4; }  // conflict-free fragment rows

struct HsArgs {
  const void *L, *R, *W, *in;
  void* out;
  int cL, cR, dd, Dl, Dr;
  int Ta, El, ks1, ks3, pA, pX, pY;
  const int* skip;
};

template <typename T>
struct Acc {
  double re[4];
  double im[ST<T>::cplx ? 4 : 1];
  __device__ void zero() {
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      re[r] = 0.0;
      if constexpr (ST<T>::cplx) im[r] = 0.0;
    }
  }
  __device__ T get(int r) const {
    if constexpr (ST<T>::cplx) return mkz(re[r], im[r]);
    else return re[r];
  }
};

// acc += A B for one m16n8k8 step; a[4] = A(g,t), A(g+8,t), A(g,t+4), A(g+8,t+4), b[2] = B(t,g), B(t+4,g)
template <typename T>
__device__ __forceinline__ void mma_step(Acc<T>& acc, const T (&a)[4], const T (&b)[2]) {
  if constexpr (!ST<T>::cplx) {
    dmma16x8x8(acc.re, a[0], a[1], a[2], a[3], b[0], b[1]);
  } else {
    dmma16x8x8(acc.re, a[0].re, a[1].re, a[2].re, a[3].re, b[0].re, b[1].re);
    dmma16x8x8(acc.im, a[0].re, a[1].re, a[2].re, a[3].re, b[0].im, b[1].im);
    dmma16x8x8(acc.re, -a[0].im, -a[1].im, -a[2].im, -a[3].im, b[0].im, b[1].im);
    dmma16x8x8(acc.im, a[0].im, a[1].im, a[2].im, a[3].im, b[0].re, b[1].re);
  }
}

// One 8-column tile: acc[i] = A rows (16 i ..) x B over k in [k0, k1), A in shared memory (rows
// beyond `rows` repeat the last one; their results are not stored, and A holds zeros from K
// up to the next multiple of 8), b(k) = *at(k) where k < K and at(k) is not null, else 0.
template <typename T, int MT, typename F>
__device__ __forceinline__ void tile_product(Acc<T> (&acc)[MT], const T* As, int pitch, int rows, F at, int k0, int k1,
                                             int K, int gq, int tq) {
  constexpr int U = ST<T>::cplx ? 4 : 8;  // k steps whose loads of B are in flight together
  int ra[MT][2];
#pragma unroll
  for (int i = 0; i < MT; ++i) {
    ra[i][0] = min(i * 16 + gq, rows - 1) * pitch;
    ra[i][1] = min(i * 16 + gq + 8, rows - 1) * pitch;
    acc[i].zero();
  }
  for (int k = k0; k < k1; k += 8 * U) {
    T b[U][2];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int kk = k + 8 * u + 4 * h + tq;
        const T* src = kk < min(k1, K) ? at(kk) : nullptr;
        b[u][h] = src ? *src : ST<T>::zero();
      }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (k + 8 * u < k1) {
#pragma unroll
        for (int i = 0; i < MT; ++i) {
          const int kk = k + 8 * u + tq;
          T a[4] = {As[ra[i][0] + kk], As[ra[i][1] + kk], As[ra[i][0] + kk + 4], As[ra[i][1] + kk + 4]};
          mma_step<T>(acc[i], a, b[u]);
        }
      }
    }
  }
}

template <typename T, int MT3>
__global__ void __launch_bounds__(HS_THREADS) heff_small_kernel(HsArgs g) {
  pdl_wait();
  if (g.skip && *((volatile const int*)g.skip)) return;  // constant during the launch: the whole cluster leaves
  cg::cluster_group cluster = cg::this_cluster();
  const int q = (int)cluster.block_rank(), C = (int)cluster.num_blocks();
  extern __shared__ __align__(16) unsigned char hs_smem[];
  __shared__ int koff[HS_KMAX];  // place of input k = (w, s, r) in a row block of X
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, gq = lane >> 2, tq = lane & 3;
  const int cL = g.cL, cR = g.cR, dd = g.dd, Dl = g.Dl, Dr = g.Dr, El = g.El;
  const int Kin = Dl * dd, Kout = dd * Dr, K3 = Dr * El;
  const int a0 = (blockIdx.x / C) * g.Ta, na = min(g.Ta, cL - a0);
  const int rows1 = na * Dl, rows3 = na * dd, cols = dd * El;
  const int e0 = q * El, ev = min(El, cR - e0);
  const int cRp = (cR + 7) & ~7, pO = cRp + 2;
  T* As = reinterpret_cast<T*>(hs_smem);                       // [Ta Dl][pA]
  T* Xs = As + (ll)g.Ta * Dl * g.pA;                           // [ks1][Ta Dl][pX], then [ks3][Ta dd][pO]
  const ll xs = max((ll)g.ks1 * g.Ta * Dl * g.pX, (ll)g.ks3 * g.Ta * dd * pO);
  T* Ys = Xs + xs;                                             // [Ta dd][pY]
  T* wval = Ys + (ll)g.Ta * dd * g.pY;                         // [Kout][Kin]
  unsigned char* wcol = reinterpret_cast<unsigned char*>(wval + Kout * Kin);  // [Kout][Kin]
  int* wcnt = reinterpret_cast<int*>(wcol + ((Kout * Kin + 15) & ~15));            // [Kout]
  const T* Lg = reinterpret_cast<const T*>(g.L) + (ll)a0 * Dl * cL;
  const T* Rg = reinterpret_cast<const T*>(g.R);
  const T* Wg = reinterpret_cast<const T*>(g.W);
  const T* th = reinterpret_cast<const T*>(g.in);

  // a block's rows of L are contiguous; zeros up to the next multiple of 8 columns
  const int kp1 = (cL + 7) & ~7;
  for (int r = warp; r < rows1; r += HS_WARPS)
    for (int k = lane; k < kp1; k += 32) As[r * g.pA + k] = k < cL ? Lg[(ll)r * cL + k] : ST<T>::zero();
  for (int k = tid; k < Kin; k += HS_THREADS) koff[k] = (k / dd) * g.pX + (k % dd) * El;
  // nonzeros of each row of WW, columns ascending (a warp's rows are read together)
  {
    T wv[HS_KMAX / HS_WARPS];
#pragma unroll
    for (int h = 0; h < HS_KMAX / HS_WARPS; ++h) {
      const int o = warp + h * HS_WARPS;
      wv[h] = (o < Kout && lane < Kin) ? Wg[(ll)o * Kin + lane] : ST<T>::zero();
    }
#pragma unroll
    for (int h = 0; h < HS_KMAX / HS_WARPS; ++h) {
      const int o = warp + h * HS_WARPS;
      const bool nz = ST<T>::nonzero(wv[h]);
      const unsigned m = __ballot_sync(0xffffffffu, nz);
      if (nz) {
        const int at = o * Kin + __popc(m & ((1u << lane) - 1u));
        wcol[at] = (unsigned char)lane;
        wval[at] = wv[h];
      }
      if (lane == 0 && o < Kout) wcnt[o] = __popc(m);
    }
  }
  __syncthreads();

  // ---- step 1
  bool bad = false;  // an infinity or a NaN in X
  {
    const int nt = cols / 8, et = El / 8;
    const int kc = ((kp1 / 8 + g.ks1 - 1) / g.ks1) * 8;
    for (int u = warp; u < nt * g.ks1; u += HS_WARPS) {
      const int t = u % nt, sl = u / nt;
      const int sr = t / et, el = (t % et) * 8;
      const int e = e0 + el + gq;
      Acc<T> acc[1];
      const T* bp = th + (ll)sr * cR + e;
      const ll sk = (ll)dd * cR;
      auto at = [&](int kk) { return e < cR ? bp + kk * sk : nullptr; };
      tile_product<T, 1>(acc, As, g.pA, rows1, at, sl * kc, min(sl * kc + kc, kp1), cL, gq, tq);
      T* xo = Xs + (ll)sl * g.Ta * Dl * g.pX + sr * El + el + 2 * tq;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int row = gq + ((r & 2) ? 8 : 0);
        if (row < rows1) {
          xo[row * g.pX + (r & 1)] = acc[0].get(r);
          bad |= !ST<T>::finite(acc[0].get(r));
        }
      }
    }
  }
  bad = __syncthreads_or(bad);
  // ---- step 2 (columns beyond cR get zeros: step 3 sums over them; with an infinity or a NaN in X
  // the zeros of WW count too, as in a dense product)
  {
    const ll xsl = (ll)g.Ta * Dl * g.pX;
    for (int u = tid; u < na * Kout * El; u += HS_THREADS) {
      const int e = u % El, ao = u / El, o = ao % Kout, al = ao / Kout;
      T sum = ST<T>::zero();
      if (e < ev) {
        const T* x = Xs + (ll)al * Dl * g.pX + e;
        const unsigned char* wc = wcol + o * Kin;
        const T* wl = wval + o * Kin;
        const int cnt = bad ? Kin : wcnt[o];
        for (int j = 0; j < cnt; ++j) {
          const int k = bad ? j : wc[j];
          const T* xk = x + koff[k];
          T v = xk[0];
          for (int sl = 1; sl < g.ks1; ++sl) v = v + xk[sl * xsl];
          sum = sum + ST<T>::mul(bad ? Wg[o * Kin + j] : wl[j], v);
        }
      }
      Ys[(al * dd + o / Dr) * g.pY + (o % Dr) * El + e] = sum;
    }
  }
  __syncthreads();
  // ---- step 3: the part of every column f that this CTA's e contribute
  {
    const int nt = cRp / 8;
    const int kc = ((K3 / 8 + g.ks3 - 1) / g.ks3) * 8;  // K3 = Dr El is a multiple of 8
    for (int u = warp; u < nt * g.ks3; u += HS_WARPS) {
      const int t = u % nt, sl = u / nt;
      const int f = t * 8 + gq;
      Acc<T> acc[MT3];
      const T* bp = Rg + (ll)f * Dr * cR + e0;
      auto at = [&](int kk) {
        const int n = kk / El, e = kk - n * El;
        return (f < cR && e < ev) ? bp + n * cR + e : nullptr;
      };
      tile_product<T, MT3>(acc, Ys, g.pY, rows3, at, sl * kc, min(sl * kc + kc, K3), K3, gq, tq);
      T* xo = Xs + (ll)sl * g.Ta * dd * pO + t * 8 + 2 * tq;
#pragma unroll
      for (int i = 0; i < MT3; ++i)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const int row = i * 16 + gq + ((r & 2) ? 8 : 0);
          if (row < rows3) xo[row * pO + (r & 1)] = acc[i].get(r);
        }
    }
    if (C > 1) cluster.sync();
    else __syncthreads();
    T* out = reinterpret_cast<T*>(g.out) + (ll)a0 * dd * cR;
    if (ev > 0)
      for (int u = tid; u < rows3 * El; u += HS_THREADS) {
        const int e = u % El, row = u / El;
        if (e >= ev) continue;
        T v = ST<T>::zero();
        for (int c = 0; c < C; ++c) {
          const T* p = C > 1 ? cluster.map_shared_rank(Xs, c) : Xs;
          for (int sl = 0; sl < g.ks3; ++sl) v = v + p[((ll)sl * g.Ta * dd + row) * pO + e0 + e];
        }
        out[(ll)row * cR + e0 + e] = v;
      }
    if (C > 1) cluster.sync();  // no CTA leaves while a peer may still read its partial result
  }
}

template <typename T>
HsPlan hs_plan(int cL, int cR, int dd, int Dl, int Dr) {
  HsPlan p;
  const int Kin = Dl * dd, Kout = dd * Dr;
  if (Dl > 16 || dd > 64 || Kin > HS_KMAX || Kout > HS_KMAX) return p;
  const int Ta = std::min(std::max(1, 16 / Dl), std::max(1, 64 / dd));
  const int blocks = ceil_div(cL, Ta);
  if (!heff_small_fits<T>(cL, cR, dd, Dl, Dr)) return p;
  int C = 1;  // enough CTAs for the GPU, at least one tile of 8 columns each
  while (C < 8 && blocks * C * 2 <= HS_TARGET_CTAS && ceil_div(cR, 2 * C) >= 8) C *= 2;
  for (; C <= 8; C *= 2) {  // more CTAs where the intermediates would not fit
    p.Ta = Ta;
    p.C = C;
    p.El = ceil_div(ceil_div(cR, C), 8) * 8;
    const int nt1 = dd * p.El / 8, nt3 = ceil_div(cR, 8);
    p.ks1 = std::min(std::max(1, HS_WARPS / nt1), ceil_div(cL, 8));
    p.ks3 = std::min(std::max(1, HS_WARPS / nt3), Dr * p.El / 8);
    p.pA = hs_pitch(cL);
    p.pX = dd * p.El + 2;
    p.pY = hs_pitch(Dr * p.El);
    p.MT3 = ceil_div(Ta * dd, 16);
    const size_t xs = std::max((size_t)p.ks1 * Ta * Dl * p.pX, (size_t)p.ks3 * Ta * dd * (ceil_div(cR, 8) * 8 + 2));
    p.smem = sizeof(T) * ((size_t)Ta * Dl * p.pA + xs + (size_t)Ta * dd * p.pY + (size_t)Kout * Kin) +
             (size_t)((Kout * Kin + 15) & ~15) +
             sizeof(int) * (size_t)Kout;
    if (p.smem <= HS_SMEM_MAX) return p;
  }
  p.C = 0;
  return p;
}

template <typename T>
bool overlaps(const T* a, ll na, const T* b, ll nb) {
  return (uintptr_t)a < (uintptr_t)(b + nb) && (uintptr_t)b < (uintptr_t)(a + na);
}

template <typename T, int MT3>
void hs_launch(const HsPlan& p, const HsArgs& a, cudaStream_t s) {
  static std::atomic<unsigned long long> attr{0};
  set_smem_attr_once(attr, (const void*)heff_small_kernel<T, MT3>, (int)HS_SMEM_MAX);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(ceil_div(a.cL, p.Ta) * p.C));
  cfg.blockDim = dim3(HS_THREADS);
  cfg.dynamicSmemBytes = p.smem;
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  at[1] = pdl_attribute();
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = p.C;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  DMRG2_CUDA(cudaLaunchKernelEx(&cfg, heff_small_kernel<T, MT3>, a));
  DMRG2_CHECK_LAUNCH();
}

}  // namespace

template <typename T>
bool heff_small(const T* Lenv, const T* Renv, const T* WWt, const T* in, T* out, int cL, int cR, int dd, int Dl, int Dr,
                const int* skip, cudaStream_t s) {
  // Clusters write their rows of out while others still read the operands: an out that shares memory
  // with the input or the left environment (which the tiled contractions are done with before
  // they write out) is theirs to serve.
  const ll n = (ll)cL * dd * cR;
  if (overlaps(out, n, in, n) || overlaps(out, n, Lenv, (ll)cL * Dl * cL)) return false;
  const HsPlan p = hs_plan<T>(cL, cR, dd, Dl, Dr);
  if (!p.C) return false;
  HsArgs a;
  a.L = Lenv; a.R = Renv; a.W = WWt; a.in = in; a.out = out;
  a.cL = cL; a.cR = cR; a.dd = dd; a.Dl = Dl; a.Dr = Dr;
  a.Ta = p.Ta; a.El = p.El; a.ks1 = p.ks1; a.ks3 = p.ks3; a.pA = p.pA; a.pX = p.pX; a.pY = p.pY;
  a.skip = skip;
  if (p.MT3 == 1) hs_launch<T, 1>(p, a, s);
  else if (p.MT3 == 2) hs_launch<T, 2>(p, a, s);
  else if (p.MT3 == 3) hs_launch<T, 3>(p, a, s);
  else hs_launch<T, 4>(p, a, s);
  return true;
}

template bool heff_small<double>(const double*, const double*, const double*, const double*, double*, int, int, int, int,
                                 int, const int*, cudaStream_t);
template bool heff_small<zc>(const zc*, const zc*, const zc*, const zc*, zc*, int, int, int, int, int, const int*,
                             cudaStream_t);

}  // namespace dmrg2
