// FP64 / complex128 GEMM on the sm_100a double-precision tensor cores.
//
// Blackwell's tcgen05 tensor-core instructions have no FP64 kind; FP64 tensor
// work on sm_100a is issued with the warp-level DMMA instruction
// mma.sync.m16n8k8.f64. This kernel stages A/B tiles in shared memory with a
// cp.async pipeline. Complex products are four real DMMAs on interleaved (re, im) tiles.
// The CTA tile and a split of K over a thread-block cluster are chosen by shape (gemm.cu).
//
// C[z] (M x N, row-major, ldc) = alpha * op(A[z]) * op(B[z]) + beta * C[z]
//   op(A) = A, A^T, conj(A) or A^H (M x K); op(B) = B or B^T (K x N)
//   storage: A[m*lda+k] (no trans) / A[k*lda+m] (trans), same for B.
// Batches form a 2-level grid z = z1 * nb2 + z2 with independent strides, so
// the strided views of the DMRG contractions map onto one launch each.
#pragma once

#include <cooperative_groups.h>

#include "common.cuh"

namespace dmrg2 {

struct GemmArgs {
  int M, N, K;
  const void* A;
  ll lda, sA1, sA2;
  const void* B;
  ll ldb, sB1, sB2;
  void* C;
  ll ldc, sC1, sC2;
  int nb2;
  double alpha_re, alpha_im, beta_re, beta_im;
  const int* skip;  // optional device flag: when non-zero the launch does nothing (with Cin: copies it to C)
  const void* Cin;  // the matrix beta multiplies (ld ldc); C itself when null
  int kchunk;       // split-K: blockIdx.z selects the K slice [z*kchunk, (z+1)*kchunk) (0 = off)
  int kcluster;     // slices of a split K (0 = off): those of a tile form one thread-block cluster
                    // and are summed in it, C = alpha sum + beta C written by the cluster
};

__device__ __forceinline__ void cp_async_8(void* smem, const void* gmem, bool pred) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  int n = pred ? 8 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(gmem), "r"(n));
}
__device__ __forceinline__ void cp_async_16(void* smem, const void* gmem, bool pred) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  int n = pred ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(n));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

__device__ __forceinline__ void dmma16x8x4(double (&c)[4], double a0, double a1, double b0) {
  asm volatile(
      "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, "
      "{%0,%1,%2,%3};\n"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a0), "d"(a1), "d"(b0));
}

// k index of the fragments: a0, a1 (rows g, g + 8) and b0 at k = t, a2, a3 and b1 at k = t + 4
__device__ __forceinline__ void dmma16x8x8(double (&c)[4], double a0, double a1, double a2, double a3, double b0,
                                           double b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a0), "d"(a1), "d"(a2), "d"(a3), "d"(b0), "d"(b1));
}

// CTA tile: BM x BN outputs, warps of WM x WN, STAGES pipeline stages of 128 bytes of k per row
// (16 doubles or 8 complex numbers)
template <int BM_, int BN_, int WM_, int WN_, int STAGES_>
struct TileCfg {
  static constexpr int BM = BM_, BN = BN_, WM = WM_, WN = WN_, STAGES = STAGES_;
  static constexpr int THREADS = (BM / WM) * (BN / WN) * 32;
};
using TileD64 = TileCfg<64, 64, 32, 32, 4>;
using TileD64x32 = TileCfg<64, 32, 32, 16, 4>;
using TileD32 = TileCfg<32, 32, 16, 16, 4>;
using TileZ64 = TileCfg<64, 32, 32, 16, 3>;
using TileZ32 = TileCfg<32, 32, 16, 16, 3>;

// Shared-memory image of one operand tile of MN rows (or columns) x BK, in 16-byte chunks.
// KC (contiguous along k in memory): [mn][8 chunks], chunk c of row r at c ^ 4 (r & 1), so that
// the 16-byte fragment reads of 8 lanes (two rows, four chunks) hit distinct banks without
// padding. Otherwise [k][MN + 2], where two consecutive rows or columns share a chunk of
// real data.
template <typename T, int MN, bool KC>
struct OperandTile {
  static constexpr int E = 16 / (int)sizeof(T);  // elements per chunk
  static constexpr int BK = 8 * E;
  static constexpr int P = MN + 2;
  static constexpr int ELEMS = KC ? MN * BK : BK * P;
  static constexpr int CPR = KC ? 8 : MN / E;    // chunks per row of the image
  static constexpr int CHUNKS = (KC ? MN : BK) * CPR;
};

// Loads one operand's tiles: per thread fixed chunk column, rows RS apart, one pointer that
// advances by one tile of k; edges by the byte count of each copy (the rest is zero-filled).
template <typename T, int MN, bool KC, int THREADS>
struct OperandLoader {
  using Tl = OperandTile<T, MN, KC>;
  static constexpr int J = Tl::CHUNKS / THREADS, RS = THREADS / Tl::CPR;
  static_assert(Tl::CHUNKS % THREADS == 0 && THREADS % Tl::CPR == 0, "whole rows of chunks per pass");
  static_assert(!KC || RS % 2 == 0, "the swizzle must not depend on the pass");
  const T* p;       // this thread's first chunk of the current tile
  const T* safe;    // a readable address for copies of no bytes
  ll rstride, kstep;
  unsigned dst;     // shared-memory offset (bytes) inside a stage
  unsigned rows;    // KC: valid rows, one bit per pass
  int off;          // KC: first k of the chunk; else first row k
  int bytes;        // !KC: bytes of the chunk inside the matrix
  __device__ void init(const T* base, ll ld, int mn0, int MNtot, int tid, unsigned image) {
    const int r = tid / Tl::CPR, c = tid % Tl::CPR;
    safe = base;
    rows = 0;
    bytes = 0;
    if (KC) {
      p = base + (ll)(mn0 + r) * ld + c * Tl::E;
      rstride = RS * ld;
      kstep = Tl::BK;
      off = c * Tl::E;
      dst = image + (unsigned)((r * Tl::BK + ((c ^ ((r & 1) << 2)) * Tl::E)) * (int)sizeof(T));
#pragma unroll
      for (int j = 0; j < J; ++j)
        if (mn0 + r + j * RS < MNtot) rows |= 1u << j;
    } else {
      p = base + (ll)r * ld + mn0 + c * Tl::E;
      rstride = RS * ld;
      kstep = (ll)Tl::BK * ld;
      off = r;
      dst = image + (unsigned)((r * Tl::P + c * Tl::E) * (int)sizeof(T));
      bytes = min(max(MNtot - mn0 - c * Tl::E, 0), Tl::E) * (int)sizeof(T);
    }
  }
  // copies the tile whose first k leaves krem values of k, then moves on to the next tile
  template <bool VEC>
  __device__ void load(unsigned stage, int krem) {
    constexpr unsigned DJ = (unsigned)((KC ? RS * Tl::BK : RS * Tl::P) * (int)sizeof(T));
#pragma unroll
    for (int j = 0; j < J; ++j) {
      int nb;
      if (KC) nb = ((rows >> j) & 1) ? min(max(krem - off, 0), Tl::E) * (int)sizeof(T) : 0;
      else nb = (off + j * RS < krem) ? bytes : 0;
      const T* src = nb > 0 ? p + j * rstride : safe;
      const unsigned d = stage + dst + j * DJ;
      if constexpr (VEC) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(nb));
      } else {
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(min(nb, 8)));
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d + 8), "l"(nb > 8 ? src + 1 : safe),
                     "r"(max(nb - 8, 0)));
      }
    }
    p += kstep;
  }
};

template <typename T, typename G, bool TA, bool TB>
struct GemmSmem {
  using TileA = OperandTile<T, G::BM, !TA>;
  using TileB = OperandTile<T, G::BN, TB>;
  static constexpr int SA = TileA::ELEMS, SB = TileB::ELEMS, STAGE = SA + SB;
  static constexpr size_t BYTES = (size_t)G::STAGES * STAGE * sizeof(T);
  static_assert(((size_t)SA * sizeof(T)) % 16 == 0 && ((size_t)STAGE * sizeof(T)) % 16 == 0, "16-byte tiles");
};

// What bounds it: the FP64 tensor pipe (64 multiply-adds per clock and SM) once a CTA's tiles
// stream; below about 128 tiles of work per SM the fill and drain of a CTA and the last,
// partly filled wave (see the choice of tile and K split in gemm.cu). Fragments are read with
// 16-byte loads: two values of k (contiguous along k; k is only summed over, so the two
// are handed to the instruction as its k = t and k = t + 4) or two neighbouring rows or
// columns (then rows 2 g, 2 g + 1 and columns 4 t .. 4 t + 3 of a tile belong to one thread).
// VA, VB: the operand's rows start on 16 bytes (16-byte copies, else two of 8).
template <typename T, typename G, bool TA, bool TB, bool CA, bool VA, bool VB>
__global__ void __launch_bounds__(G::THREADS) gemm_kernel(GemmArgs g) {
  using S = GemmSmem<T, G, TA, TB>;
  constexpr int BM = G::BM, BN = G::BN, WM = G::WM, WN = G::WN;
  constexpr int MI = WM / 16, NI = WN / 8, BK = S::TileA::BK;
  constexpr bool CPLX = ST<T>::cplx;
  static_assert(CPLX || NI % 2 == 0, "column pairs");
  pdl_wait();
  if (g.skip && *((volatile const int*)g.skip)) {
    if (g.Cin) {  // (a single GEMM: the slices of a split K share the tile's copy)
      const T* src = reinterpret_cast<const T*>(g.Cin);
      T* dst = reinterpret_cast<T*>(g.C);
      for (int e = blockIdx.z * G::THREADS + threadIdx.x; e < BM * BN; e += gridDim.z * G::THREADS) {
        const int row = blockIdx.y * BM + e / BN, col = blockIdx.x * BN + e % BN;
        if (row < g.M && col < g.N) dst[(ll)row * g.ldc + col] = src[(ll)row * g.ldc + col];
      }
    }
    return;
  }

  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* smem = reinterpret_cast<T*>(smem_raw);

  const int z = blockIdx.z;
  const int z1 = z / g.nb2, z2 = z - z1 * g.nb2;
  const T* Ab = reinterpret_cast<const T*>(g.A) + z1 * g.sA1 + z2 * g.sA2;
  const T* Bb = reinterpret_cast<const T*>(g.B) + z1 * g.sB1 + z2 * g.sB2;
  T* Cb = reinterpret_cast<T*>(g.C) + z1 * g.sC1 + z2 * g.sC2;
  const int M = g.M, N = g.N;
  // split-K: this CTA covers K range [kbeg, kbeg + K)
  const int kbeg = g.kchunk > 0 ? z * g.kchunk : 0;
  const int K = (g.kchunk > 0 ? min(g.K, kbeg + g.kchunk) : g.K) - kbeg;
  const ll lda = g.lda, ldb = g.ldb, ldc = g.ldc;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;

  const int tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31;
  const int wm = warp / (BN / WN) * WM, wn = warp % (BN / WN) * WN;
  const int gq = lane >> 2, tq = lane & 3;

  OperandLoader<T, BM, !TA, G::THREADS> la;
  OperandLoader<T, BN, TB, G::THREADS> lb;
  la.init(TA ? Ab + (ll)kbeg * lda : Ab + kbeg, lda, m0, M, tid, 0u);
  lb.init(TB ? Bb + kbeg : Bb + (ll)kbeg * ldb, ldb, n0, N, tid, (unsigned)(S::SA * sizeof(T)));
  const unsigned sbase = (unsigned)__cvta_generic_to_shared(smem_raw);
  constexpr unsigned SBYTES = (unsigned)(S::STAGE * sizeof(T));
  int krem = K;  // values of k not yet requested
  auto load_stage = [&](int stage) {
    la.template load<VA>(sbase + stage * SBYTES, krem);
    lb.template load<VB>(sbase + stage * SBYTES, krem);
    krem -= BK;
  };

  double acc_re[MI][NI][4];
  double acc_im[CPLX ? MI : 1][CPLX ? NI : 1][4];
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < NI; ++j)
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        acc_re[i][j][r] = 0.0;
        if constexpr (CPLX) acc_im[i][j][r] = 0.0;
      }

  const int nk = (K + BK - 1) / BK;
#pragma unroll
  for (int s = 0; s < G::STAGES - 1; ++s) {
    if (s < nk) load_stage(s);
    cp_async_commit();
  }

  int cur = 0;
  for (int kt = 0; kt < nk; ++kt) {
    cp_async_wait<G::STAGES - 2>();
    __syncthreads();
    if (krem > 0) load_stage(cur == 0 ? G::STAGES - 1 : cur - 1);
    cp_async_commit();
    const T* As = smem + cur * S::STAGE;
    const T* Bs = As + S::SA;
    if constexpr (!CPLX) {
#pragma unroll
      for (int kg = 0; kg < 2; ++kg) {
        double a[MI][4], b[NI][2];
#pragma unroll
        for (int i = 0; i < MI; ++i) {
          if constexpr (!TA) {
            const int r0 = wm + i * 16 + gq;  // r0 + 8 has the same parity
            const int c = ((kg * 4 + tq) ^ ((gq & 1) << 2)) * 2;
            const double2 x = *reinterpret_cast<const double2*>(As + r0 * BK + c);
            const double2 y = *reinterpret_cast<const double2*>(As + (r0 + 8) * BK + c);
            a[i][0] = x.x; a[i][2] = x.y; a[i][1] = y.x; a[i][3] = y.y;
          } else {
            const double* p = As + (kg * 8 + 2 * tq) * S::TileA::P + wm + i * 16 + 2 * gq;
            const double2 x = *reinterpret_cast<const double2*>(p);
            const double2 y = *reinterpret_cast<const double2*>(p + S::TileA::P);
            a[i][0] = x.x; a[i][1] = x.y; a[i][2] = y.x; a[i][3] = y.y;
          }
        }
        if constexpr (TB) {
#pragma unroll
          for (int j = 0; j < NI; ++j) {
            const int c = ((kg * 4 + tq) ^ ((gq & 1) << 2)) * 2;
            const double2 x = *reinterpret_cast<const double2*>(Bs + (wn + j * 8 + gq) * BK + c);
            b[j][0] = x.x; b[j][1] = x.y;
          }
        } else {
#pragma unroll
          for (int j = 0; j < NI; j += 2)
#pragma unroll
            for (int s = 0; s < 2; ++s) {
              const double2 x = *reinterpret_cast<const double2*>(Bs + (kg * 8 + 2 * tq + s) * S::TileB::P + wn +
                                                                  j * 8 + 2 * gq);
              b[j][s] = x.x;
              b[j + 1][s] = x.y;
            }
        }
#pragma unroll
        for (int i = 0; i < MI; ++i)
#pragma unroll
          for (int j = 0; j < NI; ++j)
            dmma16x8x8(acc_re[i][j], a[i][0], a[i][1], a[i][2], a[i][3], b[j][0], b[j][1]);
      }
    } else {
      zc a[MI][4], b[NI][2];
#pragma unroll
      for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h) {  // k = tq, tq + 4
          const int r0 = wm + i * 16 + gq, k = tq + 4 * h;
          if constexpr (!TA) {
            const int c = k ^ ((gq & 1) << 2);
            a[i][2 * h] = As[r0 * BK + c];
            a[i][2 * h + 1] = As[(r0 + 8) * BK + c];
          } else {
            a[i][2 * h] = As[k * S::TileA::P + r0];
            a[i][2 * h + 1] = As[k * S::TileA::P + r0 + 8];
          }
        }
#pragma unroll
      for (int j = 0; j < NI; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int c0 = wn + j * 8 + gq, k = tq + 4 * h;
          b[j][h] = TB ? Bs[c0 * BK + (k ^ ((gq & 1) << 2))] : Bs[k * S::TileB::P + c0];
        }
#pragma unroll
      for (int i = 0; i < MI; ++i) {
        double ar[4], ai[4], nai[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          ar[q] = a[i][q].re;
          ai[q] = CA ? -a[i][q].im : a[i][q].im;
          nai[q] = -ai[q];
        }
#pragma unroll
        for (int j = 0; j < NI; ++j) {
          dmma16x8x8(acc_re[i][j], ar[0], ar[1], ar[2], ar[3], b[j][0].re, b[j][1].re);
          dmma16x8x8(acc_im[i][j], ar[0], ar[1], ar[2], ar[3], b[j][0].im, b[j][1].im);
        }
#pragma unroll
        for (int j = 0; j < NI; ++j) {
          dmma16x8x8(acc_re[i][j], nai[0], nai[1], nai[2], nai[3], b[j][0].im, b[j][1].im);
          dmma16x8x8(acc_im[i][j], ai[0], ai[1], ai[2], ai[3], b[j][0].re, b[j][1].re);
        }
      }
    }
    cur = (cur + 1 == G::STAGES) ? 0 : cur + 1;
  }
  cp_async_wait<0>();

  // place of accumulator r of tile (i, j) inside the CTA tile
  auto row_of = [&](int i, int r) {
    return wm + i * 16 + ((!CPLX && TA) ? 2 * gq + (r >> 1) : gq + 8 * (r >> 1));
  };
  auto col_of = [&](int j, int r) {
    return wn + ((!CPLX && !TB) ? (j & ~1) * 8 + 4 * tq + 2 * (r & 1) + (j & 1) : j * 8 + 2 * tq + (r & 1));
  };
  const bool use_beta = (g.beta_re != 0.0) || (g.beta_im != 0.0);
  const T* Ib = g.Cin ? reinterpret_cast<const T*>(g.Cin) : Cb;  // (a separate Cin is not batched)
  auto store = [&](ll at, T v0) {
    T* dst = Cb + at;
    if constexpr (!CPLX) {
      double v = g.alpha_re * v0;
      if (use_beta) v += g.beta_re * Ib[at];
      *dst = v;
    } else {
      zc v = mkz(g.alpha_re * v0.re - g.alpha_im * v0.im, g.alpha_re * v0.im + g.alpha_im * v0.re);
      if (use_beta) {
        const zc o = Ib[at];
        v.re += g.beta_re * o.re - g.beta_im * o.im;
        v.im += g.beta_re * o.im + g.beta_im * o.re;
      }
      *dst = v;
    }
  };
  if (g.kcluster > 1) {
    // split-K inside a cluster: each slice leaves its partial tile in shared memory (the
    // pipeline buffers are free now), then each CTA sums a share of the tile's rows over
    // the slices, in slice order, reading its peers' tiles (distributed shared memory)
    constexpr int PP = BN + (CPLX ? 2 : 4);  // row pitch of the partial tile
    static_assert(BM * PP <= G::STAGES * S::STAGE, "partial tile must fit the pipeline buffers");
    __syncthreads();
    T* part = smem;
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
      for (int j = 0; j < NI; ++j)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          T* p = part + row_of(i, r) * PP + col_of(j, r);
          if constexpr (!CPLX) *p = acc_re[i][j][r];
          else *p = mkz(acc_re[i][j][r], acc_im[i][j][r]);
        }
    cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    cl.sync();
    const int ns = g.kcluster, q = (int)cl.block_rank();
    const int rows_per = (BM + ns - 1) / ns;
    const int rb = q * rows_per, re = min(BM, rb + rows_per);
    for (int e = tid; e < (re - rb) * BN; e += G::THREADS) {
      const int lr = rb + e / BN, lc = e % BN;
      const int row = m0 + lr, col = n0 + lc;
      if (row < M && col < N) {
        T sum = ST<T>::zero();
        for (int zs = 0; zs < ns; ++zs) sum = sum + cl.map_shared_rank(part, zs)[lr * PP + lc];
        store((ll)row * ldc + col, sum);
      }
    }
    cl.sync();  // no CTA leaves while a peer may still read its partial tile
    return;
  }

  // epilogue
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int r2 = 0; r2 < 4; r2 += 2)
#pragma unroll
      for (int j = 0; j < NI; ++j)
#pragma unroll
        for (int r = r2; r < r2 + 2; ++r) {
          const int row = m0 + row_of(i, r), col = n0 + col_of(j, r);
          if (row < M && col < N) {
            if constexpr (!CPLX) store((ll)row * ldc + col, acc_re[i][j][r]);
            else store((ll)row * ldc + col, mkz(acc_re[i][j][r], acc_im[i][j][r]));
          }
        }
}

// Host-side description of one (possibly batched) GEMM.
template <typename T>
struct Gemm {
  bool ta = false, tb = false, ca = false;
  int M = 0, N = 0, K = 0;
  const T* A = nullptr;
  ll lda = 0, sA1 = 0, sA2 = 0;
  const T* B = nullptr;
  ll ldb = 0, sB1 = 0, sB2 = 0;
  T* C = nullptr;
  ll ldc = 0, sC1 = 0, sC2 = 0;
  int nb1 = 1, nb2 = 1;
  T alpha = ST<T>::one(), beta = ST<T>::zero();
  const int* skip = nullptr;
  const T* Cin = nullptr;  // see GemmArgs (single GEMMs only)
};

template <typename T>
void launch_gemm(const Gemm<T>& d, cudaStream_t st);

}  // namespace dmrg2
