// Host launcher and instantiations of the DMMA GEMM.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <unordered_map>
#include <vector>

#include "gemm.cuh"

namespace dmrg2 {

std::atomic<long long>& launch_counter() {
  static std::atomic<long long> c{0};
  return c;
}

long long& thread_launches() {
  thread_local long long c = 0;
  return c;
}

namespace {
// the calling thread's private stream for pool calls on the current device
cudaStream_t pool_stream(int& device) {
  constexpr int kMaxDev = 64;
  // the thread's private streams, destroyed when the thread ends
  struct Streams {
    cudaStream_t s[kMaxDev] = {};
    ~Streams() {
      for (cudaStream_t x : s)
        if (x) (void)cudaStreamDestroy(x);
    }
  };
  thread_local Streams own;
  cudaStream_t* streams = own.s;
  static std::atomic<unsigned long long> pool_ready[kMaxDev];
  DMRG2_CUDA(cudaGetDevice(&device));
  if (device < 0 || device >= kMaxDev) throw std::runtime_error("dev_alloc: device index out of range");
  if (!pool_ready[device].load()) {
    // keep freed blocks in the pool instead of returning them at each synchronisation
    cudaMemPool_t pool;
    DMRG2_CUDA(cudaDeviceGetDefaultMemPool(&pool, device));
    unsigned long long keep = ~0ull;
    DMRG2_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
    pool_ready[device].store(1);
  }
  if (!streams[device]) DMRG2_CUDA(cudaStreamCreateWithFlags(&streams[device], cudaStreamNonBlocking));
  return streams[device];
}
}  // namespace

void* dev_alloc(size_t bytes) {
  int dev = 0;
  cudaStream_t s = pool_stream(dev);
  void* p = nullptr;
  DMRG2_CUDA(cudaMallocAsync(&p, bytes ? bytes : 16, s));
  DMRG2_CUDA(cudaStreamSynchronize(s));  // usable from any stream from here on
  return p;
}

void dev_free(void* p) {
  if (!p) return;
  int dev = 0;
  cudaStream_t s = pool_stream(dev);
  cudaFreeAsync(p, s);
}

namespace {
struct PinnedCache {
  std::mutex mu;
  std::map<size_t, std::vector<void*>> free_blocks;  // size class -> idle blocks
  std::unordered_map<void*, size_t> cls;             // block -> its size class
};
PinnedCache& pinned_cache() {
  static PinnedCache* c = new PinnedCache();  // lives to process exit (blocks may outlive statics)
  return *c;
}
}  // namespace

void* host_pinned(size_t bytes) {
  size_t c = 64;
  while (c < bytes) c <<= 1;
  PinnedCache& pc = pinned_cache();
  {
    std::lock_guard<std::mutex> lk(pc.mu);
    auto& v = pc.free_blocks[c];
    if (!v.empty()) {
      void* p = v.back();
      v.pop_back();
      return p;
    }
  }
  void* p = nullptr;
  DMRG2_CUDA(cudaMallocHost(&p, c));
  std::lock_guard<std::mutex> lk(pc.mu);
  pc.cls[p] = c;
  return p;
}

void host_unpin(void* p) {
  if (!p) return;
  PinnedCache& pc = pinned_cache();
  std::lock_guard<std::mutex> lk(pc.mu);
  auto it = pc.cls.find(p);
  if (it == pc.cls.end()) return;  // not from this cache
  pc.free_blocks[it->second].push_back(p);
}

bool test_unsignalled_waits() {
  static const bool on = [] {
    const char* e = std::getenv("DMRG2_TEST_UNSIGNALLED_WAITS");
    return e && e[0] == '1';
  }();
  return on;
}

bool test_unsignalled_wait(const char* kernel) {
  static const char* e = std::getenv("DMRG2_TEST_UNSIGNALLED_WAITS");
  return e && (e[0] == '1' || std::strcmp(e, kernel) == 0);
}

template <typename T, typename G, bool TA, bool TB, bool CA, bool VA, bool VB>
static void launch_impl(const Gemm<T>& d, int splitk, cudaStream_t st) {
  using S = GemmSmem<T, G, TA, TB>;
  static std::atomic<unsigned long long> attr{0};  // per instantiation, per device
  set_smem_attr_once(attr, (const void*)gemm_kernel<T, G, TA, TB, CA, VA, VB>, (int)S::BYTES);
  GemmArgs a;
  a.M = d.M; a.N = d.N; a.K = d.K;
  a.A = d.A; a.lda = d.lda; a.sA1 = d.sA1; a.sA2 = d.sA2;
  a.B = d.B; a.ldb = d.ldb; a.sB1 = d.sB1; a.sB2 = d.sB2;
  a.C = d.C; a.ldc = d.ldc; a.sC1 = d.sC1; a.sC2 = d.sC2;
  a.nb2 = d.nb2;
  a.alpha_re = ST<T>::re(d.alpha); a.alpha_im = ST<T>::im(d.alpha);
  a.beta_re = ST<T>::re(d.beta); a.beta_im = ST<T>::im(d.beta);
  a.skip = d.skip;
  a.Cin = d.Cin;
  a.kchunk = 0;
  a.kcluster = 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ceil_div(d.N, G::BN), ceil_div(d.M, G::BM), d.nb1 * d.nb2);
  cfg.blockDim = dim3(G::THREADS);
  cfg.dynamicSmemBytes = S::BYTES;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0] = pdl_attribute();
  cfg.attrs = at;
  cfg.numAttrs = 1;
  constexpr int BK = S::TileA::BK;
  const int chunk = ceil_div(ceil_div(d.K, splitk), BK) * BK;
  const int nsplit = ceil_div(d.K, chunk);
  if (nsplit > 1) {
    // the slices of a tile form one cluster and are summed in it, in slice order: no
    // workspace, no second launch
    a.kchunk = chunk;
    a.kcluster = nsplit;
    a.sA1 = a.sA2 = a.sB1 = a.sB2 = a.sC1 = a.sC2 = 0;
    a.nb2 = 1;
    cfg.gridDim.z = nsplit;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = 1;
    at[1].val.clusterDim.y = 1;
    at[1].val.clusterDim.z = nsplit;
    cfg.numAttrs = 2;
  }
  DMRG2_CUDA(cudaLaunchKernelEx(&cfg, gemm_kernel<T, G, TA, TB, CA, VA, VB>, a));
  DMRG2_CHECK_LAUNCH();
}

// whether every row of an operand starts on 16 bytes
template <typename T>
static bool rows16(const T* p, ll ld, ll s1, ll s2) {
  return sizeof(T) == 16 || (((ld | s1 | s2) & 1) == 0 && ((uintptr_t)p & 15) == 0);
}

template <typename T, typename G, bool TA, bool TB, bool CA>
static void launch_vec(const Gemm<T>& d, int splitk, cudaStream_t st) {
  if constexpr (ST<T>::cplx) {
    launch_impl<T, G, TA, TB, CA, true, true>(d, splitk, st);
  } else {
    const bool va = rows16(d.A, d.lda, d.sA1, d.sA2), vb = rows16(d.B, d.ldb, d.sB1, d.sB2);
    if (va && vb) launch_impl<T, G, TA, TB, CA, true, true>(d, splitk, st);
    else if (va) launch_impl<T, G, TA, TB, CA, true, false>(d, splitk, st);
    else if (vb) launch_impl<T, G, TA, TB, CA, false, true>(d, splitk, st);
    else launch_impl<T, G, TA, TB, CA, false, false>(d, splitk, st);
  }
}

template <typename T, typename G>
static void dispatch(const Gemm<T>& d, int splitk, cudaStream_t st) {
  const bool ca = ST<T>::cplx && d.ca;
  if (!d.ta && !d.tb && !ca) return launch_vec<T, G, false, false, false>(d, splitk, st);
  if (!d.ta && d.tb && !ca) return launch_vec<T, G, false, true, false>(d, splitk, st);
  if (d.ta && !d.tb && !ca) return launch_vec<T, G, true, false, false>(d, splitk, st);
  if (d.ta && d.tb && !ca) return launch_vec<T, G, true, true, false>(d, splitk, st);
  if constexpr (ST<T>::cplx) {
    if (!d.ta && !d.tb) return launch_vec<T, G, false, false, true>(d, splitk, st);
    if (!d.ta && d.tb) return launch_vec<T, G, false, true, true>(d, splitk, st);
    if (d.ta && !d.tb) return launch_vec<T, G, true, false, true>(d, splitk, st);
    return launch_vec<T, G, true, true, true>(d, splitk, st);
  }
}

namespace {
struct GemmChoice {
  int tile;    // index into the tiles of the scalar type (launch_choice)
  int splitk;  // K slices (a cluster of at most 8)
};

// Tile and K split by a model of the busiest SM. It runs q = ceil(CTAs / 148) tiles of
// BM BN K / splitk multiply-adds; the tensor pipe takes 64 (16 complex) a cycle, but only with
// enough warps resident to cover the latency of a warp's dependent multiply-adds: the
// share of the rate is 0.60 with 4 warps on the SM, 0.82 with 8, 0.86 with 12, 0.90 with 16 and
// 0.92 beyond (L2-resident operands, K from 64 to 1280). Moving the operands adds 0.05 cycles per row
// and column and value of k (smaller tiles read them more often), 0.25 where its rows do not start on
// 16 bytes (twice the copies, half the bytes), and a split 1200 cycles per CTA of the SM and 100
// more per slice (cluster barrier, exchange of partial tiles). Real constants fitted to 58 shapes of H_eff,
// environment and split GEMMs at chi = 64 to 512, each measured in all 24 configurations: the choice
// costs 3.9% over the best one on average (5.6% without the operands' term and with 1600 cycles
// for any split); complex ones as first measured. Some of them, M x N x K: 1280 x 1024 x 256 (64 x 64
// tiles: 2.16 CTAs an SM run as three, 35.2 us; 64 x 32 28.9; 32 x 32 26.9), 1024 x 256 x 1280 (64 x 64 in
// 5 slices 37.1; 4 slices 29.8; 32 x 32 unsplit 30.5, in 4 slices 31.9), 512 x 128 x 640 (64 x 64 in 8
// slices 11.3; 32 x 32 unsplit 13.9, in 4 slices 7.7), 320 x 256 x 64 (64 x 64 6.4; 32 x 32 4.3).
//
// Long real sums: a rounding error is made against the running value at each addition, and H_eff's
// last step at chi = 256 (K = 1280) in one chain left a matvec 7.6e-16 from the exact result, where four
// slices leave 5.4e-16 (J1-J2, 171 x 187, K = 1496: two slices 8.7e-16, eight 7.3e-16). So sums over more than
// 512 values go in slices of at most 384, where the output has fewer 64 x 64 tiles than there are SMs
// (a larger one loses up to 15% to the exchange: 1024^3 79.9 us unsplit, 91.8 in 4 slices). A
// complex product keeps its chain: two slices would take the Josephson matvec at chi = 128 (K = 512)
// from 7.0e-16 to 6.1e-16, and from 151 to 161 us.
struct TileModel {
  int bm, bn;
  int occ;  // CTAs an SM holds (four warps each)
};
constexpr TileModel TILES_D[] = {{64, 64, 3}, {64, 32, 4}, {32, 32, 6}};
constexpr TileModel TILES_Z[] = {{64, 32, 4}, {32, 32, 6}};

template <typename T>
GemmChoice choose(const Gemm<T>& d) {
  constexpr bool real = !ST<T>::cplx;
  constexpr double share[] = {real ? 0.60 : 0.62, 0.82, 0.86, 0.90, 0.92, 0.92};
  constexpr double move = real ? 0.05 : 0.0, split_cta = real ? 1200.0 : 1600.0, split_slice = real ? 100.0 : 0.0;
  const TileModel* tiles = ST<T>::cplx ? TILES_Z : TILES_D;
  const int nt = ST<T>::cplx ? 2 : 3;
  const double rate = ST<T>::cplx ? 16.0 : 64.0;
  const int bk = ST<T>::cplx ? 8 : 16;
  const int nb = d.nb1 * d.nb2;
  const double narrow_a = rows16(d.A, d.lda, d.sA1, d.sA2) ? 0.0 : 8.0 / 32;
  const double narrow_b = rows16(d.B, d.ldb, d.sB1, d.sB2) ? 0.0 : 8.0 / 32;
  const bool slices = real && nb == 1 && d.K > 512 && ceil_div(d.M, 64) * (ll)ceil_div(d.N, 64) < 148;
  GemmChoice best{0, 1};
  double best_t = 1e300;
  for (int t = 0; t < nt; ++t) {
    const double out = (double)ceil_div(d.M, tiles[t].bm) * ceil_div(d.N, tiles[t].bn) * nb;
    for (int sk = 1; sk <= (nb == 1 ? 8 : 1); ++sk) {
      if (sk > 1 && ceil_div(d.K, sk) < 2 * bk) break;  // at least two k tiles per slice
      const int kc = ceil_div(ceil_div(d.K, sk), bk) * bk, ns = ceil_div(d.K, kc);
      if (ns < sk) continue;
      if (slices && kc > 384 && sk < 8) continue;
      const double q = std::ceil(out * ns / 148.0);
      const double f = share[std::min((int)std::min(q, 6.0), tiles[t].occ) - 1];
      const double time = q * (tiles[t].bm * tiles[t].bn * (double)kc / rate / f +
                               (ns > 1 ? split_cta + split_slice * ns : 0.0) +
                               kc * ((narrow_a + move) * tiles[t].bm + (narrow_b + move) * tiles[t].bn));
      if (time < best_t) {
        best_t = time;
        best = {t, ns};
      }
    }
  }
  return best;
}

template <typename T>
void launch_choice(const Gemm<T>& d, const GemmChoice& c, cudaStream_t st) {
  if constexpr (ST<T>::cplx) {
    if (c.tile == 0) dispatch<T, TileZ64>(d, c.splitk, st);
    else dispatch<T, TileZ32>(d, c.splitk, st);
  } else {
    if (c.tile == 0) dispatch<T, TileD64>(d, c.splitk, st);
    else if (c.tile == 1) dispatch<T, TileD64x32>(d, c.splitk, st);
    else dispatch<T, TileD32>(d, c.splitk, st);
  }
}
}  // namespace

// ---------------------------------------------------------------- autotuner
// A single real GEMM of at least TUNE_MIN_FLOP is run in each configuration (every tile with 1, 2, 4
// or 8 K slices) the first time its shape (transposes, M, N, K) occurs in the process, on the
// caller's stream and operands, writing into a scratch output (never the caller's C, no skip
// flag); the fastest by CUDA events serves every later GEMM of that shape. Smaller GEMMs
// are latency-bound and keep the model's choice: their many distinct shapes (chain ends,
// bond-dimension ramps) would cost more to time than a configuration can save. The tuning is off
// unless DMRG2_GEMM_TUNE=1: measured on the L=100, chi=256 sweep it gains 2% on steady sweeps but
// loses 10% on a run that starts from a fresh engine (the choices timed in isolation, on
// L2-resident operands, do not carry over to the sweep's own cache state), and off, results do not
// depend on timing.
namespace {
struct TuneKey {
  int ta, tb, M, N, K, dev;
  bool operator==(const TuneKey& o) const {
    return ta == o.ta && tb == o.tb && M == o.M && N == o.N && K == o.K && dev == o.dev;
  }
};
struct TuneKeyHash {
  size_t operator()(const TuneKey& k) const {
    size_t h = (size_t)k.M * 1000003u ^ (size_t)k.N * 9176u ^ (size_t)k.K * 31u;
    return h ^ (size_t)(k.ta * 2 + k.tb) ^ ((size_t)k.dev << 40);
  }
};
constexpr double TUNE_MIN_FLOP = 1e8;
std::mutex& tune_mutex() {
  static std::mutex m;
  return m;
}
std::unordered_map<TuneKey, GemmChoice, TuneKeyHash>& tune_cache() {
  static auto* c = new std::unordered_map<TuneKey, GemmChoice, TuneKeyHash>();
  return *c;
}
}  // namespace

bool tune_enabled() {
  static const bool on = [] {
    const char* e = std::getenv("DMRG2_GEMM_TUNE");
    return e && e[0] == '1';
  }();
  return on;
}

namespace {
GemmChoice tuned(const Gemm<double>& d, cudaStream_t st) {
  int dev = 0;
  DMRG2_CUDA(cudaGetDevice(&dev));
  const TuneKey key{d.ta ? 1 : 0, d.tb ? 1 : 0, d.M, d.N, d.K, dev};
  std::lock_guard<std::mutex> lk(tune_mutex());
  auto it = tune_cache().find(key);
  if (it != tune_cache().end()) return it->second;
  Gemm<double> t = d;
  t.skip = nullptr;
  t.Cin = nullptr;
  t.beta = 0.0;
  t.ldc = d.N;
  t.sC1 = t.sC2 = 0;
  t.C = (double*)dev_alloc(sizeof(double) * (size_t)d.M * d.N);
  cudaEvent_t e0, e1;
  DMRG2_CUDA(cudaEventCreate(&e0));
  DMRG2_CUDA(cudaEventCreate(&e1));
  GemmChoice best{0, 1};
  float best_ms = 1e30f;
  for (int tile = 0; tile < 3; ++tile)
    for (int sk = 1; sk <= 8; sk *= 2) {
      if (sk > 1 && d.K < 32 * sk) continue;  // at least two k-tiles per slice
      auto run = [&]() { launch_choice<double>(t, {tile, sk}, st); };
      run();  // first launch: attributes, instruction cache
      DMRG2_CUDA(cudaEventRecord(e0, st));
      for (int r = 0; r < 2; ++r) run();
      DMRG2_CUDA(cudaEventRecord(e1, st));
      DMRG2_CUDA(cudaEventSynchronize(e1));
      float ms = 0.f;
      DMRG2_CUDA(cudaEventElapsedTime(&ms, e0, e1));
      if (ms < best_ms) {
        best_ms = ms;
        best = {tile, sk};
      }
    }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  dev_free(t.C);  // the stream is idle after the last event
  tune_cache()[key] = best;
  return best;
}
}  // namespace

template <typename T>
void launch_gemm(const Gemm<T>& d, cudaStream_t st) {
  if (d.M <= 0 || d.N <= 0 || d.nb1 * d.nb2 <= 0) return;
  if (d.nb1 * d.nb2 > 65535) throw std::runtime_error("gemm: batch count exceeds 65535");
  if (d.Cin && d.nb1 * d.nb2 != 1) throw std::runtime_error("gemm: a separate Cin needs a single GEMM");
  if (ceil_div(d.M, TileD32::BM) > 65535) throw std::runtime_error("gemm: M too large");
  if constexpr (!ST<T>::cplx) {
    if (d.nb1 * d.nb2 == 1 && 2.0 * d.M * d.N * d.K >= TUNE_MIN_FLOP && tune_enabled()) {
      return launch_choice<T>(d, tuned(d, st), st);
    }
  }
  launch_choice<T>(d, choose<T>(d), st);
}

template void launch_gemm<double>(const Gemm<double>&, cudaStream_t);
template void launch_gemm<zc>(const Gemm<zc>&, cudaStream_t);

}  // namespace dmrg2
