// Host driver of one Lanczos ground-state solve on the device.
//
// Two forms, the same arithmetic:
//  - host-driven: the host enqueues Krylov iterations ahead of the device and polls the
//    device-side `done` flag through a small pinned ring with a lookahead of POLL_LOOK
//    iterations, so the GPU never idles on the host and at most POLL_LOOK iterations of
//    no-op launches are issued after convergence;
//  - device-looped: one CUDA graph per matvec identity (operator shapes and the fixed
//    buffers it reads and writes) holds the whole solve: the start (norms, reset, first
//    vector), a conditional WHILE node whose body is one Krylov step (matvec, then the
//    step kernel, which also advances the index and ends the loop on convergence or after
//    kmax bodies), then the Ritz vector, with the solver's report into pinned host memory.
//    The host writes a seed there, launches the graph once per restart and waits once; no flags cross to the host between steps and no no-op steps are issued. A call
//    site opts in by passing a key; solves run host-driven until a key is met the second
//    time, when the solve is followed by the capture (graphs.cuh holds the cache).
#pragma once

#include <algorithm>
#include <array>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <stdexcept>
#include <vector>

#include "common.cuh"
#include "graphs.cuh"
#include "kernels.cuh"

namespace dmrg2 {

// identifies a matvec for the graph cache: operator shapes and device pointers, chosen by
// the caller (unused entries 0); the solve adds n, kmax, the tolerance and its buffers
using LzKey = std::array<long long, 11>;

// a converged chi=256 sweep of 100 sites meets ~100 distinct (cL, cR) bond shapes (bonds
// below the cap keep what the cutoff leaves); a graph is a few kilobytes
constexpr int LZ_GRAPH_CAP = 1024;

// Blocks a solve's cooperative kernels may have (vectors beyond the cluster form): one per SM this
// context has (fewer than 148 in a partition of the GPU). None where other streams run Jacobi
// kernels beside the solve (`shared`): a cooperative kernel starts only once every SM can take
// one of its blocks, a Jacobi split holds some SMs for tens of milliseconds, and all solves wait for
// it at every Krylov step, where the streaming passes fit in between. Segments of a parallel sweep
// (L = 100, chi = 256, ms per iteration of 2 / 4 / 8 segments): 281 / 431 / 1235 cooperative,
// 239 / 400 / 509 with 74 blocks, 243 / 360 / 494 streaming. Engines with Jacobi splits (L = 30,
// chi = 128, s for 1 / 4 / 6 at once): 2.31 / 2.60 / 2.98 cooperative, 2.31 / 2.39 / 2.51 streaming.
// Engines with the other splits gain from the cooperative form also together (8 requests at
// L = 40, chi = 256: 1.36 s streaming, 0.77 s with all of the cooperative form's changes).
// DMRG2_TEST_STEP_BLOCKS caps the count (tests).
inline int cooperative_step_blocks(bool shared) {
  if (shared) return 0;
  int dev = 0, sms = 0;
  DMRG2_CUDA(cudaGetDevice(&dev));
  DMRG2_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  if (const char* e = std::getenv("DMRG2_TEST_STEP_BLOCKS")) sms = std::min(sms, std::atoi(e));
  return std::min(sms, STEP_BLOCKS);
}

template <typename T>
struct LanczosWork {
  static constexpr int POLL_RING = 8;
  static constexpr int POLL_LOOK = 2;
  T* krylov = nullptr;  // kcap vectors of length >= n
  T* w = nullptr;       // work vector
  T* cur = nullptr;     // the device-looped matvec's input (a copy of the current Krylov vector)
  GraphCache graphs;    // device-looped solves, by key
  int kcap = 0;
  LanczosDev* st = nullptr;
  RedScratch red;
  int* h_flags = nullptr;
  LanczosHost* h_st = nullptr;  // the solve's report (pinned, written by its last kernel)
  bool pending = false;         // a deferred solve has not been collected
  unsigned* h_seed = nullptr;   // the device-looped solve's seed (pinned, read by its first kernel)
  std::vector<cudaEvent_t> ev_poll, ev_mv;
  std::vector<void*> owned;

  // timing: the host-driven form measures its matvecs (an event pair per Krylov step)
  // shared: see cooperative_step_blocks
  void init(int kcap_, ll nmax, bool timing = true, bool shared = false) {
    red.step_blocks = cooperative_step_blocks(shared);
    graphs.cap = LZ_GRAPH_CAP;
    graphs.name = "lanczos";
    kcap = std::min(kcap_, KRYLOV_CAP);
    red.nblk = red_blocks(nmax);
    DevSlab slab;
    slab.add(krylov, sizeof(T) * (size_t)kcap * std::max<ll>(nmax, 1));
    slab.add(w, sizeof(T) * (size_t)std::max<ll>(nmax, 1));
    slab.add(cur, sizeof(T) * (size_t)std::max<ll>(nmax, 1));
    slab.add(st, sizeof(LanczosDev));
    slab.add(red.part, sizeof(double) * (size_t)red.nblk * 2 * (KRYLOV_CAP + 2));
    slab.add(red.counter, sizeof(unsigned) * 4);
    owned.push_back(slab.commit());
    DMRG2_CUDA(cudaMemset(red.counter, 0, sizeof(unsigned) * 4));
    DMRG2_CUDA(cudaMemset(st, 0, sizeof(LanczosDev)));
    // the barrier counters are zero before the solve's own stream, which does not wait for the
    // legacy one, may count on them
    DMRG2_CUDA(cudaStreamSynchronize(cudaStreamLegacy));
    h_flags = (int*)host_pinned(sizeof(int) * POLL_RING);
    h_st = (LanczosHost*)host_pinned(sizeof(LanczosHost));
    h_seed = (unsigned*)host_pinned(sizeof(unsigned));
    ev_poll.resize(POLL_RING);
    for (auto& e : ev_poll) DMRG2_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    ev_mv.resize(timing ? 2 * (size_t)kcap : 0);
    for (auto& e : ev_mv) DMRG2_CUDA(cudaEventCreate(&e));
  }
  size_t bytes(ll nmax) const {
    return sizeof(T) * ((size_t)kcap + 2) * (size_t)nmax + sizeof(LanczosDev) +
           sizeof(double) * (size_t)red.nblk * 2 * (KRYLOV_CAP + 2);
  }
  void release() {
    graphs.clear();
    for (void* p : owned) dev_free(p);
    owned.clear();
    if (h_flags) host_unpin(h_flags);
    if (h_st) host_unpin(h_st);
    if (h_seed) host_unpin(h_seed);
    h_flags = nullptr;
    h_st = nullptr;
    h_seed = nullptr;
    for (auto e : ev_poll) cudaEventDestroy(e);
    for (auto e : ev_mv) cudaEventDestroy(e);
    ev_poll.clear();
    ev_mv.clear();
  }
};

struct LanczosResult {
  double energy = 0.0;
  int iters = 0;         // Krylov vectors built (all passes)
  int matvecs = 0;
  int converged = 0;
  double matvec_s = 0.0;  // device time of the matvecs
  int device_loops = 0;   // restarts run as the device-looped graph
  int lowprec = 0;        // of the matvecs, those on the split-BF16 operator (set by the engine)
  bool pending = false;   // enqueued only: lanczos_collect completes it once the stream has run it
  long long launches = 0, fixed = 0;  // kernels per loop body and around the loop (pending solves)
};

// throws where the finished solve (W.h_st) left no result
template <typename T>
void lanczos_check(LanczosWork<T>& W, cudaStream_t s) {
  const LanczosHost& h = *W.h_st;
  if (h.done && h.n_iter >= 1 && !h.gave_up) return;
  // (a grid barrier that gave up leaves its counters behind)
  DMRG2_CUDA(cudaMemsetAsync(W.st, 0, sizeof(LanczosDev), s));
  throw std::runtime_error("Lanczos did not terminate");
}

// Adds what the finished solve reported (W.h_st) to res; s: its stream (idle up to the solve's end).
template <typename T>
void lanczos_collect(LanczosWork<T>& W, LanczosResult& res, cudaStream_t s) {
  const LanczosHost& h = *W.h_st;
  W.pending = false;
  lanczos_check(W, s);
  launch_counter() += h.guard * res.launches + res.fixed;
  thread_launches() += h.guard * res.launches + res.fixed;
  res.matvecs += h.guard;
  res.iters += h.n_iter;
  res.energy = h.e_cur;
  res.matvec_s += (double)h.mv_ns * 1e-9;
  res.converged = h.converged;
  res.device_loops += 1;
  res.pending = false;
}

// Captures one solve of W's buffers and this matvec into G (nothing runs): the start
// (norm, first vector), the WHILE node over the Krylov steps, the Ritz vector with the
// report to W.h_st.
template <typename T>
void lz_build_graph(LanczosWork<T>& W, GraphEntry& G, T* theta, ll n, int kmax, double tol,
                    const std::function<void(const T*, T*, const int*)>& matvec, cudaStream_t s) {
  DMRG2_CUDA(cudaGraphCreate(&G.g, 0));
  G.fixed = capture_to_graph(s, G.g, [&]() {
    lz_start(theta, W.krylov, n, W.st, W.red, 0u, tol, kmax, s, W.cur, W.h_seed);
  });
  const cudaGraphNode_t start = graph_leaf(G.g);
  cudaGraphConditionalHandle h;
  DMRG2_CUDA(cudaGraphConditionalHandleCreate(&h, G.g, 1, cudaGraphCondAssignDefault));
  cudaGraphNodeParams p{};
  p.type = cudaGraphNodeTypeConditional;
  p.conditional.handle = h;
  p.conditional.type = cudaGraphCondTypeWhile;
  p.conditional.size = 1;
  cudaGraphNode_t loop;
  DMRG2_CUDA(cudaGraphAddNode(&loop, G.g, &start, 1, &p));
  G.launches = capture_to_graph(s, p.conditional.phGraph_out[0], [&]() {
    matvec(W.cur, W.w, &W.st->done);
    lz_step_dev(W.krylov, n, W.w, W.cur, W.st, W.red, kmax, h, s);
  });
  G.fixed += capture_to_graph(
      s, G.g,
      [&]() {
        lz_ritz(W.krylov, n, theta, W.st, W.red, W.h_st, s);
      },
      &loop);
  graph_instantiate(W.graphs, G);
}

// matvec(in, out, skip_flag) enqueues out = H in on stream s, doing nothing when
// *skip_flag != 0 on the device. theta: start vector on entry, normalised Ritz
// vector on exit. With a key: the device-looped form, cached in W.graphs (the key must
// identify everything the matvec reads and writes besides in and out). With defer, a
// device-looped solve without restarts is only enqueued (res.pending): the caller enqueues what
// follows, waits for the stream and calls lanczos_collect, one host round trip less. Until then
// what follows may write what must outlast a failed solve only where W.st->gave_up is not set.
template <typename T>
LanczosResult lanczos_solve(LanczosWork<T>& W, T* theta, ll n, int krylov_max, double tol,
                            int max_restarts, unsigned seed,
                            const std::function<void(const T*, T*, const int*)>& matvec,
                            cudaStream_t s, const LzKey* key = nullptr, bool defer = false) {
  LanczosResult res;
  if (W.pending) {  // an error kept the caller from collecting the last solve: leave nothing of it
    W.pending = false;
    DMRG2_CUDA(cudaStreamSynchronize(s));
    DMRG2_CUDA(cudaMemsetAsync(W.st, 0, sizeof(LanczosDev), s));
  }
  const bool timed = !W.ev_mv.empty();
  const int kmax = (int)std::min<ll>(std::min(krylov_max, W.kcap), n);
  if (kmax < 1) throw std::runtime_error("lanczos: empty problem");
  GraphEntry* G = nullptr;
  bool build = false;
  if (key && graphs_enabled()) {
    GraphKey k{};
    std::copy(key->begin(), key->end(), k.begin());
    double tol_key = tol;
    long long tol_bits = 0;
    std::memcpy(&tol_bits, &tol_key, sizeof(tol_bits));
    k[11] = n;
    k[12] = kmax;
    k[13] = tol_bits;
    k[14] = (ll)theta;
    k[15] = (ll)&W;
    G = W.graphs.find(k);
    if (!G && W.graphs.seen_before(k)) {
      G = W.graphs.slot(k);
      build = true;
    }
  }
  for (int rs = 0; rs <= max_restarts; ++rs) {
    W.h_st->gave_up = 0;  // (the last solve on W has been waited for)
    if (G && G->ex) {
      // the solve reads the pinned seed before the host writes it again (the wait below)
      *W.h_seed = seed + 104729u * (unsigned)rs;
      DMRG2_CUDA(cudaGraphLaunch(G->ex, s));
      W.graphs.replays += 1;
      res.launches = G->launches;
      res.fixed = G->fixed;
      if (defer && max_restarts == 0) {
        int left = lz_fail_countdown().load();
        if (left > 0 && --lz_fail_countdown() == 0) lz_fail(W.st, W.h_st, s);
        W.pending = res.pending = true;
        return res;
      }
      DMRG2_CUDA(cudaStreamSynchronize(s));
      lanczos_collect(W, res, s);
      if (res.converged) break;
      continue;
    }
    lz_start(theta, W.krylov, n, W.st, W.red, seed + 104729u * (unsigned)rs, tol, kmax, s);
    int issued = 0;
    for (int j = 0; j < kmax; ++j) {
      if (j >= LanczosWork<T>::POLL_LOOK) {
        int jj = j - LanczosWork<T>::POLL_LOOK;
        DMRG2_CUDA(cudaEventSynchronize(W.ev_poll[jj % LanczosWork<T>::POLL_RING]));
        if (W.h_flags[jj % LanczosWork<T>::POLL_RING]) break;
      }
      T* vj = W.krylov + (ll)j * n;
      if (timed) DMRG2_CUDA(cudaEventRecord(W.ev_mv[2 * j], s));
      matvec(vj, W.w, &W.st->done);
      if (timed) DMRG2_CUDA(cudaEventRecord(W.ev_mv[2 * j + 1], s));
      lz_step(W.krylov, j + 1, n, W.w, W.st, W.red, kmax, &W.h_flags[j % LanczosWork<T>::POLL_RING], s);
      DMRG2_CUDA(cudaEventRecord(W.ev_poll[j % LanczosWork<T>::POLL_RING], s));
      issued = j + 1;
    }
    lz_ritz(W.krylov, n, theta, W.st, W.red, W.h_st, s);
    DMRG2_CUDA(cudaStreamSynchronize(s));
    lanczos_check(W, s);
    const int used = std::min(issued, W.h_st->n_iter);
    for (int j = 0; timed && j < used; ++j) {
      float ms = 0.f;
      DMRG2_CUDA(cudaEventElapsedTime(&ms, W.ev_mv[2 * j], W.ev_mv[2 * j + 1]));
      res.matvec_s += ms * 1e-3;
    }
    res.matvecs += used;
    res.iters += W.h_st->n_iter;
    res.energy = W.h_st->e_cur;
    res.converged = W.h_st->converged;
    if (res.converged) break;
  }
  if (build) {
    try {
      const auto t0 = std::chrono::steady_clock::now();
      lz_build_graph(W, *G, theta, n, kmax, tol, matvec, s);
      W.graphs.builds += 1;
      W.graphs.build_s += std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    } catch (const std::exception& e) {
      G->reset();
      graphs_disable(e.what());
    }
  }
  return res;
}

}  // namespace dmrg2
