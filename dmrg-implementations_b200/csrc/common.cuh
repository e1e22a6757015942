// Shared scalar types, error handling and small device helpers.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <stdexcept>
#include <string>
#include <vector>

namespace dmrg2 {

typedef long long ll;

struct __align__(16) zc {
  double re, im;
};

__host__ __device__ inline zc mkz(double r, double i) { zc z; z.re = r; z.im = i; return z; }
__host__ __device__ inline zc operator+(zc a, zc b) { return mkz(a.re + b.re, a.im + b.im); }
__host__ __device__ inline zc operator-(zc a, zc b) { return mkz(a.re - b.re, a.im - b.im); }
__host__ __device__ inline zc operator*(zc a, zc b) {
  return mkz(a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re);
}
__host__ __device__ inline zc operator*(double s, zc a) { return mkz(s * a.re, s * a.im); }

// Scalar traits: real double or complex double (interleaved re, im).
template <typename T> struct ST;
template <> struct ST<double> {
  static constexpr bool cplx = false;
  __host__ __device__ static double zero() { return 0.0; }
  __host__ __device__ static double one() { return 1.0; }
  __host__ __device__ static double conj(double a) { return a; }
  __host__ __device__ static double re(double a) { return a; }
  __host__ __device__ static double im(double) { return 0.0; }
  __host__ __device__ static double abs2(double a) { return a * a; }
  __host__ __device__ static bool finite(double a) { return a - a == 0.0; }
  __host__ __device__ static bool nonzero(double a) { return a != 0.0; }
#ifdef __CUDACC__
  // the top half without its sign: at least 0x7ff00000 for an infinity or a NaN only
  __device__ static unsigned exponent_bits(double a) { return (unsigned)__double2hiint(a) & 0x7fffffffu; }
#endif
  __host__ __device__ static double make(double r, double) { return r; }
  __host__ __device__ static double mul(double a, double b) { return a * b; }
  __host__ __device__ static double add(double a, double b) { return a + b; }
  __host__ __device__ static double scale(double s, double a) { return s * a; }
  // conj(a) * b
  __host__ __device__ static double cmul(double a, double b) { return a * b; }
};
template <> struct ST<zc> {
  static constexpr bool cplx = true;
  __host__ __device__ static zc zero() { return mkz(0, 0); }
  __host__ __device__ static zc one() { return mkz(1, 0); }
  __host__ __device__ static zc conj(zc a) { return mkz(a.re, -a.im); }
  __host__ __device__ static double re(zc a) { return a.re; }
  __host__ __device__ static double im(zc a) { return a.im; }
  __host__ __device__ static double abs2(zc a) { return a.re * a.re + a.im * a.im; }
  __host__ __device__ static bool finite(zc a) { return a.re - a.re == 0.0 && a.im - a.im == 0.0; }
  __host__ __device__ static bool nonzero(zc a) { return a.re != 0.0 || a.im != 0.0; }
#ifdef __CUDACC__
  __device__ static unsigned exponent_bits(zc a) {
    const unsigned r = ST<double>::exponent_bits(a.re), i = ST<double>::exponent_bits(a.im);
    return r > i ? r : i;
  }
#endif
  __host__ __device__ static zc make(double r, double i) { return mkz(r, i); }
  __host__ __device__ static zc mul(zc a, zc b) { return a * b; }
  __host__ __device__ static zc add(zc a, zc b) { return a + b; }
  __host__ __device__ static zc scale(double s, zc a) { return mkz(s * a.re, s * a.im); }
  __host__ __device__ static zc cmul(zc a, zc b) {
    return mkz(a.re * b.re + a.im * b.im, a.re * b.im - a.im * b.re);
  }
};

struct CudaError : public std::runtime_error {
  explicit CudaError(const std::string& s) : std::runtime_error(s) {}
};

// A numerical method did not reach its accuracy (reported as DMRG2_ERR_NUMERIC).
struct NumericError : public std::runtime_error {
  explicit NumericError(const std::string& s) : std::runtime_error(s) {}
};

#define DMRG2_CUDA(call)                                                              \
  do {                                                                                \
    cudaError_t e_ = (call);                                                          \
    if (e_ != cudaSuccess) {                                                          \
      throw ::dmrg2::CudaError(std::string("CUDA error ") + cudaGetErrorString(e_) +  \
                               " at " + __FILE__ + ":" + std::to_string(__LINE__) +   \
                               " (" #call ")");                                       \
    }                                                                                 \
  } while (0)

// Every kernel launch of the library goes through DMRG2_CHECK_LAUNCH, which
// also counts it (reported through dmrg2_get_launch_count).
std::atomic<long long>& launch_counter();  // kernels launched by this library (all threads)
long long& thread_launches();              // the same, by the calling thread
#define DMRG2_CHECK_LAUNCH()            \
  do {                                  \
    DMRG2_CUDA(cudaGetLastError());     \
    ++::dmrg2::launch_counter();        \
    ++::dmrg2::thread_launches();       \
  } while (0)

// Programmatic dependent launch. A kernel launched by launch_pdl (or with pdl_attribute) may be
// scheduled as its predecessor in the stream drains; it waits for the predecessor's completion
// (and its memory) in pdl_wait, which every thread calls before it reads or writes global
// memory and before any early return, so the order of the stream is kept. Between kernels of a
// few microseconds this hides part of the launch latency (a matvec at 8 x 16: 14.3 -> 10.3 us).
// No kernel triggers its successor early (griddepcontrol.launch_dependents): successors that
// wait on the SMs unbalance the running kernel's CTAs (a matvec at chi = 256: 75 -> 104 us).
#ifdef __CUDACC__
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
inline cudaLaunchAttribute pdl_attribute() {
  cudaLaunchAttribute a{};
  a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  a.val.programmaticStreamSerializationAllowed = 1;
  return a;
}
template <typename... P, typename... A>
void launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at = pdl_attribute();
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  DMRG2_CUDA(cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...));
  DMRG2_CHECK_LAUNCH();
}
#endif

// GEMMs pick their tile shapes by timing candidates (DMRG2_GEMM_TUNE=1)
bool tune_enabled();

inline int ceil_div(ll a, ll b) { return (int)((a + b - 1) / b); }

// Test hook for the bounded device waits: with DMRG2_TEST_UNSIGNALLED_WAITS=1 in the
// environment, the kernels that wait on a completion (the tensor-core commit of the
// split GEMM, the grid barriers of the cooperative Jacobi SVD and of the cooperative Lanczos
// kernels) wait on one that nothing signals, with a short poll limit, so a test can see the
// timeout reported as DMRG2_ERR_NUMERIC while the device stays usable. The value start, step
// or ritz picks that Lanczos kernel alone. In the Lanczos kernels it is the last block's wait.
bool test_unsignalled_waits();
bool test_unsignalled_wait(const char* kernel);

// Device memory of the library, from the device's stream-ordered pool (cudaMallocAsync
// on a private stream of the calling thread, which the call then waits for). Unlike
// cudaMalloc / cudaFree, neither call synchronises the device, so an engine that is created
// or destroyed while others run (the served form) does not stall their streams; the pool
// keeps released memory for the next allocation. dev_free requires that no stream still
// uses the memory (owners synchronise their stream first).
void* dev_alloc(size_t bytes);
void dev_free(void* p);

// Several buffers in one dev_alloc: every buffer is asked for first (add), then carved in 256-byte
// aligned slices (commit). An allocation and its wait cost about 10 us; a truncation's or a
// Lanczos solve's workspace has a dozen buffers.
class DevSlab {
 public:
  template <typename P>
  void add(P*& p, size_t bytes) {
    items_.push_back({(void**)&p, bytes});
  }
  // returns the block to free with dev_free
  void* commit() {
    size_t total = 0;
    for (const Item& i : items_) total += round(i.bytes);
    char* base = (char*)dev_alloc(total);
    size_t off = 0;
    for (const Item& i : items_) {
      *i.p = base + off;
      off += round(i.bytes);
    }
    items_.clear();
    return base;
  }

 private:
  struct Item {
    void** p;
    size_t bytes;
  };
  static size_t round(size_t b) { return ((b ? b : 1) + 255) & ~(size_t)255; }
  std::vector<Item> items_;
};

// Page-locked host memory from a process-wide cache of blocks in power-of-two size
// classes: a block is page-locked once and reused, never handed back to the driver
// (cudaFreeHost synchronises the device, which would stall every other engine's stream).
void* host_pinned(size_t bytes);
void host_unpin(void* p);

// cudaFuncSetAttribute acts on the current device only; `done` records, one bit
// per device ordinal (mod 64), where the attribute was already set.
inline void func_attr_once(std::atomic<unsigned long long>& done, const void* func, cudaFuncAttribute attr,
                           int value) {
  int dev = 0;
  DMRG2_CUDA(cudaGetDevice(&dev));
  const unsigned long long bit = 1ull << (dev & 63);
  if (done.load(std::memory_order_acquire) & bit) return;
  DMRG2_CUDA(cudaFuncSetAttribute(func, attr, value));
  done.fetch_or(bit, std::memory_order_acq_rel);
}

inline void set_smem_attr_once(std::atomic<unsigned long long>& done, const void* func, int bytes) {
  func_attr_once(done, func, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

}  // namespace dmrg2
