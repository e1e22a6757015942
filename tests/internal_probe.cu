// Entry points on host arrays for internal pieces that no call of the public interface reaches at
// the values a test needs. Compiled by internal.py and linked against the engine's library.
#include "kernels.cuh"

using namespace dmrg2;

namespace {
struct Dev {  // a device copy of host data
  void* p = nullptr;
  Dev(const void* h, size_t b) {
    DMRG2_CUDA(cudaMalloc(&p, b));
    DMRG2_CUDA(h ? cudaMemcpy(p, h, b, cudaMemcpyHostToDevice) : cudaMemset(p, 0, b));
  }
  ~Dev() { cudaFree(p); }
  template <typename T>
  T* as() const { return (T*)p; }
  void to(void* h, size_t b) const { DMRG2_CUDA(cudaMemcpy(h, p, b, cudaMemcpyDeviceToHost)); }
};
template <typename F>
int guarded(F f) {
  try {
    f();
    return 0;
  } catch (...) {
    return 1;
  }
}
}  // namespace

extern "C" {

// the polish's decision on S = Z^T Z (K x K, leading k x k block): flags = {ns_done, ns_near}
int probe_ns_check(const double* S, int K, int k, double tol, int* flags) {
  return guarded([&] {
    Dev s(S, sizeof(double) * K * K), part(nullptr, sizeof(double) * 64), counter(nullptr, sizeof(unsigned) * 4),
        status(nullptr, sizeof(int)), out(nullptr, sizeof(SvdOut));
    split_begin(status.as<int>(), out.as<SvdOut>(), k, 0);
    ns_check(s.as<double>(), K, out.as<SvdOut>(), tol, part.as<double>(), counter.as<unsigned>(), 0);
    SvdOut o;
    out.to(&o, sizeof(o));
    flags[0] = o.ns_done;
    flags[1] = o.ns_near;
  });
}

// the n-th deferred Lanczos solve from now fails
void probe_fail_solve(int n) { lz_fail_countdown() = n; }

}  // extern "C"
