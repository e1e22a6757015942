// Entry points on host arrays for internal pieces that no call of the public interface reaches at
// the values a test needs. Compiled by internal.py and linked against the engine's library.
#include "contract.cuh"
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
template <typename T>
void heff_nonzeros(int cL, int cR, int d, int Dl, int Dm, int Dr, const void* L, const void* R, const void* WL,
                   const void* WR, const void* theta, void* out, int* nnz) {
  const size_t b = sizeof(T), dd = (size_t)d * d, n = cL * dd * cR, Kin = Dl * dd, Kout = dd * Dr;
  std::vector<T> w;
  build_wwt((const T*)WL, (const T*)WR, Dl, Dm, Dr, d, w);
  *nnz = wwt_sparse_block(w, (int)Kin, (int)Kout);
  const size_t xs = (size_t)cL * cR * (Kin > Kout ? Kin : Kout);
  Dev dL(L, b * cL * Dl * cL), dR(R, b * cR * Dr * cR), dW(w.data(), b * w.size()), in(theta, b * n), o(nullptr, b * n),
      X(nullptr, b * xs), Y(nullptr, b * xs);
  heff_apply(dL.as<T>(), dR.as<T>(), dW.as<T>(), in.as<T>(), o.as<T>(), X.as<T>(), Y.as<T>(), cL, cR, d, Dl, Dr, nullptr,
             0, dW.as<T>() + Kin * Kout);
  o.to(out, b * n);
}
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

// H_eff with the MPO's nonzero form beside the dense one, as the engine calls it
int probe_heff_nonzeros(int cplx, int cL, int cR, int d, int Dl, int Dm, int Dr, const void* L, const void* R,
                        const void* WL, const void* WR, const void* theta, void* out, int* nnz) {
  return guarded([&] {
    if (cplx) heff_nonzeros<zc>(cL, cR, d, Dl, Dm, Dr, L, R, WL, WR, theta, out, nnz);
    else heff_nonzeros<double>(cL, cR, d, Dl, Dm, Dr, L, R, WL, WR, theta, out, nnz);
  });
}

}  // extern "C"
