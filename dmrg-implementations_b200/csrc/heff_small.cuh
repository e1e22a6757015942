// H_eff in one launch for small bonds (heff_small.cu).
#pragma once

#include "common.cuh"

namespace dmrg2 {

constexpr int HS_TARGET_CTAS = 352;
// Measured against the three tiled contractions (us per matvec in a CUDA graph, d = 2, both forms
// behind the same MPO kernel; cL = cR):
//   D = 5: 4: 10.1 / 11.8, 16: 11.6 / 13.2, 32: 12.9 / 14.7, 64: 16.0 / 16.7, 80: 26.2 / 17.3
//   D = 8: 8: 10.8 / 15.6, 32: 13.7 / 16.6, 64: 17.5 / 18.7, 96: 38.8 / 23.7
// so the line lies at the work of D = 8, 64 x 64.
constexpr double HS_MAX_FLOP = 3.4e7;

// where the one-launch form is the faster one (see heff_small.cu)
template <typename T>
inline bool heff_small_fits(int cL, int cR, int dd, int Dl, int Dr) {
  const double f = 2.0 * dd * cL * (double)cR * (Dl * (double)cL + Dr * (double)cR) * (ST<T>::cplx ? 4.0 : 1.0);
  return f <= HS_MAX_FLOP;
}

// out = H_eff in, with dd the physical dimension of the block (d^2 of a two-site bond, d of one
// site) and WWt the (dd Dr) x (Dl dd) mixing matrix; false, with nothing launched, where the
// shape is not one for this kernel, or out overlaps in or Lenv
template <typename T>
bool heff_small(const T* Lenv, const T* Renv, const T* WWt, const T* in, T* out, int cL, int cR, int dd, int Dl, int Dr,
                const int* skip, cudaStream_t s);

}  // namespace dmrg2
