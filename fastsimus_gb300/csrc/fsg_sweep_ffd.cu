// Instantiations of the pfield kernel with full-frequency directivity
// (full_frequency_directivity=True): each Green's term is weighted by sinc(k_f seg/2 sin(theta))
// at every frequency, as in the step body
// _pfield_strategies.py:44-45 (driven from :77-81).  Kept in a translation unit of their own so that they compile
// in parallel with the default kernels of fsg_sweep.cu.

#include "fsg_sweep_kernels.cuh"

namespace fsg {

cudaError_t launch_pfield_band_ffd(const SweepConfig& c, const BandArgs& A, cudaStream_t s) {
  return A.C.ffd == kSincShort ? launch_pfield_band_gn<kSincShort>(c, A, s) : launch_pfield_band_gn<kSincTerms>(c, A, s);
}

}  // namespace fsg
