// simus_lane_kernel instantiations with full-frequency directivity.
#include "fsg_sweep_lane.cuh"

namespace fsg {

cudaError_t launch_simus_lane_ffd(int U, const SweepConfig& c, const BandArgs& A, cudaStream_t s) {
  return A.C.ffd == kSincShort ? launch_lane_any<kSincShort>(U, c, A, s) : launch_lane_any<kSincTerms>(U, c, A, s);
}

}  // namespace fsg
