// simus_lane_kernel instantiations with full-frequency directivity.
#include "fsg_sweep_lane.cuh"

namespace fsg {

cudaError_t launch_simus_lane_ffd(int U, const SweepConfig& c, const BandArgs& A, cudaStream_t s) {
  return launch_lane_any<true>(U, c, A, s);
}

}  // namespace fsg
