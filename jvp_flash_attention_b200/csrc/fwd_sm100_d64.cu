// Forward kernels of the 64-column geometry (head dimensions 8 to 64).
#include "fwd_sm100.cuh"

namespace jvpfa {

int launch_fwd_sm100_d64(const jvpfa_fwd_args& a, int* status, cudaStream_t stream) {
  return a.D == 64 ? launch_by_mode<64, false>(a, status, stream) : launch_by_mode<64, true>(a, status, stream);
}

}  // namespace jvpfa
