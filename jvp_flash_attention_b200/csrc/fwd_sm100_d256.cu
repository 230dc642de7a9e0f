// Forward kernels of the 256-column geometry (head dimensions 136 to 256).
#include "fwd_sm100.cuh"

namespace jvpfa {

int launch_fwd_sm100_d256(const jvpfa_fwd_args& a, int* status, cudaStream_t stream) {
  return a.D == 256 ? launch_by_mode<256, false>(a, status, stream) : launch_by_mode<256, true>(a, status, stream);
}

}  // namespace jvpfa
