// Forward kernels of the 128-column geometry (head dimensions 72 to 128).
#include "fwd_sm100.cuh"

namespace jvpfa {

int launch_fwd_sm100_d128(const jvpfa_fwd_args& a, int* status, cudaStream_t stream) {
  return a.D == 128 ? launch_by_mode<128, false>(a, status, stream) : launch_by_mode<128, true>(a, status, stream);
}

}  // namespace jvpfa
