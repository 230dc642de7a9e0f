// Forward kernels for head dimensions 8 to 64, 16-bit inputs.
#include "fwd_sm100_d64.cuh"

namespace jvpfa {

int launch_fwd_sm100_d64(const jvpfa_fwd_args& a, int* status, cudaStream_t stream) {
  return a.D == 64 ? launch_fwd64_by_mode<false>(a, status, stream) : launch_fwd64_by_mode<true>(a, status, stream);
}

}  // namespace jvpfa
