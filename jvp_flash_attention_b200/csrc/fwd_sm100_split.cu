// Forward kernels of the split-fp32 mode.
#include "fwd_sm100.cuh"

namespace jvpfa {

int launch_fwd_sm100_split(const jvpfa_fwd_args& a, int* status, cudaStream_t stream) {
  if (a.dropout_p > 0.f) return a.tq != nullptr ? launch_split<true, true>(a, status, stream) : launch_split<false, true>(a, status, stream);
  return a.tq != nullptr ? launch_split<true, false>(a, status, stream) : launch_split<false, false>(a, status, stream);
}

}  // namespace jvpfa
