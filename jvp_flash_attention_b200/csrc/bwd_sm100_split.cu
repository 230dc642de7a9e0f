// Backward kernels of the split-fp32 mode.
#include "bwd_sm100.cuh"

namespace jvpfa {

int launch_bwd_sm100_split(const jvpfa_bwd_args& a, int* status, cudaStream_t stream, const LaunchMarks& marks) {
  if (a.dropout_p > 0.f)
    return a.tq != nullptr ? launch_split<true, true>(a, status, stream, marks) : launch_split<false, true>(a, status, stream, marks);
  return a.tq != nullptr ? launch_split<true, false>(a, status, stream, marks) : launch_split<false, false>(a, status, stream, marks);
}

}  // namespace jvpfa
