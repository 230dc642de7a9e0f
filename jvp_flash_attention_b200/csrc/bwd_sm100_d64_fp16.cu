// Backward kernels for head dimensions 8 to 64, fp16.
#include "bwd_sm100_d64.cuh"

namespace jvpfa {

int launch_bwd_sm100_d64_fp16(const jvpfa_bwd_args& a, int* status, cudaStream_t stream, const LaunchMarks& marks) {
  return launch_bwd64_by_mode<false>(a, status, stream, marks);
}

}  // namespace jvpfa
