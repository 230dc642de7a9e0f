// Backward kernels of the 64-column geometry, fp16.
#include "bwd_sm100.cuh"

namespace jvpfa {

int launch_bwd_sm100_d64_fp16(const jvpfa_bwd_args& a, int* status, cudaStream_t stream, const LaunchMarks& marks) {
  return launch_all<64, false>(a, status, stream, marks);
}

}  // namespace jvpfa
