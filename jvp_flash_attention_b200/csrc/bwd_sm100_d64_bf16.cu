// Backward kernels of the 64-column geometry, bf16.
#include "bwd_sm100.cuh"

namespace jvpfa {

int launch_bwd_sm100_d64_bf16(const jvpfa_bwd_args& a, int* status, cudaStream_t stream, const LaunchMarks& marks) {
  return launch_all<64, true>(a, status, stream, marks);
}

}  // namespace jvpfa
