// Which backward kernels take a call, and what they want of the workspace.
#include "host_common.h"

namespace jvpfa {

size_t bwd_sm100_split_workspace_bytes(const jvpfa_bwd_args& a) {
  const size_t rows = static_cast<size_t>(a.B) * a.H * a.N;
  return kStatusBytes + align_up(rows * sizeof(float4), 256) + (a.tq != nullptr ? 8 : 4) * rows * kSplitRowBytes;
}

size_t bwd_sm100_workspace_bytes(const jvpfa_bwd_args& a) {
  return kStatusBytes + static_cast<size_t>(a.B) * a.H * a.N * sizeof(float4);
}

// bf16: what every path takes. fp16: the split operands of the output products behind it.
size_t bwd_sm100_wide_workspace_bytes(const jvpfa_bwd_args& a) {
  const size_t stats = static_cast<size_t>(a.B) * a.H * a.N * sizeof(float4);
  return a.dtype == JVPFA_F16 ? kStatusBytes + align_up(stats, 256) + split_f16_bytes(a.tq != nullptr ? 6 : 3, a.B, a.H, a.N, a.D)
                              : kStatusBytes + stats;
}

int launch_bwd_sm100(const jvpfa_bwd_args& a, int* status, cudaStream_t stream, const LaunchMarks& marks) {
  const bool bf = a.dtype == JVPFA_BF16;
  if (a.D > 128) return launch_bwd_sm100_d256(a, status, stream, marks);
  if (a.D <= 64) return bf ? launch_bwd_sm100_d64_bf16(a, status, stream, marks) : launch_bwd_sm100_d64_fp16(a, status, stream, marks);
  return bf ? launch_bwd_sm100_d128_bf16(a, status, stream, marks) : launch_bwd_sm100_d128_fp16(a, status, stream, marks);
}

}  // namespace jvpfa
