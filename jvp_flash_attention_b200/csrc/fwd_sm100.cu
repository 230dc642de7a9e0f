// Which forward kernel takes a call, and what it wants of the workspace.
#include "host_common.h"

namespace jvpfa {

bool sm100_path_supported(int dtype, int D, int N) {
  // head dimensions other than 64 / 128 run on the next wider kernel with zero-filled columns
  return (dtype == JVPFA_BF16 || dtype == JVPFA_F16) && D >= 8 && D <= 128 && (D % 8) == 0 && N >= 1;
}

bool sm100_wide_path_supported(int dtype, int D, int N) {
  return (dtype == JVPFA_BF16 || dtype == JVPFA_F16) && D > 128 && D <= 256 && (D % 8) == 0 && N >= 1;
}

bool sm100_split_path_supported(int dtype, int D, int N) {
  return dtype == JVPFA_F32 && D >= 8 && D <= 64 && (D % 8) == 0 && N >= 1;
}

size_t fwd_sm100_split_workspace_bytes(const jvpfa_fwd_args& a) {
  const size_t rows = static_cast<size_t>(a.B) * a.H * a.N;
  return kStatusBytes + (a.tq != nullptr ? 6 : 3) * rows * kSplitRowBytes;
}

size_t fwd_sm100_wide_workspace_bytes(const jvpfa_fwd_args& a) {
  return kStatusBytes + (a.dtype == JVPFA_F16 ? split_f16_bytes(a.tq != nullptr ? 2 : 1, a.B, a.H, a.N, a.D) : 0);
}

int launch_fwd_sm100(const jvpfa_fwd_args& a, int* status, cudaStream_t stream) {
  if (a.D <= 64) return launch_fwd_sm100_d64(a, status, stream);
  return a.D <= 128 ? launch_fwd_sm100_d128(a, status, stream) : launch_fwd_sm100_d256(a, status, stream);
}

}  // namespace jvpfa
