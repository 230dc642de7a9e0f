// Forward kernels for head dimensions 8 to 64, 16-bit inputs.
#include "fwd_sm100_d64.cuh"

namespace jvpfa {

// Two CTAs per SM (fwd_sm100_d64.cuh) pay when there is a second CTA for the SMs: from more than one block per SM on. A CTA
// of that kernel alone on its SM has half the element-wise warps of the other kernel and takes longer per tile; under a causal
// mask the blocks differ in length, and up to 1.5 blocks per SM the longest ones alone decide.
// Forward, bf16, D = 64, one CTA per SM -> two, us: 160 blocks (H 10, N 2048) 68.2 -> 54.0, causal 37.2 -> 39.6; 192 blocks
// 69.6 -> 55.8, causal 38.6 -> 45.2; 224 blocks 70.5 -> 56.5, causal 53.2 -> 52.3; 288 blocks 70.8 -> 56.6, causal 62.5 -> 53.7;
// 1024 blocks (B 4, H 16) 236.7 -> 204.4, causal 157.8 -> 132.8; B 32, H 16, N 256 64.5 -> 47.4. At 128 blocks (B 2, H 8, N 1024,
// boolean mask) 29.2 -> 38.8.
constexpr int64_t kSms = 148;

int launch_fwd_sm100_d64(const jvpfa_fwd_args& a, int* status, cudaStream_t stream) {
  const int64_t blocks = static_cast<int64_t>(a.B) * a.H * ((a.N + 127) / 128);
  if (a.causal ? 2 * blocks >= 3 * kSms : blocks > kSms)
    return a.D == 64 ? launch_fwd64_by_mode<false>(a, status, stream) : launch_fwd64_by_mode<true>(a, status, stream);
  return a.D == 64 ? launch_by_mode<64, false>(a, status, stream) : launch_by_mode<64, true>(a, status, stream);
}

}  // namespace jvpfa
