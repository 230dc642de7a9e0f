// Dual (JVP) attention forward for sm_100a: O = softmax(s QK^T + mask) V and its tangent tO in one
// pass, with tcgen05 MMAs accumulating in TMEM and K/tK/V/tV tiles staged by TMA.
//
// Replaces the reference's _attn_fwd_tma / _attn_fwd_inner_tma (jvp_flash_attention/jvp_attention.py:
// 1100-1392, 350-559). Per (128-row query tile, batch*head) one CTA of 12 warps:
//   warps 0-7  two softmax warpgroups that split the 64 columns of every score tile: thread r of a
//              warpgroup owns score row r (TMEM lane r) and 32 columns; keeps m, l, mu in registers, turns the
//              score tile S and tangent-score tile tS into 16-bit P and W = P o (s tS) written back to TMEM;
//              the two halves of a row exchange their maxima (and, at the end, their sums) through shared memory
//   warp 8     TMA producer of Q, tQ and the stacked [K; tK] pairs (one lane)
//   warp 11    TMA producer of the V, tV tiles (one lane)
//   warp 9     issues the score products (lane 0); owns the TMEM allocation
//   warp 10    issues the output products (lane 0). tcgen05.mma issue blocks once three to four instructions are
//              queued, so one issuing thread idles the tensor pipe during each of its barrier waits and commits;
//              two instruction streams keep it fed.
// Per 64-column key tile: [S | Q tK^T] = Q [K; tK]^T as one N = 128 product against the stacked pair, then
// tS += tQ K^T (operands in shared memory), then O += P V, T += W V + P tV (P, W read from TMEM; V, tV as
// MN-major shared-memory operands). Epilogue: O/l, tO = T/l - (mu/l) O/l, lse2 = m + log2 l, mu/l.
// TMEM columns: O [0,D), T [D,2D), one score buffer (S 64 | tS 64), then two buffers of 16-bit (P 32 | W 32). The score
// buffer is released as soon as every softmax thread holds its part of S, tS in registers, so that the next tile's
// score products are queued behind the running output products instead of waiting for them to complete.
#pragma once
#include <type_traits>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include "host_common.h"
#include "dropout.cuh"
#include "mask_common.cuh"
#include "sm100_prims.cuh"

namespace jvpfa {
using namespace sm100;

namespace {


struct FwdKParams {
  int H, N;
  int n_qt, n_units;   // query tiles per (batch, head) unit, number of units: the grid has n_qt * n_units blocks
  int unit_group;      // units per group of the block order
  int D;       // head dimension of the tensors (the kernel is compiled for it rounded up to 64, 128 or 256)
  int causal;
  float c1;      // sm_scale * log2(e)
  float s;       // sm_scale
  float thresh;  // lazy-rescale threshold in the log2 domain
  int b0;        // D = 256: first batch of this launch (fp16: where the tensor maps of the split V, tV begin)
  MaskView mv;
  void* o;
  void* to;
  float* lse2;
  float* mu;
  int* status;
  uint64_t budget_ns;
  DropoutParams drop;
};

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <bool BF16>
__device__ __forceinline__ uint32_t pack2(float a, float b) {
  if constexpr (BF16) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
  } else {
    __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
  }
}

__device__ __forceinline__ uint32_t pack2_residual(float a, float b, uint32_t hi) {
  return pack2<true>(a - __uint_as_float(hi << 16), b - __uint_as_float(hi & 0xFFFF0000u));
}

// SPLIT: fp32 inputs on the tensor cores. A pre-pass splits every fp32 operand x into two bf16 numbers hi + lo (x - hi - lo
// is below 2^-18 |x|) and writes them side by side as one 128-column row [hi(64) | lo(64)], so the tiles have the
// shared-memory geometry of the D = 128 kernel with the hi part in slab 0 and the lo part in slab 1; every product a b is
// then accumulated in fp32 as a_hi b_hi + a_lo b_hi + a_hi b_lo (what is left out is of the order 2^-18 |a||b|; an fp16 lo
// part would carry three more bits, but one product cannot take an fp16 operand against a bf16 one). The accumulators are 64
// columns wide, P and W = P o (s tS) go back to TMEM as hi and lo parts, and the outputs are written as fp32.
template <int D, bool SPLIT = false>
struct FwdCfg {
  static constexpr int BM = 128;
  static constexpr int BN = 64;
  static constexpr bool WIDE = D > 128;           // half of the output columns per CTA, see the kernel
  static constexpr bool HILO = SPLIT || WIDE;     // P and W as bf16 hi and lo parts
  static constexpr int STAGES = (D == 64) ? 4 : 2;                // slots of V, tV tiles (WIDE: of one tile of either)
  static constexpr int KSB = WIDE ? 1 : D / 64;   // 64-column slabs of [K; tK] per barrier
  static constexpr int KST = WIDE ? D / 64 : STAGES;              // ring slots of KSB slabs
  static constexpr int DV = SPLIT ? 64 : (WIDE ? D / 2 : D);      // columns of the O and T accumulators
  static constexpr int TILE_Q = BM * D * 2;
  static constexpr int TILE_V = BN * (WIDE ? DV : D) * 2;
  static constexpr int SLOT_V = WIDE ? TILE_V : 2 * TILE_V;
  static constexpr int SLAB = 128 * 128;          // bytes of one 64-column slab of a 128-row tile
  static constexpr int SLOT_K = KSB * SLAB;       // K and tK stacked as one 128-row operand
  static constexpr int HALF = BN * 128;           // byte offset of tK inside a slab of the pair
  static constexpr int TMEM_O = 0;
  static constexpr int TMEM_T = DV;
  static constexpr int TMEM_S = 2 * DV;       // S 64 columns, tS 64 columns further (one buffer)
  static constexpr int TMEM_P = 2 * DV + 128; // 16-bit P (32 columns) and W (32 columns further), buffer b at + PBUF b;
  static constexpr int PBUF = HILO ? 128 : 64;   // HILO: P hi, P lo, W hi, W lo, 32 columns each
  static constexpr int PBUFS = WIDE ? 1 : 2;
  static constexpr int TMEM_COLS = 512;
  static constexpr int NBAR = 4 + 2 * KST + 2 * STAGES + 4 + 2;
  static constexpr size_t smem_bytes() {
    return 2 * TILE_Q + KST * SLOT_K + STAGES * SLOT_V + 2 * 2 * 128 * 4 + (NBAR + 2) * 8;
  }
};

// Warps 0-7: two softmax warpgroups that split the 64 columns of every score tile (thread = TMEM lane =
// one score row, 32 columns; the row maximum and the final row sums are exchanged through shared
// memory); warps 8, 11: TMA producers (one lane each: Q and K pairs / V tiles); warps 9, 10: MMA issuers (one lane each: scores / outputs), warp 9 owns the
// TMEM allocation.
// D = 256 (head dimensions 136 to 256): O and T alone would fill TMEM, so two CTAs share a query tile, each with half of
// the output columns (V, tV columns) and all of the score products: 9 tile products where one CTA would run 6. Q, tQ take
// 128 KB of shared memory; K, tK go through four 16 KB slots by 64-column slab, V, tV through two of one tile.
// P and W keep 16 bits of significand and the range of fp32: they go to TMEM as bf16 hi and lo parts (one buffer, where the
// narrower kernels have two of 16-bit numbers). bf16 inputs: P V = P_hi V + P_lo V. fp16 inputs: a product cannot take an fp16
// operand against a bf16 one, so V, tV come split into bf16 hi and lo (exact, a pre-pass writes them to the workspace) and P V =
// P_hi V_hi + P_lo V_hi + P_hi V_lo. With P and W rounded to the inputs' 16 bits the outputs' errors were 1.24 to 1.5 times those
// of the fp32 CUDA-core kernels.
// B=2 H=8 N=1024 D=256 causal, us: bf16 72, fp16 108 with its pre-pass (16-bit P and W: 76, 77; CUDA cores, fp16: 3314); B=4 H=8
// N=2048: 330, 482 (292, 285). Errors against 64 bits over those of the CUDA cores (D = 136, 192, 256, N = 64 to 1024): bf16 1.000,
// fp16 1.000 to 1.001; 1.010 at N = 4096 (the tensor cores' fp32 accumulation).
// PAD: the tensors' head dimension is smaller than D (columns beyond it are zero-filled by TMA); the K steps and
// output columns that would only see zeros are then skipped at run time.
// DROP: dropout on the attention probabilities (dropout.cuh): P and W reach TMEM dropped out and rescaled, the row sums l
// and mu are those of the probabilities before dropout.
template <int D, bool DUAL, bool BF16, bool PAD, bool SPLIT = false, bool DROP = false>
__global__ void __launch_bounds__(384, 1)
fwd_sm100_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmTQ,
                 const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmTK,
                 const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmTV,
                 const FwdKParams p) {
  using C = FwdCfg<D, SPLIT>;
  constexpr int ST = C::STAGES, KST = C::KST;
  constexpr int SLABS = D / 64;
  constexpr int DV = C::DV;
  constexpr int VSLABS = DV / 64;                     // WIDE: slabs of a V tile,
  constexpr int VD = DUAL ? 2 : 1, VT = BF16 ? VD : 2 * VD;   // tiles of V, tV (fp16: their hi parts, then the lo parts) per key tile
  static_assert(!SPLIT || (D == 128 && BF16 && !PAD), "the split-fp32 mode runs on the 128-column geometry in bf16");

  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sQ = smem;
  uint8_t* sTQ = sQ + C::TILE_Q;
  auto sK = [&](int slot) { return smem + 2 * C::TILE_Q + slot * C::SLOT_K; };   // slabs of the [K; tK] pair
  auto sV = [&](int st) { return smem + 2 * C::TILE_Q + KST * C::SLOT_K + st * C::SLOT_V; };
  auto sTV = [&](int st) { return sV(st) + C::TILE_V; };
  uint8_t* tail = smem + 2 * C::TILE_Q + KST * C::SLOT_K + ST * C::SLOT_V;
  float(*xch)[2][128] = reinterpret_cast<float(*)[2][128]>(tail);          // [parity][warpgroup][row]
  uint64_t* bars = reinterpret_cast<uint64_t*>(tail + 2 * 2 * 128 * 4);
  uint64_t& q_full = bars[0];
  uint64_t& o_done = bars[1];
  uint64_t& o_final = bars[2];
  uint64_t& s_full = bars[4];        // S, tS of the current tile are complete
  uint64_t& s_free = bars[5];        // all 256 softmax threads have S, tS in registers: the next tile's products may overwrite them
  uint64_t* p_full = bars + 6;       // [2]
  uint64_t* k_full = bars + 8;
  uint64_t* v_full = k_full + KST;
  uint64_t* k_empty = v_full + ST;
  uint64_t* v_empty = k_empty + KST;
  uint64_t* p_free = v_empty + ST;   // [2]: the PV products that read P, W buffer b have completed
  uint32_t& tmem_base_s = *reinterpret_cast<uint32_t*>(bars + C::NBAR);
  int& poisoned = *reinterpret_cast<int*>(bars + C::NBAR + 1);
  if ((smem_u32(smem) & 1023u) != 0u) {  // the swizzled layouts need this; never observed otherwise
    if (threadIdx.x == 0) atomicCAS(p.status, 0, WAIT_TIMEOUT_BASE + 99);
    return;
  }

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // heavy query tiles first; the two column halves of a tile are neighbours (they read the same K, tK)
  const BlockWork work = block_work(C::WIDE ? blockIdx.x >> 1 : blockIdx.x, p.n_qt, p.n_units, p.unit_group, p.causal != 0);
  const int half = C::WIDE ? blockIdx.x & 1 : 0;
  const int dcols = C::WIDE ? (((p.D + 1) / 2 + 15) & ~15) : p.D;         // output columns of this CTA: [dcol0, dcol0 + dcols)
  const int dcol0 = half * dcols;
  const int n_slabs = C::WIDE && PAD ? (p.D + 63) / 64 : SLABS;           // slabs of K, tK that hold data
  const int qt = work.tile;
  const int bh = C::WIDE ? work.unit + p.b0 * p.H : work.unit;
  const int b = bh / p.H, h = bh % p.H;
  const int q0 = qt * C::BM;
  const int N = p.N;
  const int row_base = bh * N;
  int n_kt = (N + C::BN - 1) / C::BN;
  if (p.causal) n_kt = min(n_kt, (q0 + C::BM - 1) / C::BN + 1);

  const WaitCtx w{p.status, &poisoned, p.budget_ns};

  if (tid == 0) {
    poisoned = 0;
    mbar_init(&q_full, 1);
    for (int i = 0; i < KST; ++i) {
      mbar_init(&k_full[i], 1);
      mbar_init(&k_empty[i], 1);
    }
    for (int i = 0; i < ST; ++i) {
      mbar_init(&v_full[i], 1);
      mbar_init(&v_empty[i], 1);
    }
    mbar_init(&s_full, 1);
    mbar_init(&s_free, 256);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&p_full[i], 256);
      mbar_init(&p_free[i], 1);
    }
    mbar_init(&o_done, 1);
    mbar_init(&o_final, 1);
    fence_mbar_init();
  }
  __syncthreads();
  if (warp == 9) {
    tmem_alloc(&tmem_base_s, C::TMEM_COLS);
    tmem_relinquish();
  }
  // the TMA producers need the barriers but not the TMEM address: they start loading while TMEM is being allocated
  const bool producer = (warp == 8 || warp == 11);
  tc_fence_before_sync();
  if (!producer) named_bar_sync(2, 320);
  tc_fence_after_sync();
  const uint32_t tmem = producer ? 0u : tmem_base_s;

  // Key tile j takes part unless the mask summary says that nothing in it is kept.
  auto tile_bits = [&](int j) -> uint8_t {
    if (p.mv.kind == JVPFA_MASK_NONE) return kTileAnyKept;
    uint8_t bits = mask_tile_bits(p.mv, b, h, 2 * qt, j);
    if (2 * qt + 1 < p.mv.n64) bits |= mask_tile_bits(p.mv, b, h, 2 * qt + 1, j);
    return bits;
  };

  if (warp == 11) {
    // ------------------------------------------------------------------ TMA producer of the V, tV tiles (a warp of
    // its own: V slots free up a tile later than K slots, one producer waiting for them would hold the K loads back)
    if (lane == 0) {
      int it = 0;
      for (int j = 0; j < n_kt; ++j) {
        if (!(tile_bits(j) & kTileAnyKept)) continue;
        const int krow = j * C::BN;   // first key row of the tile inside its (batch, head) unit
        if constexpr (C::WIDE) {      // V, tV, and with fp16 inputs their lo parts: a slot each
#pragma unroll
          for (int n = 0; n < VT; ++n, ++it) {
            const int st = it % ST, x = (n / VD) * p.D + dcol0;
            const CUtensorMap* tm = DUAL && n % VD == 1 ? &tmTV : &tmV;
            mbar_wait(&v_empty[st], ((it / ST) & 1) ^ 1, w, 11);
            mbar_arrive_expect_tx(&v_full[st], C::TILE_V);
#pragma unroll
            for (int sl = 0; sl < VSLABS; ++sl)
              tma_load_tile(sV(st) + sl * C::HALF, tm, &v_full[st], x + 64 * sl, krow, h, BF16 ? b : b - p.b0);
          }
          continue;
        }
        const int st = it % ST;
        const uint32_t ph = (it / ST) & 1;
        mbar_wait(&v_empty[st], ph ^ 1, w, 11);
        mbar_arrive_expect_tx(&v_full[st], (DUAL ? 2 : 1) * C::TILE_V);
        if constexpr (!PAD && SLABS > 1) {
          // the slabs of a V tile are consecutive in shared memory: one box per tensor through the 3-D map
          tma_load_slabs(sV(st), &tmV, &v_full[st], krow, h, b);
          if constexpr (DUAL) tma_load_slabs(sTV(st), &tmTV, &v_full[st], krow, h, b);
        } else {
#pragma unroll
          for (int sl = 0; sl < SLABS; ++sl) {
            tma_load_tile(sV(st) + sl * C::HALF, &tmV, &v_full[st], 64 * sl, krow, h, b);
            if constexpr (DUAL) tma_load_tile(sTV(st) + sl * C::HALF, &tmTV, &v_full[st], 64 * sl, krow, h, b);
          }
        }
        ++it;
      }
    }
    __syncwarp();
  } else if (warp == 8) {
    // ------------------------------------------------------------------ TMA producer of Q, tQ and the [K; tK] pairs
    if (lane == 0) {
      tma_prefetch_desc(&tmQ);
      tma_prefetch_desc(&tmK);
      tma_prefetch_desc(&tmV);
      mbar_arrive_expect_tx(&q_full, (DUAL ? 2 : 1) * C::TILE_Q);
#pragma unroll
      for (int sl = 0; sl < SLABS; ++sl) {
        tma_load_tile(sQ + sl * C::SLAB, &tmQ, &q_full, 64 * sl, q0, h, b);
        if constexpr (DUAL) tma_load_tile(sTQ + sl * C::SLAB, &tmTQ, &q_full, 64 * sl, q0, h, b);
      }
      int it = 0;
      for (int j = 0; j < n_kt; ++j) {
        if (!(tile_bits(j) & kTileAnyKept)) continue;
        const int krow = j * C::BN;   // first key row of the tile inside its (batch, head) unit
#pragma unroll
        for (int g = 0; g < (C::WIDE ? n_slabs : SLABS / C::KSB); ++g) {
          const int slot = C::WIDE ? g : it % KST;
          const uint32_t ph = (C::WIDE ? it : it / KST) & 1;
          mbar_wait(&k_empty[slot], ph ^ 1, w, 10);
          mbar_arrive_expect_tx(&k_full[slot], (DUAL ? 2 : 1) * C::KSB * C::HALF);
#pragma unroll
          for (int sl = 0; sl < C::KSB; ++sl) {
            const int x = 64 * (g * C::KSB + sl);
            tma_load_tile(sK(slot) + sl * C::SLAB, &tmK, &k_full[slot], x, krow, h, b);
            if constexpr (DUAL) tma_load_tile(sK(slot) + sl * C::SLAB + C::HALF, &tmTK, &k_full[slot], x, krow, h, b);
          }
        }
        ++it;
      }
    }
    __syncwarp();
  } else if (warp >= 9) {
    // ------------------------------------------------------------------ MMA issuers: warp 9 scores, warp 10 outputs
    // all lanes run the loops (waits included) so that the warp stays converged; the elected lane issues
    const bool leader = elect_one_sync();
    auto wait_all = [&](uint64_t* bar, uint32_t parity, int site) {
      mbar_wait(bar, parity, w, site);
      __syncwarp();
    };
    {
    constexpr uint32_t FMT = BF16 ? FMT_BF16 : FMT_F16;
    const uint32_t idesc_64 = make_idesc(FMT, 128, 64, 0, 0);
    const uint32_t idesc_128 = make_idesc(FMT, 128, 128, 0, 0);
    const int dn = SPLIT ? 64 : (C::WIDE ? dcols : (PAD ? ((p.D + 15) & ~15) : D));   // columns of the output products (rounded up to the MMA granularity)
    const int ksteps = C::WIDE ? (p.D + 15) / 16 : dn / 16;   // K steps of the score products that hold data
    const uint32_t idesc_pv = make_idesc(C::HILO ? FMT_BF16 : FMT, 128, dn, 0, 1);
    const uint64_t dQ = desc_kmajor_sw128(smem_u32(sQ)), dTQ = desc_kmajor_sw128(smem_u32(sTQ));

    auto issue_qk = [&](int it) {
      const uint32_t S_t = tmem + C::TMEM_S;
      if constexpr (C::WIDE) {
        // slab by slab: a slot of the ring is free again as soon as its slab has been multiplied
        if (it >= 1) wait_all(&s_free, (it - 1) & 1, 24);
        for (int g = 0; g < n_slabs; ++g) {
          wait_all(&k_full[g], it & 1, 20);
          tc_fence_after_sync();
          const uint64_t dK = desc_kmajor_sw128(smem_u32(sK(g))), slab = static_cast<uint64_t>((g * C::SLAB) >> 4);
          if (leader) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const uint64_t o = static_cast<uint64_t>((k * 32) >> 4);
              if (!PAD || 4 * g + k < ksteps) umma_ss(S_t, dQ + slab + o, dK + o, DUAL ? idesc_128 : idesc_64, g > 0 || k > 0);   // [S | Q tK^T]
            }
            if constexpr (DUAL) {
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                const uint64_t o = static_cast<uint64_t>((k * 32) >> 4);
                if (!PAD || 4 * g + k < ksteps) umma_ss(S_t + 64, dTQ + slab + o, dK + o, idesc_64, 1);                             // tS += tQ K^T
              }
            }
            if (g == n_slabs - 1) umma_commit(&s_full);
            umma_commit(&k_empty[g]);
          }
        }
        return;
      }
      const int st = it % ST;
      const uint32_t ph = (it / ST) & 1;
      wait_all(&k_full[st], ph, 20);
      if (it >= 1) wait_all(&s_free, (it - 1) & 1, 24);
      tc_fence_after_sync();
      const uint64_t dK = desc_kmajor_sw128(smem_u32(sK(st)));
      if (leader) {
        if constexpr (SPLIT) {
          // hi hi + lo hi + hi lo: K steps 0-3 of the left (a) and right (b) operand's slab 0 (hi) or slab 1 (lo)
#pragma unroll
          for (int k = 0; k < 12; ++k) {
            const int a_slab = (k >> 2) == 1, b_slab = (k >> 2) == 2;
            const uint64_t oa = static_cast<uint64_t>((a_slab * C::SLAB + (k & 3) * 32) >> 4);
            const uint64_t ob = static_cast<uint64_t>((b_slab * C::SLAB + (k & 3) * 32) >> 4);
            umma_ss(S_t, dQ + oa, dK + ob, DUAL ? idesc_128 : idesc_64, k > 0);                        // [S | Q tK^T]
          }
          if constexpr (DUAL) {
#pragma unroll
            for (int k = 0; k < 12; ++k) {
              const int a_slab = (k >> 2) == 1, b_slab = (k >> 2) == 2;
              const uint64_t oa = static_cast<uint64_t>((a_slab * C::SLAB + (k & 3) * 32) >> 4);
              const uint64_t ob = static_cast<uint64_t>((b_slab * C::SLAB + (k & 3) * 32) >> 4);
              umma_ss(S_t + 64, dTQ + oa, dK + ob, idesc_64, 1);                                        // tS += tQ K^T
            }
          }
        } else {
#pragma unroll
          for (int k = 0; k < D / 16; ++k) {
            const uint64_t o = static_cast<uint64_t>(((k >> 2) * C::SLAB + (k & 3) * 32) >> 4);
            if (!PAD || k < ksteps) umma_ss(S_t, dQ + o, dK + o, DUAL ? idesc_128 : idesc_64, k > 0);   // [S | Q tK^T]
          }
          if constexpr (DUAL) {
#pragma unroll
            for (int k = 0; k < D / 16; ++k) {
              const uint64_t o = static_cast<uint64_t>(((k >> 2) * C::SLAB + (k & 3) * 32) >> 4);
              if (!PAD || k < ksteps) umma_ss(S_t + 64, dTQ + o, dK + o, idesc_64, 1);                    // tS += tQ K^T
            }
          }
        }
        umma_commit(&s_full);
        umma_commit(&k_empty[st]);
      }
    };
    auto issue_pv = [&](int it, bool last) {
      const int st = it % ST;
      const uint32_t ph = (it / ST) & 1;
      const uint32_t P_t = tmem + C::TMEM_P + (it % C::PBUFS) * C::PBUF;
      const uint32_t W_t = P_t + (C::HILO ? 64 : 32);
      wait_all(&p_full[it % C::PBUFS], (it / C::PBUFS) & 1, 21);
      if constexpr (C::WIDE) {
#pragma unroll
        for (int n = 0; n < VT; ++n) {
          const int c = it * VT + n, slot = c % ST;
          wait_all(&v_full[slot], (c / ST) & 1, 22);
          tc_fence_after_sync();
          if (leader) {
            const uint64_t dV = desc_mnmajor_sw128(smem_u32(sV(slot)), C::BN * 128);
            const bool lo = n >= VD;       // the lo part of V, tV: multiplies the hi parts of P, W only
            // acc += e_hi c (+ e_lo c)
            auto mul = [&](uint32_t accum, uint32_t e, uint64_t d, uint32_t first_acc) {
              umma_ts(accum, e, d, idesc_pv, first_acc);
              if (!lo) umma_ts(accum, e + 32, d, idesc_pv, 1);
            };
#pragma unroll
            for (int k = 0; k < C::BN / 16; ++k) {
              const uint64_t d = dV + static_cast<uint64_t>((k * 2048) >> 4);
              const uint32_t acc = it > 0 || n > 0 || k > 0;
              if (n % VD == 0) {
                mul(tmem + C::TMEM_O, P_t + 8 * k, d, acc);
                if constexpr (DUAL) mul(tmem + C::TMEM_T, W_t + 8 * k, d, acc);
              } else {
                mul(tmem + C::TMEM_T, P_t + 8 * k, d, 1);
              }
            }
            umma_commit(&v_empty[slot]);
            if (n == VT - 1) {
              umma_commit(&p_free[0]);
              umma_commit(&o_done);
              if (last) umma_commit(&o_final);
            }
          }
        }
        return;
      }
      wait_all(&v_full[st], ph, 22);
      tc_fence_after_sync();
      const uint64_t dV0 = desc_mnmajor_sw128(smem_u32(sV(st)), C::BN * 128);
      const uint64_t dTV0 = desc_mnmajor_sw128(smem_u32(sTV(st)), C::BN * 128);
      const uint32_t acc0 = it > 0;
      if (leader) {
#pragma unroll
        for (int k = 0; k < C::BN / 16; ++k) {
          const uint64_t ok = static_cast<uint64_t>((k * 2048) >> 4);
          const uint32_t eo = k * 8;
          if constexpr (SPLIT) {
            // the lo part of an operand in TMEM sits 32 columns after its hi part, the lo slab of V, tV one slab further
            const uint64_t lo = static_cast<uint64_t>(C::HALF >> 4);
            // acc += e_hi c_hi + e_lo c_hi + e_hi c_lo
            auto three = [&](uint32_t accum, uint32_t e, uint64_t c, uint32_t first_acc) {
              umma_ts(accum, e, c, idesc_pv, first_acc);
              umma_ts(accum, e + 32, c, idesc_pv, 1);
              umma_ts(accum, e, c + lo, idesc_pv, 1);
            };
            three(tmem + C::TMEM_O, P_t + eo, dV0 + ok, acc0 | (k > 0));
            if constexpr (DUAL) {
              three(tmem + C::TMEM_T, W_t + eo, dV0 + ok, acc0 | (k > 0));
              three(tmem + C::TMEM_T, P_t + eo, dTV0 + ok, 1);
            }
          } else {
            umma_ts(tmem + C::TMEM_O, P_t + eo, dV0 + ok, idesc_pv, acc0 | (k > 0));
            if constexpr (DUAL) {
              umma_ts(tmem + C::TMEM_T, W_t + eo, dV0 + ok, idesc_pv, acc0 | (k > 0));
              umma_ts(tmem + C::TMEM_T, P_t + eo, dTV0 + ok, idesc_pv, 1);
            }
          }
        }
        umma_commit(&v_empty[st]);
        umma_commit(&p_free[it & 1]);
        umma_commit(&o_done);
        if (last) umma_commit(&o_final);
      }
    };

    int it = 0;
    if (warp == 9) {
      wait_all(&q_full, 0, 23);
      for (int j = 0; j < n_kt; ++j) {
        if (!(tile_bits(j) & kTileAnyKept)) continue;
        issue_qk(it);
        ++it;
      }
    } else {
      for (int j = 0; j < n_kt; ++j) {
        if (!(tile_bits(j) & kTileAnyKept)) continue;
        if (it > 0) issue_pv(it - 1, false);
        ++it;
      }
      if (it > 0) issue_pv(it - 1, true);
    }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ softmax, correction, epilogue
    const int wg = warp >> 2;
    const int r = (warp & 3) * 32 + lane;
    const int qi = q0 + r;
    const int qi_c = min(qi, N - 1);
    const uint32_t lane_off = static_cast<uint32_t>((warp & 3) * 32) << 16;
    float m_used = -INFINITY;
    float2 l2 = make_float2(0.f, 0.f), mu2 = make_float2(0.f, 0.f);   // partial row sums over this thread's columns
    const float2 c1_2 = make_float2(p.c1, p.c1), s_2 = make_float2(p.s, p.s);
    int it = 0;
    for (int j = 0; j < n_kt; ++j) {
      const uint8_t bits = tile_bits(j);
      if (!(bits & kTileAnyKept)) continue;
      const uint32_t S_t = tmem + C::TMEM_S + lane_off + 32 * wg;
      const uint32_t tS_t = S_t + 64;
      const uint32_t P_t = tmem + C::TMEM_P + (it % C::PBUFS) * C::PBUF + lane_off + 16 * wg;   // this thread's 16 columns of P
      const uint32_t W_t = P_t + (C::HILO ? 64 : 32);
      mbar_wait(&s_full, it & 1, w, 30);
      tc_fence_after_sync();
      // scores of this thread's 32 columns in the log2 domain, two per register pair (packed fp32x2
      // arithmetic: the softmax warps share their schedulers with the MMA-issuing warp)
      float2 x2[16];
      uint32_t ts[32];
      {
        uint32_t r0[32];
        tmem_ld_x32(S_t, r0);
        if constexpr (DUAL) tmem_ld_x32(tS_t, ts);
        tmem_wait_ld();
        // S and tS are in registers: the next tile's score products may overwrite them
        tc_fence_before_sync();
        mbar_arrive(&s_free);
#pragma unroll
        for (int i = 0; i < 16; ++i)
          x2[i] = __fmul2_rn(make_float2(__uint_as_float(r0[2 * i]), __uint_as_float(r0[2 * i + 1])), c1_2);
      }
      const int k0 = j * C::BN + 32 * wg;   // first key of this thread's columns
      const bool need_causal = p.causal && j * C::BN + C::BN - 1 > q0;
      const bool need_bound = j * C::BN + C::BN > N;
      const bool need_mask = p.mv.kind != JVPFA_MASK_NONE && (bits & kTileAnyMasked);
      // The mask as this thread sees it: the flags of its own 64x64 tile (the two 64-row halves of the query tile may
      // differ). Packed by the summary pre-pass (a boolean mask, or a two-valued tile of an additive one), this row's 32
      // entries of the tile are one word; anything else is read element by element below.
      int mask_mode = 0;
      if (need_mask) mask_mode = mask_tile_mode(p.mv, mask_tile_bits(p.mv, b, h, qi_c >> 6, j));
      if (mask_mode == 1) {
        const float other = p.mv.kind == JVPFA_MASK_BOOL ? -INFINITY : mask_tile_value(p.mv, b, h, qi_c >> 6, j) * 1.4426950408889634f;
        mask_apply_bits(x2, mask_row_bits(p.mv, b, h, qi_c, j, wg), other);
      }
      const bool mask_elems = mask_mode == 2;
      // (keys past the end of the sequence: zero bits of a boolean mask already exclude them)
      if (need_causal || (need_bound && !(mask_mode == 1 && p.mv.kind == JVPFA_MASK_BOOL)) || mask_elems) {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          float bias[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) bias[i] = 0.f;
          if (mask_elems) mask_bias_run<16>(bias, p.mv, b, h, qi_c, k0 + 16 * c, N, true);
          if (need_causal) {
#pragma unroll
            for (int i = 0; i < 16; ++i)
              if (k0 + 16 * c + i > qi) bias[i] = -INFINITY;
          }
          if (need_bound) {
#pragma unroll
            for (int i = 0; i < 16; ++i)
              if (k0 + 16 * c + i >= N) bias[i] = -INFINITY;
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) x2[8 * c + i] = __fadd2_rn(x2[8 * c + i], make_float2(bias[2 * i], bias[2 * i + 1]));
        }
      }
      float m_tile = fmaxf(x2[0].x, x2[0].y);
#pragma unroll
      for (int i = 1; i < 16; ++i) m_tile = fmaxf(m_tile, fmaxf(x2[i].x, x2[i].y));
      // row maximum over both warpgroups: the two warps that share these 32 rows meet on a barrier of their own
      xch[it & 1][wg][r] = m_tile;
      named_bar_sync(3 + (warp & 3), 64);
      m_tile = fmaxf(m_tile, xch[it & 1][wg ^ 1][r]);
      const float m_new = fmaxf(m_used, m_tile);
      const bool need = m_new > m_used + p.thresh;
      if (__any_sync(0xFFFFFFFFu, need)) {   // same rows, same values in both warpgroups: same decision
        const float alpha = (m_used == -INFINITY) ? 1.0f : fast_exp2(m_used - m_new);
        if (it > 0) {
          mbar_wait(&o_done, (it - 1) & 1, w, 31);
          tc_fence_after_sync();
          // warpgroup 0 rescales O, warpgroup 1 rescales T
          if (DUAL || wg == 0) {
            const uint32_t base = tmem + lane_off + (wg == 0 ? C::TMEM_O : C::TMEM_T);
#pragma unroll
            for (int c = 0; c < DV / 32; ++c) {
              uint32_t a[32];
              tmem_ld_x32(base + c * 32, a);
              tmem_wait_ld();
#pragma unroll
              for (int i = 0; i < 32; ++i) a[i] = __float_as_uint(__uint_as_float(a[i]) * alpha);
              tmem_st_x32(base + c * 32, a);
            }
          }
        }
        l2.x *= alpha; l2.y *= alpha;
        mu2.x *= alpha; mu2.y *= alpha;
        m_used = m_new;
      }
      const float m_eff = (m_used == -INFINITY) ? 0.f : m_used;
      const float2 nm2 = make_float2(-m_eff, -m_eff);
      uint32_t keep_bits = 0xFFFFFFFFu;
      if constexpr (DROP) keep_bits = dropout_keep_along_k(p.drop, bh, qi, k0);
      {
        // the PV products of tile it - PBUFS read this P, W buffer
        if (it >= C::PBUFS) {
          mbar_wait(&p_free[it % C::PBUFS], (it / C::PBUFS - 1) & 1, w, 33);
          tc_fence_after_sync();
        }
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t pk[8], wk[8], pkl[8], wkl[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int ip = 8 * c + i;
            const float2 e = __fadd2_rn(x2[ip], nm2);
            const float2 pp = make_float2(fast_exp2(e.x), fast_exp2(e.y));
            l2 = __fadd2_rn(l2, pp);
            float2 keep2 = make_float2(1.f, 1.f);
            if constexpr (DROP) keep2 = dropout_factors(keep_bits, ip, p.drop.inv_keep);
            const float2 pd = DROP ? __fmul2_rn(pp, keep2) : pp;     // what multiplies V, tV
            pk[i] = pack2<BF16 || C::HILO>(pd.x, pd.y);
            if constexpr (C::HILO) pkl[i] = pack2_residual(pd.x, pd.y, pk[i]);
            if constexpr (DUAL) {
              const float2 tsv = __fmul2_rn(make_float2(__uint_as_float(ts[2 * ip]), __uint_as_float(ts[2 * ip + 1])), s_2);
              const float2 ww = __fmul2_rn(pp, tsv);
              mu2 = __fadd2_rn(mu2, ww);
              const float2 wd = DROP ? __fmul2_rn(ww, keep2) : ww;
              wk[i] = pack2<BF16 || C::HILO>(wd.x, wd.y);
              if constexpr (C::HILO) wkl[i] = pack2_residual(wd.x, wd.y, wk[i]);
            }
          }
          tmem_st_x8(P_t + 8 * c, pk);
          if constexpr (C::HILO) tmem_st_x8(P_t + 32 + 8 * c, pkl);
          if constexpr (DUAL) {
            tmem_st_x8(W_t + 8 * c, wk);
            if constexpr (C::HILO) tmem_st_x8(W_t + 32 + 8 * c, wkl);
          }
        }
      }
      tmem_wait_st();
      tc_fence_before_sync();
      mbar_arrive(&p_full[it % C::PBUFS]);
      ++it;
    }
    // epilogue: total row sums over both warpgroups, then each warpgroup writes half of the head dimension.
    // o_done flips once per key tile and a parity wait is only meaningful within one phase of the
    // barrier, so the end of the last accumulation has a barrier of its own.
    float l = l2.x + l2.y, mu = mu2.x + mu2.y;
    named_bar_sync(3 + (warp & 3), 64);
    xch[0][wg][r] = l;
    xch[1][wg][r] = mu;
    named_bar_sync(3 + (warp & 3), 64);
    l += xch[0][wg ^ 1][r];
    mu += xch[1][wg ^ 1][r];
    if (it > 0) {
      mbar_wait(&o_final, 0, w, 32);
      tc_fence_after_sync();
    }
    const float linv = (l > 0.f) ? 1.0f / l : 0.f;
    const float mul = mu * linv;
    // Each warpgroup writes half of the head dimension; the rows go through this warp's patch of shared memory (the Q
    // tile is no longer needed: every product that reads it has completed) so that the global stores are row segments.
    if (it == 0) mbar_wait(&q_full, 0, w, 34);   // nothing was multiplied: the Q load itself may still be in flight
    if constexpr (SPLIT) {
      // fp32 outputs: this warpgroup's 32 columns are 128 bytes per row
      uint8_t* patch = sQ + warp * (32 * 128);
      uint32_t po[2][16], pt[2][16];
      {
        uint32_t ov[32], tv[32];
        if (it > 0) {
          tmem_ld_x32(tmem + lane_off + C::TMEM_O + wg * 32, ov);
          if constexpr (DUAL) tmem_ld_x32(tmem + lane_off + C::TMEM_T + wg * 32, tv);
          tmem_wait_ld();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) { ov[i] = 0u; tv[i] = 0u; }
        }
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const float o = __uint_as_float(ov[i]) * linv;
          po[i >> 4][i & 15] = __float_as_uint(o);
          if constexpr (DUAL) pt[i >> 4][i & 15] = __float_as_uint(__uint_as_float(tv[i]) * linv - mul * o);
        }
      }
      const int col0 = wg * 32;
      const int wrow0 = q0 + (warp & 3) * 32;
      const size_t goff = (static_cast<size_t>(row_base) + wrow0) * p.D + col0;      // in fp32 elements
      const int rows = N - wrow0, cols16 = 2 * (p.D - col0);                          // columns in 16-bit units
      store_rows_via_smem<2>(patch, po, reinterpret_cast<uint16_t*>(static_cast<float*>(p.o) + goff), 2 * static_cast<size_t>(p.D),
                             rows, cols16, lane);
      if constexpr (DUAL)
        store_rows_via_smem<2>(patch, pt, reinterpret_cast<uint16_t*>(static_cast<float*>(p.to) + goff),
                               2 * static_cast<size_t>(p.D), rows, cols16, lane);
    } else {
      constexpr int CH = DV / 64;
      uint8_t* patch = sQ + warp * (32 * CH * 64);
      uint32_t po[CH][16], pt[CH][16];
#pragma unroll
      for (int cc = 0; cc < CH; ++cc) {
        const int c = wg * CH + cc;
        uint32_t ov[32], tv[32];
        if (it > 0) {
          tmem_ld_x32(tmem + lane_off + C::TMEM_O + c * 32, ov);
          if constexpr (DUAL) tmem_ld_x32(tmem + lane_off + C::TMEM_T + c * 32, tv);
          tmem_wait_ld();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) { ov[i] = 0u; tv[i] = 0u; }
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float o0 = __uint_as_float(ov[2 * i]) * linv, o1 = __uint_as_float(ov[2 * i + 1]) * linv;
          po[cc][i] = pack2<BF16>(o0, o1);
          if constexpr (DUAL) {
            const float t0 = __uint_as_float(tv[2 * i]) * linv - mul * o0;
            const float t1 = __uint_as_float(tv[2 * i + 1]) * linv - mul * o1;
            pt[cc][i] = pack2<BF16>(t0, t1);
          }
        }
      }
      const int col0 = dcol0 + wg * (DV / 2);                          // first column of this warpgroup
      const int wrow0 = q0 + (warp & 3) * 32;                          // first row of this warp
      const size_t goff = (static_cast<size_t>(row_base) + wrow0) * p.D + col0;
      const int rows = N - wrow0, cols = min(dcol0 + dcols, p.D) - col0;
      store_rows_via_smem<CH>(patch, po, static_cast<uint16_t*>(p.o) + goff, p.D, rows, cols, lane);
      if constexpr (DUAL) store_rows_via_smem<CH>(patch, pt, static_cast<uint16_t*>(p.to) + goff, p.D, rows, cols, lane);
    }
    if (qi < N && wg == 0 && half == 0) {
      p.lse2[static_cast<size_t>(row_base) + qi] = (l > 0.f) ? m_used + log2f(l) : -INFINITY;
      p.mu[static_cast<size_t>(row_base) + qi] = mul;
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 9) tmem_dealloc(tmem, C::TMEM_COLS);
}

template <bool BF16>
FwdKParams make_fwd_params(const jvpfa_fwd_args& a, int* status) {
  FwdKParams p{};
  p.H = a.H; p.N = a.N; p.D = a.D; p.causal = a.causal;
  p.s = a.sm_scale;
  p.c1 = a.sm_scale * 1.4426950408889634f;
  p.thresh = BF16 ? 8.0f : 6.0f;
  p.mv = make_mask_view(a.mask, a.mask_summary, a.B, a.H, a.N);
  p.o = a.o; p.to = a.to; p.lse2 = a.lse2; p.mu = a.mu;
  p.status = status;
  p.budget_ns = wait_budget_ns();
  p.drop = make_dropout_params(a.dropout_p, a.dropout_seed);
  p.n_qt = (a.N + 127) / 128;
  p.n_units = a.B * a.H;
  p.unit_group = unit_group_size(p.n_units);
  return p;
}

template <int D, bool DUAL, bool BF16, bool PAD, bool DROP = false>
int launch_one(const jvpfa_fwd_args& a, int* status, cudaStream_t stream) {
  using C = FwdCfg<D>;
  CUtensorMap mQ, mTQ, mK, mTK, mV, mTV;
  auto tile = [&](CUtensorMap* m, const void* ptr, const jvpfa_strides& st, int box_rows) {
    return make_tile_map(m, make_view(ptr, st, a.H, a.N, a.D), a.B, a.H, a.N, a.D, box_rows, a.dtype);
  };
  auto vmap = [&](CUtensorMap* m, const void* ptr, const jvpfa_strides& st) {
    return (!PAD && D == 128) ? make_slab_map(m, make_view(ptr, st, a.H, a.N, a.D), a.B, a.H, a.N, a.D, C::BN, a.dtype)
                            : tile(m, ptr, st, C::BN);
  };
  constexpr bool SPLIT_V = C::WIDE && !BF16;   // V, tV are read as bf16 hi and lo parts
  bool ok = tile(&mQ, a.q, a.q_strides, C::BM) && tile(&mK, a.k, a.k_strides, C::BN) && (SPLIT_V || vmap(&mV, a.v, a.v_strides));
  if (DUAL) {
    ok = ok && tile(&mTQ, a.tq, a.tq_strides, C::BM) && tile(&mTK, a.tk, a.tk_strides, C::BN) && (SPLIT_V || vmap(&mTV, a.tv, a.tv_strides));
  } else {
    mTQ = mQ; mTK = mK; mTV = mV;
  }
  if (!ok) return JVPFA_ERR_LAUNCH;
  FwdKParams p = make_fwd_params<BF16>(a, status);
  auto kern = fwd_sm100_kernel<D, DUAL, BF16, PAD, false, DROP>;
  const size_t smem = C::smem_bytes();
  static SmemOptIn opt_in;
  if (!opt_in.set(reinterpret_cast<const void*>(kern), smem)) return JVPFA_ERR_LAUNCH;
  if constexpr (SPLIT_V) {
    // a launch per group of batches whose split tensors fit the workspace
    const void* src[2] = {a.v, a.tv};
    const jvpfa_strides* st[2] = {&a.v_strides, &a.tv_strides};
    uint16_t* dst[2];
    const int n_t = DUAL ? 2 : 1, step = split_f16_batches(n_t, a.B, a.H, a.N, a.D);
    for (int i = 0; i < n_t; ++i)
      dst[i] = reinterpret_cast<uint16_t*>(static_cast<uint8_t*>(a.workspace) + kStatusBytes) + i * split_f16_elems(step, a.H, a.N, a.D);
    for (int b0 = 0; b0 < a.B; b0 += step) {
      const int nb = a.B - b0 < step ? a.B - b0 : step;
      TensorView views[2];
      for (int i = 0; i < n_t; ++i) views[i] = batches_from(make_view(src[i], *st[i], a.H, a.N, a.D), b0, 2);
      const int rc = launch_split_f16(views, dst, n_t, nb, a.H, a.N, a.D, stream);
      if (rc != JVPFA_OK) return rc;
      if (!make_split_f16_map(&mV, dst[0], nb, a.H, a.N, a.D, C::BN) || !make_split_f16_map(&mTV, dst[n_t - 1], nb, a.H, a.N, a.D, C::BN))
        return JVPFA_ERR_LAUNCH;
      p.b0 = b0;
      p.n_units = nb * a.H;
      p.unit_group = unit_group_size(p.n_units);
      kern<<<static_cast<unsigned>(p.n_qt) * static_cast<unsigned>(p.n_units) * 2u, 384, smem, stream>>>(mQ, mTQ, mK, mTK, mV, mTV, p);
      if (cudaGetLastError() != cudaSuccess) return JVPFA_ERR_LAUNCH;
    }
    return JVPFA_OK;
  }
  dim3 grid(static_cast<unsigned>(p.n_qt) * static_cast<unsigned>(p.n_units) * (C::WIDE ? 2u : 1u));
  kern<<<grid, 384, smem, stream>>>(mQ, mTQ, mK, mTK, mV, mTV, p);
  return cudaGetLastError() == cudaSuccess ? JVPFA_OK : JVPFA_ERR_LAUNCH;
}

// fp32 inputs: split pre-pass into the workspace, then the 128-column kernel in its split mode on the split tensors.
template <bool DUAL, bool DROP>
int launch_split(const jvpfa_fwd_args& a, int* status, cudaStream_t stream) {
  using C = FwdCfg<128, true>;
  const int64_t rows = static_cast<int64_t>(a.B) * a.H * a.N;
  const int n_t = DUAL ? 6 : 3;
  const void* src[6] = {a.q, a.k, a.v, a.tq, a.tk, a.tv};
  uint16_t* dst[6];
  uint8_t* base = static_cast<uint8_t*>(a.workspace) + kStatusBytes;
  for (int i = 0; i < n_t; ++i) dst[i] = reinterpret_cast<uint16_t*>(base + static_cast<size_t>(i) * rows * kSplitRowBytes);
  const jvpfa_strides* sst[6] = {&a.q_strides, &a.k_strides, &a.v_strides, &a.tq_strides, &a.tk_strides, &a.tv_strides};
  TensorView views[6];
  for (int i = 0; i < n_t; ++i) views[i] = make_view(src[i], *sst[i], a.H, a.N, a.D);
  int rc = launch_split_fp32(views, dst, n_t, a.B, a.H, a.N, a.D, stream);
  if (rc != JVPFA_OK) return rc;
  CUtensorMap mQ, mTQ, mK, mTK, mV, mTV;
  const jvpfa_strides none{0, 0, 0};
  auto tile = [&](CUtensorMap* m, const void* ptr, int box_rows) {
    return make_tile_map(m, make_view(ptr, none, a.H, a.N, 128), a.B, a.H, a.N, 128, box_rows, JVPFA_BF16);
  };
  auto slab = [&](CUtensorMap* m, const void* ptr) {
    return make_slab_map(m, make_view(ptr, none, a.H, a.N, 128), a.B, a.H, a.N, 128, C::BN, JVPFA_BF16);
  };
  bool ok = tile(&mQ, dst[0], C::BM) && tile(&mK, dst[1], C::BN) && slab(&mV, dst[2]);
  if (DUAL) {
    ok = ok && tile(&mTQ, dst[3], C::BM) && tile(&mTK, dst[4], C::BN) && slab(&mTV, dst[5]);
  } else {
    mTQ = mQ; mTK = mK; mTV = mV;
  }
  if (!ok) return JVPFA_ERR_LAUNCH;
  const FwdKParams p = make_fwd_params<true>(a, status);
  auto kern = fwd_sm100_kernel<128, DUAL, true, false, true, DROP>;
  const size_t smem = C::smem_bytes();
  static SmemOptIn opt_in;
  if (!opt_in.set(reinterpret_cast<const void*>(kern), smem)) return JVPFA_ERR_LAUNCH;
  dim3 grid(static_cast<unsigned>(p.n_qt) * static_cast<unsigned>(p.n_units));
  kern<<<grid, 384, smem, stream>>>(mQ, mTQ, mK, mTK, mV, mTV, p);
  return cudaGetLastError() == cudaSuccess ? JVPFA_OK : JVPFA_ERR_LAUNCH;
}

template <int D, bool PAD>
int launch_by_mode(const jvpfa_fwd_args& a, int* status, cudaStream_t stream) {
  const bool dual = a.tq != nullptr;
  const bool bf = a.dtype == JVPFA_BF16;
  if constexpr (D <= 128) if (a.dropout_p > 0.f) {
    if (dual) return bf ? launch_one<D, true, true, PAD, true>(a, status, stream) : launch_one<D, true, false, PAD, true>(a, status, stream);
    return bf ? launch_one<D, false, true, PAD, true>(a, status, stream) : launch_one<D, false, false, PAD, true>(a, status, stream);
  }
  if (dual) return bf ? launch_one<D, true, true, PAD>(a, status, stream) : launch_one<D, true, false, PAD>(a, status, stream);
  return bf ? launch_one<D, false, true, PAD>(a, status, stream) : launch_one<D, false, false, PAD>(a, status, stream);
}
}  // namespace
}  // namespace jvpfa
