// Dual (JVP) attention forward for head dimensions up to 64, 16-bit inputs: two CTAs per SM.
//
// At these widths the products of a 128 x 64 tile take 832 cycles of the tensor pipe, the exponentials 512 of the
// special-function unit, and the chain from the score products over maximum, exponentials and packing back to the output
// products is longer than either. One CTA per SM whose eight element-wise warps walk that chain in step (the structure of
// fwd_sm100.cuh) needed 1888 cycles a tile: every unit idles while the others work. Here a CTA is half as large --
// 256 TMEM columns, 96 KB of shared memory, four element-wise warps whose threads own a whole score row -- so that two of
// them share an SM out of step: one CTA's products run beside the other's element-wise work, and its start-up and
// epilogue (10 k cycles, six tile periods) beside the other's tiles.
//   warps 0-3  thread = TMEM lane = one score row, all 64 columns: no exchange between warps
//   warp 4     TMA producer (one lane): Q, tQ, then per key tile K, tK and V, tV
//   warp 5     MMA issuer (one lane): S(0), tS(0), then per tile S(i + 1), outputs(i), tS(i + 1)
// TMEM: O 64 | T 64 | S 64 | tS 64. The 16-bit P and W of 16 keys take the place of those keys' 16 columns of tS, so S is free
// as soon as it has been read: the next S is ready before the element-wise warps ask for it, and only tS(i + 1) waits for
// outputs(i) (behind them in the pipe, issued by the same thread), which the next tile's maximum and first exponentials
// cover. That costs the stacked N = 128 product [S | Q tK^T] (S and tS are three N = 64 products, 960 cycles a tile with the
// outputs) and takes the products off the chain.
#pragma once
#include "fwd_sm100.cuh"

namespace jvpfa {
namespace {

struct Fwd64Cfg {
  static constexpr int STAGES = 2;
  static constexpr int TILE_Q = 128 * 128;        // 128 rows of 64 16-bit columns
  static constexpr int HALF = 64 * 128;           // a 64-row tile
  static constexpr int STAGE = 4 * HALF;          // K, tK, V, tV
  static constexpr int NBAR = 8 + 4 * STAGES;
  static constexpr size_t smem_bytes() { return 2 * TILE_Q + STAGES * STAGE + (NBAR + 2) * 8; }
};

// PAD, DUAL, DROP as in fwd_sm100_kernel.
template <bool DUAL, bool BF16, bool PAD, bool DROP>
__global__ void __launch_bounds__(192, 2)
fwd64_sm100_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmTQ,
                   const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmTK,
                   const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmTV, const FwdKParams p) {
  using C = Fwd64Cfg;
  constexpr int ST = C::STAGES;
  // TMEM columns. Primal only: O, S and a buffer of P; P, W of 16 keys are 8 + 8 columns (primal only: 8)
  constexpr uint32_t COLS = 256;
  constexpr uint32_t T_T = 64, T_S = DUAL ? 128 : 64, T_TS = 192, T_P = DUAL ? T_TS : 128, PSTEP = DUAL ? 16 : 8;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t *sQ = smem, *sTQ = smem + C::TILE_Q;
  auto sK = [&](int st) { return smem + 2 * C::TILE_Q + st * C::STAGE; };
  auto sV = [&](int st) { return sK(st) + 2 * C::HALF; };
  auto sTV = [&](int st) { return sK(st) + 3 * C::HALF; };
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 2 * C::TILE_Q + ST * C::STAGE);
  uint64_t &q_full = bars[0], &s_full = bars[1], &ts_full = bars[2], &o_final = bars[3];
  uint64_t* p_full = bars + 4;   // [2] P, W of the tile's first / second 32 keys are in TMEM
  uint64_t &s_free = bars[6], &o_done = bars[7];
  uint64_t *k_full = bars + 8, *k_empty = k_full + ST, *v_full = k_empty + ST, *v_empty = v_full + ST;
  uint32_t& tmem_base_s = *reinterpret_cast<uint32_t*>(bars + C::NBAR);
  int& poisoned = *reinterpret_cast<int*>(bars + C::NBAR + 1);
  if ((smem_u32(smem) & 1023u) != 0u) {  // the swizzled layouts need this; never observed otherwise
    if (threadIdx.x == 0) atomicCAS(p.status, 0, WAIT_TIMEOUT_BASE + 99);
    return;
  }
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const BlockWork work = block_work(blockIdx.x, p.n_qt, p.n_units, p.unit_group, p.causal != 0);   // heavy query tiles first
  const int qt = work.tile, bh = work.unit;
  const int b = bh / p.H, h = bh % p.H;
  const int q0 = qt * 128, N = p.N;
  int n_kt = (N + 63) / 64;
  if (p.causal) n_kt = min(n_kt, (q0 + 127) / 64 + 1);
  const WaitCtx w{p.status, &poisoned, p.budget_ns};
  if (tid == 0) {
    poisoned = 0;
    for (int i = 0; i < C::NBAR; ++i) mbar_init(&bars[i], i >= 4 && i <= 6 ? 4 : 1);
    fence_mbar_init();
  }
  __syncthreads();
  if (warp == 5) {
    tmem_alloc(&tmem_base_s, COLS);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  if (warp != 4) named_bar_sync(2, 160);   // the TMA producer starts loading while TMEM is being allocated
  tc_fence_after_sync();
  const uint32_t tmem = warp == 4 ? 0u : tmem_base_s;

  // Key tile j takes part unless the mask summary says that nothing in it is kept.
  auto tile_bits = [&](int j) -> uint8_t {
    if (p.mv.kind == JVPFA_MASK_NONE) return kTileAnyKept;
    uint8_t bits = mask_tile_bits(p.mv, b, h, 2 * qt, j);
    if (2 * qt + 1 < p.mv.n64) bits |= mask_tile_bits(p.mv, b, h, 2 * qt + 1, j);
    return bits;
  };
  auto next_active = [&](int j) {
    while (j < n_kt && !(tile_bits(j) & kTileAnyKept)) ++j;
    return j;
  };

  if (warp == 4) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      mbar_arrive_expect_tx(&q_full, (DUAL ? 2 : 1) * C::TILE_Q);
      tma_load_tile(sQ, &tmQ, &q_full, 0, q0, h, b);
      if constexpr (DUAL) tma_load_tile(sTQ, &tmTQ, &q_full, 0, q0, h, b);
      int it = 0;
      for (int j = next_active(0); j < n_kt; j = next_active(j + 1), ++it) {
        const int st = it % ST, krow = j * 64;
        const uint32_t ph = (it / ST) & 1;
        mbar_wait(&k_empty[st], ph ^ 1, w, 10);
        mbar_arrive_expect_tx(&k_full[st], (DUAL ? 2 : 1) * C::HALF);
        tma_load_tile(sK(st), &tmK, &k_full[st], 0, krow, h, b);
        if constexpr (DUAL) tma_load_tile(sK(st) + C::HALF, &tmTK, &k_full[st], 0, krow, h, b);
        mbar_wait(&v_empty[st], ph ^ 1, w, 11);
        mbar_arrive_expect_tx(&v_full[st], (DUAL ? 2 : 1) * C::HALF);
        tma_load_tile(sV(st), &tmV, &v_full[st], 0, krow, h, b);
        if constexpr (DUAL) tma_load_tile(sTV(st), &tmTV, &v_full[st], 0, krow, h, b);
      }
    }
    __syncwarp();
  } else if (warp == 5) {
    // ------------------------------------------------------------------ MMA issuer: all lanes walk the loop (waits included)
    // so that the warp stays converged, the elected lane issues
    const bool leader = elect_one_sync();
    auto wait_all = [&](uint64_t* bar, uint32_t parity, int site) {
      mbar_wait(bar, parity, w, site);
      __syncwarp();
    };
    constexpr uint32_t FMT = BF16 ? FMT_BF16 : FMT_F16;
    const int dn = PAD ? ((p.D + 15) & ~15) : 64;      // columns of the output products, 16 per K step of the score products
    const int ksteps = dn / 16;
    const uint32_t idesc_s = make_idesc(FMT, 128, 64, 0, 0), idesc_pv = make_idesc(FMT, 128, dn, 0, 1);
    const uint64_t dQ = desc_kmajor_sw128(smem_u32(sQ)), dTQ = desc_kmajor_sw128(smem_u32(sTQ));
    auto nt = [&](uint32_t dst, uint64_t da, uint64_t db, bool first) {
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (!PAD || k < ksteps) umma_ss(dst, da + 2 * k, db + 2 * k, idesc_s, !(first && k == 0));
    };
    auto scores = [&](int it) {          // S = Q K^T
      wait_all(&k_full[it % ST], (it / ST) & 1, 20);
      tc_fence_after_sync();
      if (leader) {
        nt(tmem + T_S, dQ, desc_kmajor_sw128(smem_u32(sK(it % ST))), true);
        umma_commit(&s_full);
        if constexpr (!DUAL) umma_commit(&k_empty[it % ST]);
      }
    };
    auto tangent_scores = [&](int it) {  // tS = Q tK^T + tQ K^T
      if constexpr (DUAL) {
        if (leader) {
          const uint64_t dK = desc_kmajor_sw128(smem_u32(sK(it % ST)));
          nt(tmem + T_TS, dQ, dK + (C::HALF >> 4), true);
          nt(tmem + T_TS, dTQ, dK, false);
          umma_commit(&ts_full);
          umma_commit(&k_empty[it % ST]);
        }
      }
    };
    wait_all(&q_full, 0, 23);
    int it = 0;
    int j = next_active(0);
    if (j < n_kt) {
      scores(0);
      tangent_scores(0);
    }
    for (; j < n_kt; ++it) {
      j = next_active(j + 1);
      const int st = it % ST;
      if (j < n_kt) {
        wait_all(&s_free, it & 1, 24);
        scores(it + 1);
      }
      wait_all(&v_full[st], (it / ST) & 1, 22);
      const uint64_t dV = desc_mnmajor_sw128(smem_u32(sV(st)), C::HALF), dTV = desc_mnmajor_sw128(smem_u32(sTV(st)), C::HALF);
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        wait_all(&p_full[g], it & 1, 21);
        tc_fence_after_sync();
        if (leader) {
#pragma unroll
        for (int k = 2 * g; k < 2 * g + 2; ++k) {
          const uint64_t ok = static_cast<uint64_t>((k * 2048) >> 4);
          const uint32_t P = tmem + T_P + PSTEP * k, W = P + 8;
          umma_ts(tmem, P, dV + ok, idesc_pv, it > 0 || k > 0);                  // O += P V
          if constexpr (DUAL) {
            umma_ts(tmem + T_T, W, dV + ok, idesc_pv, it > 0 || k > 0);          // T += W V
            umma_ts(tmem + T_T, P, dTV + ok, idesc_pv, 1);                       // T += P tV
          }
        }
        }
      }
      if (leader) {
        umma_commit(&v_empty[st]);
        umma_commit(&o_done);
        if (j >= n_kt) umma_commit(&o_final);
      }
      if (j < n_kt) tangent_scores(it + 1);
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ softmax, correction, epilogue
    const int qi = q0 + tid, qi_c = min(qi, N - 1);
    const uint32_t base = tmem + (static_cast<uint32_t>(warp * 32) << 16);
    float m_used = -INFINITY;
    float2 l2 = make_float2(0.f, 0.f), mu2 = make_float2(0.f, 0.f);
    const float2 c1_2 = make_float2(p.c1, p.c1), s_2 = make_float2(p.s, p.s);
    int it = 0;
    int j_next = next_active(0);
    MaskRow mask_next = mask_row_of(p.mv, b, h, qi_c, j_next, n_kt);
    for (int j = j_next; j < n_kt; j = j_next, ++it) {
      const MaskRow mask = mask_next;
      mbar_wait(&s_full, it & 1, w, 30);
      tc_fence_after_sync();
      // the row's scores in the log2 domain, two per register pair (packed fp32x2 arithmetic)
      float2 x2[2][16];
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        uint32_t s[32];
        tmem_ld_x32(base + T_S + 32 * g, s);
#pragma unroll
        for (int i = 0; i < 16; ++i) x2[g][i] = make_float2(__uint_as_float(s[2 * i]), __uint_as_float(s[2 * i + 1]));
      }
      tmem_wait_ld();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&s_free);      // S is in registers: the next one may overwrite it
      // what the mask says about the next tile is fetched now, a tile ahead of its use
      j_next = next_active(j + 1);
      mask_next = mask_row_of(p.mv, b, h, qi_c, j_next, n_kt);
      const int k0 = j * 64;
      const bool need_causal = p.causal && k0 + 63 > q0;
      const bool need_bound = k0 + 64 > N;
      // from here on: x2 times `c` is the score in the log2 domain
      float2 c_2 = c1_2;
      if (need_causal || need_bound || mask.mode != 0 || !(p.c1 > 0.f)) {
        c_2 = make_float2(1.f, 1.f);
#pragma unroll
        for (int g = 0; g < 2; ++g) {
#pragma unroll
          for (int i = 0; i < 16; ++i) x2[g][i] = __fmul2_rn(x2[g][i], c1_2);
          if (mask.mode == 1) mask_apply_bits(x2[g], mask.bits[g], mask.other);
        }
        if (mask.mode == 2) mask_add_row64(x2, p.mv, b, h, qi_c, k0, N);
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          // keys beyond the query (causal) or the end of the sequence
          const int last = (need_causal ? min(qi, N - 1) : N - 1) - (k0 + 32 * g);   // last key of this half that takes part
          if (last < 31) {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              if (2 * i > last) x2[g][i].x = -INFINITY;
              if (2 * i + 1 > last) x2[g][i].y = -INFINITY;
            }
          }
        }
      }
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};   // four chains instead of one of 64 comparisons
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        mx[0] = fmaxf(mx[0], x2[0][i].x); mx[1] = fmaxf(mx[1], x2[0][i].y);
        mx[2] = fmaxf(mx[2], x2[1][i].x); mx[3] = fmaxf(mx[3], x2[1][i].y);
      }
      const float m_new = fmaxf(m_used, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * c_2.x);
      if (__any_sync(0xFFFFFFFFu, m_new > m_used + p.thresh)) {
        const float alpha = (m_used == -INFINITY) ? 1.0f : fast_exp2(m_used - m_new);
        if (it > 0) {
          mbar_wait(&o_done, (it - 1) & 1, w, 33);
          tc_fence_after_sync();
#pragma unroll
          for (int c = 0; c < (DUAL ? 4 : 2); ++c) {
            uint32_t a[32];
            tmem_ld_x32(base + c * 32, a);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 32; ++i) a[i] = __float_as_uint(__uint_as_float(a[i]) * alpha);
            tmem_st_x32(base + c * 32, a);
          }
        }
        l2.x *= alpha; l2.y *= alpha;
        mu2.x *= alpha; mu2.y *= alpha;
        m_used = m_new;
      }
      const float m_eff = (m_used == -INFINITY) ? 0.f : m_used;
      const float2 nm2 = make_float2(-m_eff, -m_eff);
      // 16 keys at a time: the exponentials of chunk c + 1 are in the code before what chunk c does with its tangent scores,
      // so that the special-function unit and the FMA pipe work at the same time within the one warp a scheduler has here
      uint32_t keep_bits[2] = {0xFFFFFFFFu, 0xFFFFFFFFu};
      if constexpr (DROP) {
        keep_bits[0] = dropout_keep_along_k(p.drop, bh, qi, k0);
        keep_bits[1] = dropout_keep_along_k(p.drop, bh, qi, k0 + 32);
      }
      auto sum8 = [](const float2 (&v)[8]) {   // a tree: one link of the accumulator's chain per chunk instead of eight
        return __fadd2_rn(__fadd2_rn(__fadd2_rn(v[0], v[1]), __fadd2_rn(v[2], v[3])), __fadd2_rn(__fadd2_rn(v[4], v[5]), __fadd2_rn(v[6], v[7])));
      };
      auto exps = [&](int c) {
        float2 pp[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          float2& x = x2[c >> 1][8 * (c & 1) + i];
          const float2 e = __ffma2_rn(x, c_2, nm2);
          x = pp[i] = make_float2(fast_exp2(e.x), fast_exp2(e.y));
        }
        l2 = __fadd2_rn(l2, sum8(pp));
      };
      exps(0);
      exps(1);
      if constexpr (DUAL) {
        mbar_wait(&ts_full, it & 1, w, 31);
        tc_fence_after_sync();
      } else if (it > 0) {   // the outputs of the previous tile have read P
        mbar_wait(&o_done, (it - 1) & 1, w, 33);
        tc_fence_after_sync();
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t ts[16], pw[16];
        if constexpr (DUAL) tmem_ld_x16(base + T_TS + 16 * c, ts);
        if (c < 2) exps(c + 2);
        if constexpr (DUAL) tmem_wait_ld();
        float2 ww[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float2 pp = x2[c >> 1][8 * (c & 1) + i];
          float2 keep = make_float2(1.f, 1.f);
          if constexpr (DROP) keep = dropout_factors(keep_bits[c >> 1], 8 * (c & 1) + i, p.drop.inv_keep);
          const float2 pd = DROP ? __fmul2_rn(pp, keep) : pp;     // what multiplies V, tV
          pw[i] = pack2<BF16>(pd.x, pd.y);
          if constexpr (DUAL) {
            const float2 tsv = __fmul2_rn(make_float2(__uint_as_float(ts[2 * i]), __uint_as_float(ts[2 * i + 1])), s_2);
            ww[i] = __fmul2_rn(pp, tsv);
            const float2 wd = DROP ? __fmul2_rn(ww[i], keep) : ww[i];
            pw[8 + i] = pack2<BF16>(wd.x, wd.y);
          }
        }
        if constexpr (DUAL) {
          mu2 = __fadd2_rn(mu2, sum8(ww));
          tmem_st_x16(base + T_P + PSTEP * c, pw);
        } else {
          tmem_st_x8(base + T_P + PSTEP * c, reinterpret_cast<uint32_t(&)[8]>(pw));
        }
        if (c & 1) {   // P, W of 32 keys are complete
          tmem_wait_st();
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(&p_full[c >> 1]);
        }
      }
    }
    const float l = l2.x + l2.y, mu = mu2.x + mu2.y;
    if (it > 0) {
      mbar_wait(&o_final, 0, w, 32);
      tc_fence_after_sync();
    } else {
      mbar_wait(&q_full, 0, w, 34);   // nothing was multiplied: the Q load itself may still be in flight
    }
    const float linv = (l > 0.f) ? 1.0f / l : 0.f;
    const float mul = mu * linv;
    // the rows go through this warp's patch of shared memory (the Q tile is no longer needed) so that the global stores are
    // row segments
    uint32_t po[2][16], pt[2][16];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      uint32_t ov[32], tv[32];
      if (it > 0) {
        tmem_ld_x32(base + 32 * c, ov);
        if constexpr (DUAL) tmem_ld_x32(base + T_T + 32 * c, tv);
        tmem_wait_ld();
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) { ov[i] = 0u; tv[i] = 0u; }
      }
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float o0 = __uint_as_float(ov[2 * i]) * linv, o1 = __uint_as_float(ov[2 * i + 1]) * linv;
        po[c][i] = pack2<BF16>(o0, o1);
        if constexpr (DUAL)
          pt[c][i] = pack2<BF16>(__uint_as_float(tv[2 * i]) * linv - mul * o0, __uint_as_float(tv[2 * i + 1]) * linv - mul * o1);
      }
    }
    uint8_t* patch = sQ + warp * (32 * 128);
    const int wrow0 = q0 + warp * 32, rows = N - wrow0;
    const size_t goff = (static_cast<size_t>(bh) * N + wrow0) * p.D;
    store_rows_via_smem<2>(patch, po, static_cast<uint16_t*>(p.o) + goff, p.D, rows, p.D, lane);
    if constexpr (DUAL) store_rows_via_smem<2>(patch, pt, static_cast<uint16_t*>(p.to) + goff, p.D, rows, p.D, lane);
    if (qi < N) {
      p.lse2[static_cast<size_t>(bh) * N + qi] = (l > 0.f) ? m_used + log2f(l) : -INFINITY;
      p.mu[static_cast<size_t>(bh) * N + qi] = mul;
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 5) tmem_dealloc(tmem, COLS);
}

template <bool DUAL, bool BF16, bool PAD, bool DROP>
int launch_fwd64(const jvpfa_fwd_args& a, int* status, cudaStream_t stream) {
  CUtensorMap mQ, mTQ, mK, mTK, mV, mTV;
  auto tile = [&](CUtensorMap* m, const void* ptr, const jvpfa_strides& st, int box_rows) {
    return make_tile_map(m, make_view(ptr, st, a.H, a.N, a.D), a.B, a.H, a.N, a.D, box_rows, a.dtype);
  };
  bool ok = tile(&mQ, a.q, a.q_strides, 128) && tile(&mK, a.k, a.k_strides, 64) && tile(&mV, a.v, a.v_strides, 64);
  if (DUAL) {
    ok = ok && tile(&mTQ, a.tq, a.tq_strides, 128) && tile(&mTK, a.tk, a.tk_strides, 64) && tile(&mTV, a.tv, a.tv_strides, 64);
  } else {
    mTQ = mQ; mTK = mK; mTV = mV;
  }
  if (!ok) return JVPFA_ERR_LAUNCH;
  FwdKParams p = make_fwd_params<BF16>(a, status);
  auto kern = fwd64_sm100_kernel<DUAL, BF16, PAD, DROP>;
  static SmemOptIn opt_in;
  if (!opt_in.set(reinterpret_cast<const void*>(kern), Fwd64Cfg::smem_bytes())) return JVPFA_ERR_LAUNCH;
  kern<<<static_cast<unsigned>(p.n_qt) * static_cast<unsigned>(p.n_units), 192, Fwd64Cfg::smem_bytes(), stream>>>(mQ, mTQ, mK, mTK, mV, mTV, p);
  return cudaGetLastError() == cudaSuccess ? JVPFA_OK : JVPFA_ERR_LAUNCH;
}

template <bool PAD>
int launch_fwd64_by_mode(const jvpfa_fwd_args& a, int* status, cudaStream_t stream) {
  auto go = [&](auto dual, auto bf, auto drop) {
    return launch_fwd64<decltype(dual)::value, decltype(bf)::value, PAD, decltype(drop)::value>(a, status, stream);
  };
  auto by_drop = [&](auto dual, auto bf) {
    return a.dropout_p > 0.f ? go(dual, bf, std::true_type{}) : go(dual, bf, std::false_type{});
  };
  auto by_type = [&](auto dual) {
    return a.dtype == JVPFA_BF16 ? by_drop(dual, std::true_type{}) : by_drop(dual, std::false_type{});
  };
  return a.tq != nullptr ? by_type(std::true_type{}) : by_type(std::false_type{});
}

}  // namespace
}  // namespace jvpfa
