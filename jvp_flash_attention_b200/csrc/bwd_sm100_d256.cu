// Dual (JVP) attention backward for head dimensions 136 to 256, 16-bit inputs (same gradients as bwd_sm100.cuh).
//
// Why another split. At these widths neither the accumulators of a family (2 x 256 TMEM columns) leave room for score
// tiles nor do the four row-side operands of the full score set (4 x 64 KB) fit in shared memory. So
//   * every gradient has a launch family of its own with one 256-column accumulator (its TMEM partner is the 256 columns of
//     S, tS, X, A): dQ and dK need all four score tiles, dtQ = s dtS K and dtK only S and A, dV only S and tS, dtV only S.
//     29 tile products where the mathematics has 15; halving the output columns over two blocks instead would take 39;
//   * the operands that S, tS are made of stay resident (128 KB), everything else streams through a ring of six 16 KB slots
//     in 64-column slabs: a slab of a stacked column pair [c0; c1], a slab of a row-side operand of X and A, and the
//     column slabs once more for the output products.
//   * probabilities and score gradients keep 16 bits of significand and the range of fp32: they go to TMEM as bf16 hi and lo parts,
//     which take the place of the 32-bit score tile they come from, and meet bf16 columns c as e_hi c + e_lo c. fp16 columns come
//     split into bf16 hi + lo (exact; a product cannot take an fp16 operand against a bf16 one; a pre-pass writes them to the
//     workspace): e_hi c_hi + e_lo c_hi + e_hi c_lo. Rounded to the inputs' 16 bits instead, the gradients' errors were 1.3 to 1.5
//     times those of the fp32 CUDA-core kernels, and fp16 score gradients above 65504 overflowed.
// One launch holds the blocks of all families, heaviest family first: a launch per family leaves most of the SMs idle
// behind the longest row tile of a causal problem when there are few (batch, head) units.
// Whole call, us, B=2 H=8 N=1024 D=256 causal: bf16 268, fp16 325 with its pre-pass (16-bit probabilities and score gradients: 282,
// 286; CUDA cores, fp16: 12364); B=4 H=8 N=2048 causal: 1615, 2026 (1480, 1494); B=16 H=16 N=256: 579, 749 (586, 583).
// Bound: the slab stream (320 KB per 128 x 64 tile of dQ or dK at 256 columns, fp16 384 KB) and the output products (twice, fp16
// three times, those of 16-bit operands).
//
// Warps 0-7 element-wise (two warpgroups that split the 64 columns of a tile), warp 8 TMA producer, warp 9 MMA issuer; one
// static order of slots per block that producer and issuer both walk:
//   scores(0), grads(0), then per tile i: scores(i + 1), outputs(i), grads(i + 1)
#include "bwd_sm100.cuh"

namespace jvpfa {
namespace {

enum { KIND_FULL = 0, KIND_ONE = 1, KIND_PV2 = 2, KIND_PV1 = 3 };
// (the columns c of the output products are operands out[] of the maps)
//   FULL: S, tS, X, A -> out = dS c0 + dtS c1          (dQ, dK)
//   ONE:  S, Y        -> out = E c0, E = P (Y - stat)  (dtQ, dtK with Y = A, stat a; primal-only dQ, dK with Y = X, stat Delta)
//   PV2:  S, tS       -> out = P c2 + tP c3            (dV)
//   PV1:  S           -> out = P c2                    (dtV; primal-only dV)

struct WideFamily {
  int kind, qside;
  int r[4], c[4];   // operands (OP_*): rows of the S, tS products, rows of the X, A products; first and second column pair
  int stat;         // KIND_ONE: which negated statistic (2 = Delta, 3 = a)
  float scale;
  void* out;
};
constexpr int kMaxFamilies = 6;

struct WideMaps {
  BwdMaps in;
  CUtensorMap out[N_OPS];   // columns of the output products: bf16 inputs as they are, fp16 inputs split (hi at column 0, lo at D)
};

struct WideParams {
  int H, N, D;
  int b0;                   // first batch of this launch; fp16: where the out maps begin
  int n_rt, n_units, unit_group, n_fam;
  int causal;
  float c1, s;
  MaskView mv;
  const float4* stats;
  int* status;
  uint64_t budget_ns;
  WideFamily fam[kMaxFamilies];
};

constexpr int kSlots = 6;
constexpr int kSlotBytes = 128 * 128;       // 128 rows of 64 16-bit columns
constexpr int kHalfSlot = kSlotBytes / 2;   // the second tile of a stacked column pair
constexpr int kRowTile = 4 * kSlotBytes;    // a resident row-side operand: four slabs
constexpr int kWideBars = 2 * kSlots + 10;
constexpr size_t kWideSmem = 2 * kRowTile + kSlots * kSlotBytes + 2 * 4 * 64 * 4 + (kWideBars + 2) * 8;

template <int KIND, bool QSIDE, bool BF16>
__device__ __forceinline__ void wide_body(const WideMaps& wm, const WideParams& p, const WideFamily& f, int rt, int bh, uint8_t* smem,
                                          uint32_t tmem, const WaitCtx& w) {
  constexpr bool TS = KIND == KIND_FULL || KIND == KIND_PV2;     // tangent scores
  constexpr bool GR = KIND == KIND_FULL || KIND == KIND_ONE;     // score products of the upstream gradients
  constexpr int PARTS = BF16 ? 1 : 2;                            // column slabs of an output product: c, or c_hi and c_lo
  const BwdMaps& maps = wm.in;
  uint8_t* const sRA = smem;
  uint8_t* const sRB = smem + kRowTile;
  uint8_t* const ring = smem + 2 * kRowTile;
  float(*stats_s)[4][64] = reinterpret_cast<float(*)[4][64]>(ring + kSlots * kSlotBytes);   // [buffer][field, negated][column]
  uint64_t* bars = reinterpret_cast<uint64_t*>(ring + kSlots * kSlotBytes + 2 * 4 * 64 * 4);
  uint64_t *full = bars, *empty = bars + kSlots;
  uint64_t &ra_full = bars[2 * kSlots], &rb_full = bars[2 * kSlots + 1], &s_full = bars[2 * kSlots + 2], &s_free = bars[2 * kSlots + 3],
           &g_full = bars[2 * kSlots + 4], &acc_final = bars[2 * kSlots + 5];
  // A barrier must not complete a second phase before its waiter has seen the first. With X, A the element-wise warps meet
  // the issuer every tile (g_full of tile i + 1 is committed behind outputs(i)), with P, tP in one buffer they wait for e_free of
  // outputs(i), so one e_full does. With two buffers nothing holds tile i + 1 back while the issuer is between its commit of
  // S(i + 1) and its wait for e_full of tile i: every buffer has an e_full of its own, and tile i + 2 waits for e_free of outputs(i).
  constexpr int NE = KIND == KIND_PV1 ? 2 : 1;   // 64 columns of P hi, lo; P, tP hi, lo take all 128
  uint64_t* e_full = bars + 2 * kSlots + 6;   // [NE]
  uint64_t* e_free = bars + 2 * kSlots + 8;   // [NE]

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int b = bh / p.H, h = bh % p.H;
  const int r0 = rt * 128, N = p.N, D = p.D;
  const int n_ct = (N + 63) / 64, n_slabs = (D + 63) / 64;
  int j_begin = 0, j_end = n_ct;
  if (p.causal) {
    if (QSIDE) j_end = min(n_ct, (r0 + 127) / 64 + 1);
    else j_begin = r0 / 64;
  }
  auto tile_bits = [&](int j) -> uint8_t {
    if (p.mv.kind == JVPFA_MASK_NONE) return kTileAnyKept;
    uint8_t bits = QSIDE ? mask_tile_bits(p.mv, b, h, 2 * rt, j) : mask_tile_bits(p.mv, b, h, j, 2 * rt);
    if (2 * rt + 1 < p.mv.n64) bits |= QSIDE ? mask_tile_bits(p.mv, b, h, 2 * rt + 1, j) : mask_tile_bits(p.mv, b, h, j, 2 * rt + 1);
    return bits;
  };
  auto next_active = [&](int j) {
    while (j < j_end && !(tile_bits(j) & kTileAnyKept)) ++j;
    return j;
  };
  int slot = 0;
  uint32_t phase = 0;
  auto advance = [&]() {
    if (++slot == kSlots) { slot = 0; phase ^= 1; }
  };

  if (warp == 8) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      auto load_rows = [&](uint8_t* dst, int op, uint64_t* bar) {
        mbar_arrive_expect_tx(bar, n_slabs * kSlotBytes);
        for (int sl = 0; sl < n_slabs; ++sl) tma_load_tile(dst + sl * kSlotBytes, &maps.row[op], bar, 64 * sl, r0, h, b);
      };
      // one slot: a slab of a column pair (second tile only if c1 >= 0) or of a row-side operand
      auto slot_cols = [&](int c0, int c1, int sl, int crow) {
        mbar_wait(&empty[slot], phase ^ 1, w, 10);
        mbar_arrive_expect_tx(&full[slot], c1 >= 0 ? kSlotBytes : kHalfSlot);
        tma_load_tile(ring + slot * kSlotBytes, &maps.col[c0], &full[slot], 64 * sl, crow, h, b);
        if (c1 >= 0) tma_load_tile(ring + slot * kSlotBytes + kHalfSlot, &maps.col[c1], &full[slot], 64 * sl, crow, h, b);
        advance();
      };
      auto slot_rows = [&](int op, int sl) {
        mbar_wait(&empty[slot], phase ^ 1, w, 11);
        mbar_arrive_expect_tx(&full[slot], kSlotBytes);
        tma_load_tile(ring + slot * kSlotBytes, &maps.row[op], &full[slot], 64 * sl, r0, h, b);
        advance();
      };
      auto scores = [&](int j) {
        for (int sl = 0; sl < n_slabs; ++sl) slot_cols(f.c[0], TS ? f.c[1] : -1, sl, j * 64);
      };
      auto grads = [&](int j) {
        if constexpr (KIND == KIND_FULL) {
          for (int sl = 0; sl < n_slabs; ++sl) {
            slot_cols(f.c[2], f.c[3], sl, j * 64);
            slot_rows(QSIDE ? f.r[3] : f.r[2], sl);   // the operand that multiplies the whole pair
            slot_rows(QSIDE ? f.r[2] : f.r[3], sl);   // the one that multiplies one tile of it
          }
        } else if constexpr (KIND == KIND_ONE) {
          for (int sl = 0; sl < n_slabs; ++sl) slot_cols(f.c[2], -1, sl, j * 64);
        }
      };
      auto outputs = [&](int j) {
        const CUtensorMap *m0 = &wm.out[GR ? f.c[0] : f.c[2]], *m1 = &wm.out[GR ? f.c[1] : f.c[3]];
        for (int sl = 0; sl < n_slabs; ++sl) {
#pragma unroll
          for (int part = 0; part < PARTS; ++part) {
            const int x = part * D + 64 * sl, bo = BF16 ? b : b - p.b0;
            mbar_wait(&empty[slot], phase ^ 1, w, 12);
            mbar_arrive_expect_tx(&full[slot], TS ? kSlotBytes : kHalfSlot);
            tma_load_tile(ring + slot * kSlotBytes, m0, &full[slot], x, j * 64, h, bo);
            if constexpr (TS) tma_load_tile(ring + slot * kSlotBytes + kHalfSlot, m1, &full[slot], x, j * 64, h, bo);
            advance();
          }
        }
      };
      load_rows(sRA, f.r[0], &ra_full);
      if constexpr (TS) load_rows(sRB, f.r[1], &rb_full);
      else if constexpr (KIND == KIND_ONE) load_rows(sRB, f.r[2], &rb_full);
      int j = next_active(j_begin);
      if (j < j_end) {
        scores(j);
        grads(j);
      }
      while (j < j_end) {
        const int jn = next_active(j + 1);
        if (jn < j_end) scores(jn);
        outputs(j);
        if (jn < j_end) grads(jn);
        j = jn;
      }
    }
    __syncwarp();
  } else if (warp == 9) {
    // ------------------------------------------------------------------ MMA issuer (all lanes walk the loops, one issues)
    const bool leader = elect_one_sync();
    const uint32_t lead = leader ? 1u : 0u;
    auto wait_all = [&](uint64_t* bar, uint32_t parity, int site) {
      mbar_wait(bar, parity, w, site);
      __syncwarp();
    };
    constexpr uint32_t FMT = BF16 ? FMT_BF16 : FMT_F16;
    const uint32_t idesc_64 = make_idesc(FMT, 128, 64, 0, 0), idesc_128 = make_idesc(FMT, 128, 128, 0, 0);
    const uint32_t idesc_out = make_idesc(FMT_BF16, 128, 64, 0, 1);
    const uint32_t T0 = tmem + 256, T2 = T0 + 128;
    const int ksteps = (D + 15) / 16;
    auto wait_slot = [&]() {
      wait_all(&full[slot], phase, 20);
      tc_fence_after_sync();
    };
    // dst (+)= a slab [128 x 64] * b slab^T, the K steps of slab sl that hold data
    auto nt = [&](uint32_t dst, const uint8_t* a, const uint8_t* c, uint32_t idesc, int sl, bool first) {
      const uint64_t da = desc_kmajor_sw128(smem_u32(a)), db = desc_kmajor_sw128(smem_u32(c));
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (4 * sl + k < ksteps) umma_ss_pred(dst, da + 2 * k, db + 2 * k, idesc, !(first && k == 0), lead);
    };
    auto release = [&](uint64_t* bar) {
      if (leader) umma_commit(bar);
    };
    auto scores = [&](int i) {
      if (i >= 1) wait_all(&s_free, (i - 1) & 1, 21);
      for (int sl = 0; sl < n_slabs; ++sl) {
        wait_slot();
        const uint8_t* c = ring + slot * kSlotBytes;
        nt(T0, sRA + sl * kSlotBytes, c, TS ? idesc_128 : idesc_64, sl, sl == 0);              // [S | R0 c1^T]
        if constexpr (TS) nt(T0 + 64, sRB + sl * kSlotBytes, c, idesc_64, sl, false);          // tS += R1 c0^T
        release(&empty[slot]);
        advance();
      }
      release(&s_full);
    };
    auto grads = [&]() {
      if constexpr (KIND == KIND_FULL) {
        for (int sl = 0; sl < n_slabs; ++sl) {
          const int cs = slot;
          wait_slot();
          advance();
          wait_slot();
          nt(T2, ring + slot * kSlotBytes, ring + cs * kSlotBytes, idesc_128, sl, sl == 0);     // Q: [A | gtO tV^T], K: [V gO^T | A^T]
          release(&empty[slot]);
          advance();
          wait_slot();
          if constexpr (QSIDE) nt(T2 + 64, ring + slot * kSlotBytes, ring + cs * kSlotBytes, idesc_64, sl, false);          // X += gO V^T
          else nt(T2, ring + slot * kSlotBytes, ring + cs * kSlotBytes + kHalfSlot, idesc_64, sl, false);                  // X^T += tV gtO^T
          release(&empty[slot]);
          release(&empty[cs]);
          advance();
        }
        release(&g_full);
      } else if constexpr (KIND == KIND_ONE) {
        for (int sl = 0; sl < n_slabs; ++sl) {
          wait_slot();
          nt(T2, sRB + sl * kSlotBytes, ring + slot * kSlotBytes, idesc_64, sl, sl == 0);
          release(&empty[slot]);
          advance();
        }
        release(&g_full);
      }
    };
    auto outputs = [&](int i) {
      wait_all(&e_full[i % NE], (i / NE) & 1, 22);
      // FULL: dS replaces X, dtS replaces A in place, PV: P, tP beside the scores; of 64 score columns, each warpgroup's 32 become
      // 16 columns of hi and 16 of lo parts
      const uint32_t E0 = KIND == KIND_FULL ? (QSIDE ? T2 + 64 : T2) : (GR ? T2 : T2 + (i % NE) * 64);
      const uint32_t E1 = KIND == KIND_FULL && QSIDE ? T2 : T2 + 64;
      for (int sl = 0; sl < n_slabs; ++sl) {
        const uint32_t acc = tmem + 64 * sl;
#pragma unroll
        for (int part = 0; part < PARTS; ++part) {
          wait_slot();
          const uint64_t d0 = desc_mnmajor_sw128(smem_u32(ring + slot * kSlotBytes), kSlotBytes);
          const uint64_t d1 = desc_mnmajor_sw128(smem_u32(ring + slot * kSlotBytes + kHalfSlot), kSlotBytes);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const uint32_t hi = (k & 1) * 8 + (k >> 1) * 32, lo = hi + 16;
            const uint64_t dk = static_cast<uint64_t>((k * 2048) >> 4);
            umma_ts_pred(acc, E0 + hi, d0 + dk, idesc_out, i > 0 || part > 0 || k > 0, lead);
            if (part == 0) umma_ts_pred(acc, E0 + lo, d0 + dk, idesc_out, 1, lead);
            if constexpr (TS) {
              umma_ts_pred(acc, E1 + hi, d1 + dk, idesc_out, 1, lead);
              if (part == 0) umma_ts_pred(acc, E1 + lo, d1 + dk, idesc_out, 1, lead);
            }
          }
          release(&empty[slot]);
          advance();
        }
      }
      if constexpr (!GR) release(&e_free[i % NE]);
    };
    wait_all(&ra_full, 0, 23);
    if constexpr (KIND != KIND_PV1) wait_all(&rb_full, 0, 24);
    int j = next_active(j_begin), it = 0;
    if (j < j_end) {
      scores(0);
      grads();
    }
    for (; j < j_end; ++it) {
      const int jn = next_active(j + 1);
      if (jn < j_end) scores(it + 1);
      outputs(it);
      if (jn < j_end) grads();
      j = jn;
    }
    if (leader) {
      if (it > 0) umma_commit(&acc_final);
      else mbar_arrive(&acc_final);
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ element-wise + epilogue
    const int wg = warp >> 2;          // columns [32 wg, 32 wg + 32) of every tile
    const int gr = r0 + (warp & 3) * 32 + lane;   // sequence index of this thread's row
    const int gr_c = min(gr, N - 1);
    const size_t row_base = static_cast<size_t>(bh) * N;
    const uint32_t lane_off = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t T0 = tmem + 256 + lane_off;
    float4 nst = make_float4(0.f, 0.f, 0.f, 0.f);   // negated statistics of this thread's query row
    if constexpr (QSIDE) {
      const float4 st = p.stats[row_base + gr_c];
      nst = make_float4(-st.x, -st.y, -st.z, -st.w);
      if (st.x == -INFINITY) nst.x = -INFINITY;   // fully excluded query: P = 0
    }
    const float2 c1_2 = make_float2(p.c1, p.c1), s_2 = make_float2(p.s, p.s);
    // this thread's 32 values of a tile, pair i = value(i), as 16 columns of hi and 16 of lo parts from TMEM column `col` on
    auto store_hi_lo = [](uint32_t col, auto value) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        uint32_t hi[8], lo[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float2 v = value(8 * q + i);
          hi[i] = pack2<true>(v.x, v.y);
          lo[i] = pack2_residual(v.x, v.y, hi[i]);
        }
        tmem_st_x8(col + 8 * q, hi);
        tmem_st_x8(col + 16 + 8 * q, lo);
      }
    };
    auto fetch_stats = [&](int j) -> float4 {   // statistics of the next column tile, fetched one tile ahead
      float4 sv = make_float4(INFINITY, 0.f, 0.f, 0.f);
      if (!QSIDE && tid < 64 && j < j_end && j * 64 + tid < N) sv = __ldg(&p.stats[row_base + j * 64 + tid]);
      return sv;
    };
    int it = 0;
    int j_next = next_active(j_begin);
    float4 sv_next = fetch_stats(j_next);
    for (int j = j_next; j < j_end; j = j_next, ++it) {
      const uint8_t bits = tile_bits(j);
      const int c0 = j * 64, cw = c0 + 32 * wg;
      j_next = next_active(j + 1);
      if constexpr (!QSIDE) {
        if (tid < 64) {
          const float4 sv = sv_next;
          stats_s[it & 1][0][tid] = (sv.x == -INFINITY) ? -INFINITY : -sv.x;
          stats_s[it & 1][1][tid] = -sv.y;
          stats_s[it & 1][2][tid] = -sv.z;
          stats_s[it & 1][3][tid] = -sv.w;
        }
        named_bar_sync(1, 256);
        sv_next = fetch_stats(j_next);
      }
      auto stat2 = [&](int field, int i) -> float2 {
        if constexpr (QSIDE) {
          const float v = field == 0 ? nst.x : (field == 1 ? nst.y : (field == 2 ? nst.z : nst.w));
          return make_float2(v, v);
        } else {
          return *reinterpret_cast<const float2*>(&stats_s[it & 1][field][32 * wg + 2 * i]);
        }
      };
      mbar_wait(&s_full, it & 1, w, 30);
      tc_fence_after_sync();
      float2 P2[16], ts2[16];
      {
        uint32_t a0[32], a1[32];
        tmem_ld_x32(T0 + 32 * wg, a0);
        if constexpr (TS) tmem_ld_x32(T0 + 64 + 32 * wg, a1);
        tmem_wait_ld();
        tc_fence_before_sync();
        mbar_arrive(&s_free);   // S, tS are in registers: the next tile's products may overwrite them
        float2 x2[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          x2[i] = __ffma2_rn(make_float2(__uint_as_float(a0[2 * i]), __uint_as_float(a0[2 * i + 1])), c1_2, stat2(0, i));
          if constexpr (TS) ts2[i] = __fmul2_rn(make_float2(__uint_as_float(a1[2 * i]), __uint_as_float(a1[2 * i + 1])), s_2);
        }
        int mask_mode = 0;   // how this thread's own 64x64 mask tile is applied, see mask_tile_mode
        const int my_qt = QSIDE ? (gr_c >> 6) : j, my_kt = QSIDE ? j : (gr_c >> 6);
        if (p.mv.kind != JVPFA_MASK_NONE && (bits & kTileAnyMasked))
          mask_mode = mask_tile_mode(p.mv, mask_tile_bits(p.mv, b, h, my_qt, my_kt));
        if (mask_mode == 1) {
          const float other = p.mv.kind == JVPFA_MASK_BOOL ? -INFINITY : mask_tile_value(p.mv, b, h, my_qt, my_kt) * 1.4426950408889634f;
          mask_apply_bits(x2, QSIDE ? mask_row_bits(p.mv, b, h, gr_c, j, wg) : mask_col_bits(p.mv, b, h, j, gr_c, wg), other);
        }
        const bool need_causal = p.causal && (QSIDE ? (c0 + 63 > r0) : (r0 + 127 > c0));
        const bool need_bound = QSIDE && c0 + 64 > N;
        if (need_causal || need_bound || mask_mode == 2) {
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            float bias[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) bias[i] = 0.f;
            if (mask_mode == 2) {
              if constexpr (QSIDE) mask_bias_run<16>(bias, p.mv, b, h, gr_c, cw + 16 * q, N, true);
              else mask_bias_run<16>(bias, p.mv, b, h, cw + 16 * q, gr_c, N, false);
            }
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const int col = cw + 16 * q + i;
              if ((need_causal && (QSIDE ? col > gr : gr > col)) || (need_bound && col >= N)) bias[i] = -INFINITY;
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) x2[8 * q + i] = __fadd2_rn(x2[8 * q + i], make_float2(bias[2 * i], bias[2 * i + 1]));
          }
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) P2[i] = make_float2(fast_exp2(x2[i].x), fast_exp2(x2[i].y));
      }
      if constexpr (GR) {
        mbar_wait(&g_full, it & 1, w, 31);
        tc_fence_after_sync();
        const uint32_t TY = T0 + 128 + 32 * wg;                                   // KIND_ONE
        const uint32_t TA = QSIDE ? TY : TY + 64, TX = QSIDE ? TY + 64 : TY;      // KIND_FULL
        if constexpr (KIND == KIND_FULL) {   // A -> dtS = P (A - a), and everything of dS that does not need X
          uint32_t ar[32];
          tmem_ld_x32(TA, ar);
          tmem_wait_ld();
          store_hi_lo(TA, [&](int i) -> float2 {
            const float2 A = make_float2(__uint_as_float(ar[2 * i]), __uint_as_float(ar[2 * i + 1]));
            const float2 d = __fadd2_rn(A, stat2(3, i));
            const float2 t = __ffma2_rn(ts2[i], d, stat2(2, i));                // ts (A - a) - Delta
            ts2[i] = __ffma2_rn(stat2(1, i), A, t);                             // - mu A
            return __fmul2_rn(P2[i], d);
          });
        }
        // X -> dS = P (X + the above), or Y -> E = P (Y - stat)
        uint32_t xr[32];
        tmem_ld_x32(KIND == KIND_FULL ? TX : TY, xr);
        tmem_wait_ld();
        store_hi_lo(KIND == KIND_FULL ? TX : TY, [&](int i) -> float2 {
          const float2 X = make_float2(__uint_as_float(xr[2 * i]), __uint_as_float(xr[2 * i + 1]));
          const float2 add = KIND == KIND_FULL ? ts2[i] : (f.stat == 2 ? stat2(2, i) : stat2(3, i));
          return __fmul2_rn(P2[i], __fadd2_rn(X, add));
        });
      } else {
        const uint32_t EP = T0 + 128 + (it % NE) * 64 + 32 * wg;   // this thread's columns of P hi, lo; tP is 64 columns further
        if (it >= NE) {   // the output products of tile it - NE read this buffer
          mbar_wait(&e_free[it % NE], (it / NE - 1) & 1, w, 32);
          tc_fence_after_sync();
        }
        store_hi_lo(EP, [&](int i) -> float2 { return P2[i]; });
        if constexpr (TS) store_hi_lo(EP + 64, [&](int i) -> float2 { return __fmul2_rn(P2[i], __fadd2_rn(ts2[i], stat2(1, i))); });
      }
      tmem_wait_st();
      tc_fence_before_sync();
      mbar_arrive(&e_full[it % NE]);
    }
    mbar_wait(&acc_final, 0, w, 33);
    tc_fence_after_sync();
    if (it == 0) {   // nothing was multiplied: the row-side loads may still be in flight
      mbar_wait(&ra_full, 0, w, 34);
      if constexpr (KIND != KIND_PV1) mbar_wait(&rb_full, 0, w, 35);
    }
    // each warpgroup writes 128 of the 256 columns, 64 at a time, through this warp's patch of the first row-side tile
    uint8_t* patch = sRA + warp * (32 * 128);
    const int wrow0 = r0 + (warp & 3) * 32, rows = N - wrow0;
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      const int col0 = wg * 128 + g * 64;
      if (col0 >= D) break;
      uint32_t q0[2][16];
#pragma unroll
      for (int cc = 0; cc < 2; ++cc) {
        uint32_t a0[32];
        if (it > 0) {
          tmem_ld_x32(tmem + lane_off + col0 + cc * 32, a0);
          tmem_wait_ld();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) a0[i] = 0u;
        }
#pragma unroll
        for (int i = 0; i < 16; ++i)
          q0[cc][i] = pack2<BF16>(__uint_as_float(a0[2 * i]) * f.scale, __uint_as_float(a0[2 * i + 1]) * f.scale);
      }
      store_rows_via_smem<2>(patch, q0, static_cast<uint16_t*>(f.out) + (row_base + wrow0) * D + col0, D, rows, D - col0, lane);
    }
  }
}

template <bool BF16>
__global__ void __launch_bounds__(320, 1) bwd_sm100_wide_kernel(const __grid_constant__ WideMaps maps, const __grid_constant__ WideParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 2 * kRowTile + kSlots * kSlotBytes + 2 * 4 * 64 * 4);
  uint32_t& tmem_base_s = *reinterpret_cast<uint32_t*>(bars + kWideBars);
  int& poisoned = *reinterpret_cast<int*>(bars + kWideBars + 1);
  if ((smem_u32(smem) & 1023u) != 0u) {  // the swizzled layouts need this; never observed otherwise
    if (threadIdx.x == 0) atomicCAS(p.status, 0, WAIT_TIMEOUT_BASE + 99);
    return;
  }
  const int warp = threadIdx.x >> 5;
  // blocks by family first, the longest family first (the families' code must not alternate on the SMs, see bwd_sm100_kernel),
  // inside a family the heaviest row tiles first: late query tiles, early key tiles. Against families group by group, whole call:
  // B=16 H=16 N=256 D=256 bf16 724 -> 638 us, B=4 H=8 N=2048 causal 1802 -> 1735 us, B=2 H=8 N=1024 causal 298 -> 297 us
  const int per_fam = p.n_rt * p.n_units, fi = static_cast<int>(blockIdx.x) / per_fam;
  const WideFamily& f = p.fam[fi];
  const BlockWork work = block_work(static_cast<int>(blockIdx.x) - fi * per_fam, p.n_rt, p.n_units, p.unit_group, p.causal && f.qside);
  const int rt = work.tile, bh = work.unit + p.b0 * p.H;
  const WaitCtx w{p.status, &poisoned, p.budget_ns};
  if (threadIdx.x == 0) {
    poisoned = 0;
    for (int i = 0; i < 2 * kSlots + 2; ++i) mbar_init(&bars[i], 1);     // full, empty, rows A, rows B
    mbar_init(&bars[2 * kSlots + 2], 1);      // s_full
    mbar_init(&bars[2 * kSlots + 3], 256);    // s_free
    mbar_init(&bars[2 * kSlots + 4], 1);      // g_full
    mbar_init(&bars[2 * kSlots + 5], 1);      // acc_final
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars[2 * kSlots + 6 + i], 256);   // e_full
      mbar_init(&bars[2 * kSlots + 8 + i], 1);     // e_free
    }
    fence_mbar_init();
  }
  __syncthreads();
  if (warp == 9) {
    tmem_alloc(&tmem_base_s, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  if (warp != 8) named_bar_sync(2, 288);   // the TMA producer starts loading while TMEM is being allocated
  tc_fence_after_sync();
  const uint32_t tmem = warp == 8 ? 0u : tmem_base_s;
  if (f.kind == KIND_FULL) {
    if (f.qside) wide_body<KIND_FULL, true, BF16>(maps, p, f, rt, bh, smem, tmem, w);
    else wide_body<KIND_FULL, false, BF16>(maps, p, f, rt, bh, smem, tmem, w);
  } else if (f.kind == KIND_ONE) {
    if (f.qside) wide_body<KIND_ONE, true, BF16>(maps, p, f, rt, bh, smem, tmem, w);
    else wide_body<KIND_ONE, false, BF16>(maps, p, f, rt, bh, smem, tmem, w);
  } else if (f.kind == KIND_PV2) {
    wide_body<KIND_PV2, false, BF16>(maps, p, f, rt, bh, smem, tmem, w);
  } else {
    wide_body<KIND_PV1, false, BF16>(maps, p, f, rt, bh, smem, tmem, w);
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 9) tmem_dealloc(tmem, 512);
}

template <bool BF16>
int launch_wide(const jvpfa_bwd_args& a, int* status, cudaStream_t stream, const LaunchMarks& marks) {
  const bool dual = a.tq != nullptr;
  float4* stats = reinterpret_cast<float4*>(static_cast<uint8_t*>(a.workspace) + kStatusBytes);
  marks.mark(0);
  const int rc = launch_preprocess<BF16>(a, stats, stream);
  if (rc != JVPFA_OK) return rc;
  WideMaps maps;
  if (!maps.in.encode(a)) return JVPFA_ERR_LAUNCH;
  WideParams p{};
  p.H = a.H; p.N = a.N; p.D = a.D; p.causal = a.causal;
  p.s = a.sm_scale;
  p.c1 = a.sm_scale * 1.4426950408889634f;
  p.mv = make_mask_view(a.mask, a.mask_summary, a.B, a.H, a.N);
  p.stats = stats;
  p.status = status;
  p.budget_ns = wait_budget_ns();
  const int rows_q[4] = {OP_Q, OP_TQ, OP_GO, OP_GTO}, rows_k[4] = {OP_K, OP_TK, OP_V, OP_TV};
  auto add = [&](int kind, bool qside, void* out, float scale, int stat, bool through_tangent) {
    WideFamily& f = p.fam[p.n_fam++];
    f.kind = kind; f.qside = qside; f.out = out; f.scale = scale; f.stat = stat;
    for (int i = 0; i < 4; ++i) {
      f.r[i] = (qside ? rows_q : rows_k)[i];
      f.c[i] = (qside ? rows_k : rows_q)[i];
    }
    // the single score product of the gradients is Y = A = gtO V^T instead of X = gO V^T, the single output product one with
    // gtO instead of gO
    if (through_tangent) {
      if (qside) f.r[2] = OP_GTO;
      else f.c[2] = OP_GTO;
    }
  };
  if (dual) {
    add(KIND_FULL, true, a.dq, a.sm_scale, 0, false);
    add(KIND_FULL, false, a.dk, a.sm_scale, 0, false);
    add(KIND_PV2, false, a.dv, 1.f, 0, false);
    add(KIND_ONE, true, a.dtq, a.sm_scale, 3, true);
    add(KIND_ONE, false, a.dtk, a.sm_scale, 3, true);
    add(KIND_PV1, false, a.dtv, 1.f, 0, true);
  } else {
    add(KIND_ONE, true, a.dq, a.sm_scale, 2, false);
    add(KIND_ONE, false, a.dk, a.sm_scale, 2, false);
    add(KIND_PV1, false, a.dv, 1.f, 0, false);
  }
  p.n_rt = (a.N + 127) / 128;
  // All row tiles of a group of units come before the next group's, so the group bounds both the tail (heaviest blocks first
  // only inside a group) and the tensors that the running blocks stream: eight per unit, kept to half of L2.
  const size_t unit_bytes = 16 * static_cast<size_t>(a.N) * a.D;
  const int fit = static_cast<int>((size_t{64} << 20) / unit_bytes);
  auto kern = bwd_sm100_wide_kernel<BF16>;
  static SmemOptIn opt_in;
  if (!opt_in.set(reinterpret_cast<const void*>(kern), kWideSmem)) return JVPFA_ERR_LAUNCH;
  marks.mark(1);
  // the columns of the output products; fp16: a launch per group of batches whose split tensors fit the workspace
  const int n_out = dual ? 6 : 3, ops[6] = {OP_Q, OP_K, OP_GO, OP_TQ, OP_TK, OP_GTO};
  const int step = BF16 ? a.B : split_f16_batches(n_out, a.B, a.H, a.N, a.D);
  const void* const src[6] = {a.q, a.k, a.go, a.tq, a.tk, a.gto};
  const jvpfa_strides* const st[6] = {&a.q_strides, &a.k_strides, &a.go_strides, &a.tq_strides, &a.tk_strides, &a.gto_strides};
  uint16_t* const split = reinterpret_cast<uint16_t*>(reinterpret_cast<uint8_t*>(stats) +
                                                      align_up(static_cast<size_t>(a.B) * a.H * a.N * sizeof(float4), 256));
  for (int b0 = 0; b0 < a.B; b0 += step) {
    const int nb = a.B - b0 < step ? a.B - b0 : step;
    for (int i = 0; i < N_OPS; ++i) maps.out[i] = maps.in.col[i];
    if constexpr (!BF16) {
      TensorView views[6];
      uint16_t* dst[6];
      for (int i = 0; i < n_out; ++i) {
        views[i] = batches_from(make_view(src[i], *st[i], a.H, a.N, a.D), b0, 2);
        dst[i] = split + i * split_f16_elems(step, a.H, a.N, a.D);
        if (!make_split_f16_map(&maps.out[ops[i]], dst[i], nb, a.H, a.N, a.D, 64)) return JVPFA_ERR_LAUNCH;
      }
      const int rc_split = launch_split_f16(views, dst, n_out, nb, a.H, a.N, a.D, stream);
      if (rc_split != JVPFA_OK) return rc_split;
    }
    p.b0 = b0;
    p.n_units = nb * a.H;
    p.unit_group = fit < 1 ? 1 : (fit < p.n_units ? fit : p.n_units);
    kern<<<static_cast<unsigned>(p.n_fam) * p.n_rt * p.n_units, 320, kWideSmem, stream>>>(maps, p);
    if (cudaGetLastError() != cudaSuccess) return JVPFA_ERR_LAUNCH;
  }
  for (int i = 2; i < 5; ++i) marks.mark(i);
  return JVPFA_OK;
}

}  // namespace

int launch_bwd_sm100_d256(const jvpfa_bwd_args& a, int* status, cudaStream_t stream, const LaunchMarks& marks) {
  return a.dtype == JVPFA_BF16 ? launch_wide<true>(a, status, stream, marks) : launch_wide<false>(a, status, stream, marks);
}

}  // namespace jvpfa
