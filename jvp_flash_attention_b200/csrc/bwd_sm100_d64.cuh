// Dual (JVP) attention backward for head dimensions up to 64, 16-bit inputs (gradients and notation of bwd_sm100.cuh).
//
// Two families per problem, in one launch: Q (dQ, dtQ; rows = queries) and KV (dK, dtK, dV, dtV; rows = keys). A CTA owns 128
// rows and streams 64-wide column tiles.
//
// At these widths the products of a tile take 1280 (Q) / 1664 (KV) cycles of the tensor pipe while the element-wise chain of
// a tile (scores -> P -> A -> dtS -> X -> dS, with two TMEM round trips) is as long as that or longer. With all element-wise
// warps on the same tile the two run one after the other for much of the time (2363 / 3082 cycles a tile). Here the two
// element-wise warpgroups work on different tiles: warpgroup g takes tiles g, g + 2, ...; its threads own a whole row of
// 64 scores (no exchange inside a row), and one warpgroup's chain runs beside the products of the other's tile.
// TMEM: accumulators (Q: 128 columns, KV: 256), then 128 columns per warpgroup. A warpgroup's columns hold [S | tS] until its
// threads have read them, then X and A, in whose place the 16-bit operands of the output products are written: of every 16
// columns of A the first 8 become dtS (KV: the other 8 tP), of X dS (KV: and P).
//   warps 0-7   two element-wise warpgroups
//   warp 8      TMA producer: rows, then a ring of four stages with both column pairs of a tile
//   warp 9      issues the score products:  [S | tS](t + 1) when the outputs of tile t - 1 are complete, X, A(t) when the
//               threads have S, tS(t) in registers
//   warp 10     issues the output products (all of them: one thread, so the accumulators see them in order)
#pragma once
#include "bwd_sm100.cuh"

namespace jvpfa {
namespace {

struct Bwd64Cfg {
  static constexpr int STAGES = 4;
  static constexpr int TILE_R = 128 * 128;        // 128 rows of 64 16-bit columns
  static constexpr int HALF = 64 * 128;           // a 64-row tile
  static constexpr int PAIR = 2 * HALF;
  static constexpr int STAGE = 2 * PAIR;          // first and second column pair
  static constexpr int NBAR = 3 + 3 * STAGES + 14;
  static constexpr size_t smem_bytes() { return 4 * TILE_R + STAGES * STAGE + 2 * 2 * 4 * 64 * 4 + (NBAR + 2) * 8; }
};

struct Bwd64Params {
  BwdKParams k;         // of both families; out0, out1: dK, dtK; out2, out3: dV, dtV
  void *dq, *dtq;
};

template <bool QF, bool BF16, bool PAD, bool DUAL, bool DROP>
__device__ __forceinline__ void bwd64_body(const BwdMaps& maps, const Bwd64Params& pp, int rt, int bh, uint8_t* smem, uint32_t tmem,
                                           const WaitCtx& w) {
  using C = Bwd64Cfg;
  const BwdKParams& p = pp.k;
  constexpr int ST = C::STAGES;
  auto sR = [&](int i) { return smem + i * C::TILE_R; };
  auto sA = [&](int st) { return smem + 4 * C::TILE_R + st * C::STAGE; };
  auto sB = [&](int st) { return sA(st) + C::PAIR; };
  // negated statistics of a column tile's queries: [warpgroup][buffer][-lse2, -mu, -Delta, -a][column]
  float(*stats_s)[2][4][64] = reinterpret_cast<float(*)[2][4][64]>(smem + 4 * C::TILE_R + ST * C::STAGE);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 4 * C::TILE_R + ST * C::STAGE + 2 * 2 * 4 * 64 * 4);
  uint64_t &r01_full = bars[0], &r23_full = bars[1], &acc_final = bars[2];
  uint64_t *a_full = bars + 3, *b_full = a_full + ST, *empty = b_full + ST;
  uint64_t *s_full = empty + ST, *a_ready = s_full + 2, *x_full = a_ready + 2, *s_free = x_full + 2, *e1_full = s_free + 2,
           *e0_full = e1_full + 2, *o_done = e0_full + 2;   // [warpgroup]

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int b = bh / p.H, h = bh % p.H;
  const int r0 = rt * 128, N = p.N;
  int j_begin = 0, j_end = (N + 63) / 64;
  if (p.causal) {
    if (QF) j_end = min(j_end, (r0 + 127) / 64 + 1);
    else j_begin = r0 / 64;
  }
  auto next_active = [&](int j) {
    if (p.mv.kind == JVPFA_MASK_NONE) return j;
    for (; j < j_end; ++j) {
      uint8_t bits = QF ? mask_tile_bits(p.mv, b, h, 2 * rt, j) : mask_tile_bits(p.mv, b, h, j, 2 * rt);
      if (2 * rt + 1 < p.mv.n64) bits |= QF ? mask_tile_bits(p.mv, b, h, 2 * rt + 1, j) : mask_tile_bits(p.mv, b, h, j, 2 * rt + 1);
      if (bits & kTileAnyKept) break;
    }
    return j;
  };
  constexpr uint32_t TG = QF ? 128 : 256;                      // first column of warpgroup 0's score columns
  // where A and X are: family Q computes [A | gtO tV^T] and X += gO V^T, family KV [V gO^T | A^T] and X^T += tV gtO^T
  constexpr uint32_t OA = QF ? 0 : 64, OX = DUAL ? (QF ? 64 : 0) : 64;

  // 168 registers a thread at launch = 12 warps x 32 x 168: 216 for the 8 element-wise warps, 72 for the other 4 (inside
  // the branch: the compiler allocates the registers of what the instruction dominates)
  if (warp >= 8) {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
  if (warp == 8) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      constexpr int R0 = QF ? OP_Q : OP_K, R1 = QF ? OP_TQ : OP_TK, R2 = QF ? OP_GO : OP_V, R3 = QF ? OP_GTO : OP_TV;
      constexpr int C0 = QF ? OP_K : OP_Q, C1 = QF ? OP_TK : OP_TQ, C2 = QF ? OP_V : OP_GO, C3 = QF ? OP_TV : OP_GTO;
      mbar_arrive_expect_tx(&r01_full, (DUAL ? 2 : 1) * C::TILE_R);
      tma_load_tile(sR(0), &maps.row[R0], &r01_full, 0, r0, h, b);
      if constexpr (DUAL) tma_load_tile(sR(1), &maps.row[R1], &r01_full, 0, r0, h, b);
      auto load_r23 = [&]() {
        mbar_arrive_expect_tx(&r23_full, (DUAL ? 2 : 1) * C::TILE_R);
        tma_load_tile(sR(2), &maps.row[R2], &r23_full, 0, r0, h, b);
        if constexpr (DUAL) tma_load_tile(sR(3), &maps.row[R3], &r23_full, 0, r0, h, b);
      };
      int t = 0;
      for (int j = next_active(j_begin); j < j_end; j = next_active(j + 1), ++t) {
        const int st = t % ST, crow = j * 64;
        mbar_wait(&empty[st], ((t / ST) & 1) ^ 1, w, 10);
        mbar_arrive_expect_tx(&a_full[st], DUAL ? C::PAIR : C::HALF);
        tma_load_tile(sA(st), &maps.col[C0], &a_full[st], 0, crow, h, b);
        if constexpr (DUAL) tma_load_tile(sA(st) + C::HALF, &maps.col[C1], &a_full[st], 0, crow, h, b);
        if (t == 0) load_r23();
        mbar_arrive_expect_tx(&b_full[st], DUAL ? C::PAIR : C::HALF);
        tma_load_tile(sB(st), &maps.col[C2], &b_full[st], 0, crow, h, b);
        if constexpr (DUAL) tma_load_tile(sB(st) + C::HALF, &maps.col[C3], &b_full[st], 0, crow, h, b);
      }
      if (t == 0) load_r23();   // no column tile takes part: the epilogue still waits for these loads
    }
    __syncwarp();
  } else if (warp == 9 || warp == 10) {
    // ------------------------------------------------------------------ MMA issuers (all lanes walk the loops, one issues)
    const uint32_t lead = elect_one_sync() ? 1u : 0u;
    auto wait_all = [&](uint64_t* bar, uint32_t parity, int site) {
      mbar_wait(bar, parity, w, site);
      __syncwarp();
    };
    auto commit = [&](uint64_t* bar) {
      if (lead) umma_commit(bar);
    };
    constexpr uint32_t FMT = BF16 ? FMT_BF16 : FMT_F16;
    const int dn = PAD ? ((p.D + 15) & ~15) : 64;    // columns of the output products, 16 per K step of the score products
    const int ksteps = dn / 16;
    if (warp == 9) {
      const uint32_t idesc_64 = make_idesc(FMT, 128, 64, 0, 0), idesc_128 = make_idesc(FMT, 128, 128, 0, 0);
      auto nt = [&](uint32_t dst, const uint8_t* rtile, const uint8_t* ctile, uint32_t idesc, bool first) {
        const uint64_t da = desc_kmajor_sw128(smem_u32(rtile)), db = desc_kmajor_sw128(smem_u32(ctile));
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (!PAD || k < ksteps) umma_ss_pred(dst, da + 2 * k, db + 2 * k, idesc, !(first && k == 0), lead);
      };
      auto scores = [&](int t) {
        wait_all(&a_full[t % ST], (t / ST) & 1, 20);
        tc_fence_after_sync();
        const uint32_t T = tmem + TG + (t & 1) * 128;
        nt(T, sR(0), sA(t % ST), DUAL ? idesc_128 : idesc_64, true);               // [S | R0 c1^T]
        if constexpr (DUAL) nt(T + 64, sR(1), sA(t % ST), idesc_64, false);        // tS += R1 c0^T
        commit(&s_full[t & 1]);
      };
      auto grads = [&](int t) {
        wait_all(&b_full[t % ST], (t / ST) & 1, 21);
        wait_all(&s_free[t & 1], (t >> 1) & 1, 25);
        tc_fence_after_sync();
        const uint32_t T = tmem + TG + (t & 1) * 128;
        const uint8_t* c = sB(t % ST);
        if constexpr (!DUAL) {
          nt(T + OX, sR(2), c, idesc_64, true);                                      // X
        } else {
          nt(T, sR(QF ? 3 : 2), c, idesc_128, true);                                 // Q: [A | gtO tV^T], KV: [V gO^T | A^T]
          commit(&a_ready[t & 1]);
          if constexpr (QF) nt(T + OX, sR(2), c, idesc_64, false);                   // X += gO V^T
          else nt(T + OX, sR(3), c + C::HALF, idesc_64, false);                      // X^T += tV gtO^T
        }
        commit(&x_full[t & 1]);
      };
      wait_all(&r01_full, 0, 22);
      int j = next_active(j_begin), t = 0;
      if (j < j_end) scores(0);
      // the iteration of tile t issues the scores of tile t + 1 first if they are the first ones of their warpgroup
      for (; j < j_end; ++t) {
        j = next_active(j + 1);
        if (t == 0 && j < j_end) scores(1);
        if (t == 0) wait_all(&r23_full, 0, 37);
        grads(t);
        if (t >= 1 && j < j_end) {
          wait_all(&o_done[(t - 1) & 1], ((t - 1) >> 1) & 1, 27);   // the outputs that read this warpgroup's columns
          scores(t + 1);
        }
      }
    } else {
      const uint32_t idesc_out = make_idesc(FMT, 128, dn, 0, 1);
      // acc[128 x D] (+)= E[128 x 64] (TMEM: 8 columns per K step, 16 apart) * c[64 x D]
      auto out = [&](uint32_t acc, uint32_t e, const uint8_t* c, bool first) {
        const uint64_t db = desc_mnmajor_sw128(smem_u32(c), C::HALF);
#pragma unroll
        for (int k = 0; k < 4; ++k) umma_ts_pred(acc, e + 16 * k, db + static_cast<uint64_t>((k * 2048) >> 4), idesc_out, !(first && k == 0), lead);
      };
      int j = next_active(j_begin), t = 0;
      for (; j < j_end; ++t) {
        j = next_active(j + 1);
        const int st = t % ST, g = t & 1;
        const uint32_t T = tmem + TG + g * 128;
        const bool first = t == 0;
        if constexpr (DUAL) {
          wait_all(&e1_full[g], (t >> 1) & 1, 28);
          tc_fence_after_sync();
          out(tmem, T + OA, sA(st) + C::HALF, first);                               // dtS c1
          out(tmem + 64, T + OA, sA(st), first);                                    // dtS c0
          if constexpr (!QF) out(tmem + 128, T + OA + 8, sB(st) + C::HALF, first);  // dV += tP^T gtO
        }
        wait_all(&e0_full[g], (t >> 1) & 1, 26);
        tc_fence_after_sync();
        out(tmem, T + OX, sA(st), !DUAL && first);                                  // dS c0
        if constexpr (!QF) {
          out(tmem + 128, T + OX + 8, sB(st), !DUAL && first);                      // dV += P^T gO
          if constexpr (DUAL) out(tmem + 192, T + OX + 8, sB(st) + C::HALF, first); // dtV += P^T gtO
        }
        commit(&empty[st]);
        commit(&o_done[g]);
      }
      if (lead) {
        if (t > 0) umma_commit(&acc_final);
        else mbar_arrive(&acc_final);
      }
    }
    __syncwarp();
  }
  } else {
    // ------------------------------------------------------------------ element-wise + epilogue
    asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
    const int g = warp >> 2;
    const int r = (warp & 3) * 32 + lane, gr = r0 + r, gr_c = min(gr, N - 1);
    const size_t row_base = static_cast<size_t>(bh) * N;
    const uint32_t lane_off = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t T = tmem + TG + g * 128 + lane_off;
    auto arrive = [&](uint64_t* bar) {    // one arrival per warp
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar);
    };
    float4 nst = make_float4(0.f, 0.f, 0.f, 0.f);   // family Q: negated statistics of this thread's query row
    if constexpr (QF) {
      const float4 s = p.stats[row_base + gr_c];
      nst = make_float4(-s.x, -s.y, -s.z, -s.w);
      if (s.x == -INFINITY) nst.x = -INFINITY;       // fully excluded query: P = 0
    }
    const float2 c1_2 = make_float2(p.c1, p.c1), s_2 = make_float2(p.s, p.s);
    // family KV: the statistics of this warpgroup's next column tile are fetched one of its tiles ahead
    auto fetch_stats = [&](int j) -> float4 {
      float4 sv = make_float4(INFINITY, 0.f, 0.f, 0.f);
      const int i = tid & 127;
      if (!QF && i < 64 && j < j_end && j * 64 + i < N) sv = __ldg(&p.stats[row_base + j * 64 + i]);
      return sv;
    };
    auto mask_of_tile = [&](int j) {
      return QF ? mask_row_of(p.mv, b, h, gr_c, j, j_end) : mask_col_of(p.mv, b, h, j, gr_c, j_end);
    };
    // this warpgroup's tiles: every second active one
    auto next_mine = [&](int j) {
      j = next_active(j);
      return j < j_end ? next_active(j + 1) : j;
    };
    int n = 0;      // tiles of this warpgroup so far
    int j = next_active(j_begin);
    const bool any = j < j_end;
    if (g == 1 && any) j = next_active(j + 1);
    float4 sv_next = fetch_stats(j);
    MaskRow mask_next = mask_of_tile(j);
    for (; j < j_end; ++n) {
      const int c0 = j * 64;
      const MaskRow mask = mask_next;
      const uint32_t par = n & 1;
      float(*st)[64] = stats_s[g][par];
      if constexpr (!QF) {
        const int i = tid & 127;
        if (i < 64) {
          st[0][i] = (sv_next.x == -INFINITY) ? -INFINITY : -sv_next.x;   // fully excluded query: P = 0
          st[1][i] = -sv_next.y;
          st[2][i] = -sv_next.z;
          st[3][i] = -sv_next.w;
        }
        named_bar_sync(3 + g, 128);
      }
      j = next_mine(j + 1);
      sv_next = fetch_stats(j);
      mask_next = mask_of_tile(j);
      // negated statistics of columns 16 c .. 16 c + 15
      auto stats16 = [&](int field, int c, float2 (&v)[8]) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if constexpr (QF) {
            const float x = field == 0 ? nst.x : (field == 1 ? nst.y : (field == 2 ? nst.z : nst.w));
            v[2 * i] = v[2 * i + 1] = make_float2(x, x);
          } else {
            const float4 x = *reinterpret_cast<const float4*>(&st[field][16 * c + 4 * i]);
            v[2 * i] = make_float2(x.x, x.y);
            v[2 * i + 1] = make_float2(x.z, x.w);
          }
        }
      };
      mbar_wait(&s_full[g], par, w, 30);
      tc_fence_after_sync();
      // ---- P and ts of the row (packed fp32x2 arithmetic)
      float2 P2[2][16], ts2[2][16];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        uint32_t a0[32], a1[32];
        tmem_ld_x32(T + 32 * q, a0);
        if constexpr (DUAL) tmem_ld_x32(T + 64 + 32 * q, a1);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          P2[q][i] = make_float2(__uint_as_float(a0[2 * i]), __uint_as_float(a0[2 * i + 1]));
          if constexpr (DUAL) ts2[q][i] = make_float2(__uint_as_float(a1[2 * i]), __uint_as_float(a1[2 * i + 1]));
        }
      }
      tmem_wait_ld();
      arrive(&s_free[g]);       // S, tS are in registers: X, A may take their place
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        float2 nl[8];
        stats16(0, c, nl);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          float2& x = P2[c >> 1][8 * (c & 1) + i];
          x = __ffma2_rn(x, c1_2, nl[i]);
        }
      }
      {
        const bool need_causal = p.causal && (QF ? (c0 + 63 > r0) : (r0 + 127 > c0));
        const bool need_bound = QF && c0 + 64 > N;
        if (mask.mode == 1) {
#pragma unroll
          for (int q = 0; q < 2; ++q) mask_apply_bits(P2[q], mask.bits[q], mask.other);
        } else if (mask.mode == 2) {
          if constexpr (QF) mask_add_row64(P2, p.mv, b, h, gr_c, c0, N);
          else mask_add_col64(P2, p.mv, b, h, c0, gr_c, N);
        }
        if (need_causal || need_bound) {
          // family Q: keys beyond the query or the end of the sequence; family KV: queries before the key
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int last = (need_causal ? min(gr, N - 1) : N - 1) - (c0 + 32 * q), first = gr - (c0 + 32 * q);
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              if (QF ? 2 * i > last : 2 * i < first) P2[q][i].x = -INFINITY;
              if (QF ? 2 * i + 1 > last : 2 * i + 1 < first) P2[q][i].y = -INFINITY;
            }
          }
        }
      }
#pragma unroll
      for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          P2[q][i] = make_float2(fast_exp2(P2[q][i].x), fast_exp2(P2[q][i].y));
          if constexpr (DUAL) ts2[q][i] = __fmul2_rn(ts2[q][i], s_2);
        }
      uint32_t keep_bits[2] = {0xFFFFFFFFu, 0xFFFFFFFFu};
      if constexpr (DROP) {
#pragma unroll
        for (int q = 0; q < 2; ++q)
          keep_bits[q] = QF ? dropout_keep_along_k(p.drop, bh, gr, c0 + 32 * q) : dropout_keep_along_q(p.drop, bh, c0 + 32 * q, gr);
      }
      // a chunk of 16 columns at a time, the next chunk's load in flight
      if constexpr (DUAL) {
        // A -> dtS = P (A - a) (KV: and tP = P (ts - mu)); everything of dS that does not need X stays in ts2
        mbar_wait(&a_ready[g], par, w, 33);
        tc_fence_after_sync();
        uint32_t ar[2][16];
        tmem_ld_x16(T + OA, ar[0]);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          tmem_wait_ld();
          if (c < 3) tmem_ld_x16(T + OA + 16 * (c + 1), ar[(c + 1) & 1]);
          float2 nmu[8], nd[8], na[8];
          stats16(1, c, nmu);
          stats16(2, c, nd);
          stats16(3, c, na);
          uint32_t e[16];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float2 P = P2[c >> 1][8 * (c & 1) + i];
            float2& ts = ts2[c >> 1][8 * (c & 1) + i];
            float2 A = make_float2(__uint_as_float(ar[c & 1][2 * i]), __uint_as_float(ar[c & 1][2 * i + 1]));
            float2 keep = make_float2(1.f, 1.f);
            if constexpr (DROP) {
              keep = dropout_factors(keep_bits[c >> 1], 8 * (c & 1) + i, p.drop.inv_keep);
              A = __fmul2_rn(A, keep);
            }
            if constexpr (!QF) {
              float2 tp = __fmul2_rn(P, __fadd2_rn(ts, nmu[i]));
              if constexpr (DROP) tp = __fmul2_rn(tp, keep);
              e[8 + i] = pack2<BF16>(tp.x, tp.y);
            }
            const float2 d = __fadd2_rn(A, na[i]);                       // A - a
            ts = __ffma2_rn(nmu[i], A, __ffma2_rn(ts, d, nd[i]));        // ts (A - a) - Delta - mu A
            const float2 dts = __fmul2_rn(P, d);
            e[i] = pack2<BF16>(dts.x, dts.y);
          }
          if constexpr (QF) tmem_st_x8(T + OA + 16 * c, reinterpret_cast<uint32_t(&)[8]>(e));
          else tmem_st_x16(T + OA + 16 * c, e);
        }
        tmem_wait_st();
        arrive(&e1_full[g]);
      }
      // X -> dS = P (X + the above) (primal only: P (X - Delta)) (KV: and P)
      mbar_wait(&x_full[g], par, w, 31);
      tc_fence_after_sync();
      {
        uint32_t xr[2][16];
        tmem_ld_x16(T + OX, xr[0]);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          tmem_wait_ld();
          if (c < 3) tmem_ld_x16(T + OX + 16 * (c + 1), xr[(c + 1) & 1]);
          float2 nd[8];
          if constexpr (!DUAL) stats16(2, c, nd);
          uint32_t e[16];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float2 P = P2[c >> 1][8 * (c & 1) + i];
            float2 X = make_float2(__uint_as_float(xr[c & 1][2 * i]), __uint_as_float(xr[c & 1][2 * i + 1]));
            float2 keep = make_float2(1.f, 1.f);
            if constexpr (DROP) {
              keep = dropout_factors(keep_bits[c >> 1], 8 * (c & 1) + i, p.drop.inv_keep);
              X = __fmul2_rn(X, keep);
            }
            const float2 ds = __fmul2_rn(P, __fadd2_rn(X, DUAL ? ts2[c >> 1][8 * (c & 1) + i] : nd[i]));
            e[i] = pack2<BF16>(ds.x, ds.y);
            if constexpr (!QF) {
              const float2 pd = DROP ? __fmul2_rn(P, keep) : P;
              e[8 + i] = pack2<BF16>(pd.x, pd.y);
            }
          }
          if constexpr (QF) tmem_st_x8(T + OX + 16 * c, reinterpret_cast<uint32_t(&)[8]>(e));
          else tmem_st_x16(T + OX + 16 * c, e);
        }
      }
      tmem_wait_st();
      arrive(&e0_full[g]);
    }
    mbar_wait(&acc_final, 0, w, 32);
    tc_fence_after_sync();
    if (!any) {   // nothing was multiplied: the row-side loads may still be in flight
      mbar_wait(&r01_full, 0, w, 36);
      mbar_wait(&r23_full, 0, w, 38);
    }
    // each warpgroup writes half of the columns; the rows go through this warp's patch of the first row-side tile
    uint8_t* patch = sR(0) + warp * (32 * 64);
    const int wrow0 = r0 + (warp & 3) * 32, rows = N - wrow0, cols = p.D - 32 * g;
    const size_t goff = (row_base + wrow0) * p.D + 32 * g;
#pragma unroll
    for (int a = 0; a < (QF ? 2 : 4); ++a) {
      if (!DUAL && (a & 1)) continue;
      void* const o = QF ? (a == 0 ? pp.dq : pp.dtq) : (a == 0 ? p.out0 : a == 1 ? p.out1 : a == 2 ? p.out2 : p.out3);
      const float scale = a < 2 ? p.s : 1.0f;
      uint32_t v[32], q[1][16];
      if (any) {
        tmem_ld_x32(tmem + lane_off + 64 * a + 32 * g, v);
        tmem_wait_ld();
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = 0u;
      }
#pragma unroll
      for (int i = 0; i < 16; ++i) q[0][i] = pack2<BF16>(__uint_as_float(v[2 * i]) * scale, __uint_as_float(v[2 * i + 1]) * scale);
      store_rows_via_smem<1>(patch, q, static_cast<uint16_t*>(o) + goff, p.D, rows, cols, lane);
    }
  }
}

template <bool BF16, bool PAD, bool DUAL, bool DROP>
__global__ void __launch_bounds__(384, 1) bwd64_sm100_kernel(const __grid_constant__ BwdMaps maps, const __grid_constant__ Bwd64Params pp) {
  using C = Bwd64Cfg;
  const BwdKParams& p = pp.k;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 4 * C::TILE_R + C::STAGES * C::STAGE + 2 * 2 * 4 * 64 * 4);
  uint32_t& tmem_base_s = *reinterpret_cast<uint32_t*>(bars + C::NBAR);
  int& poisoned = *reinterpret_cast<int*>(bars + C::NBAR + 1);
  if ((smem_u32(smem) & 1023u) != 0u) {  // the swizzled layouts need this; never observed otherwise
    if (threadIdx.x == 0) atomicCAS(p.status, 0, WAIT_TIMEOUT_BASE + 99);
    return;
  }
  const int warp = threadIdx.x >> 5;
  // block order: the KV blocks of a group of units (the longer ones), then its Q blocks; heavier row tiles first under a
  // causal mask: early key tiles, late query tiles
  const BlockWork work = block_work(blockIdx.x, 2 * p.n_rt, p.n_units, p.unit_group, false);
  const bool qf = work.tile >= p.n_rt;
  const int rt = qf ? (p.causal ? 2 * p.n_rt - 1 - work.tile : work.tile - p.n_rt) : work.tile;
  const WaitCtx w{p.status, &poisoned, p.budget_ns};
  if (threadIdx.x == 0) {
    poisoned = 0;
    constexpr int kPerWarp = 3 + 3 * C::STAGES + 6;    // from here on: s_free, e1_full, e0_full (one arrival per warp), o_done
    for (int i = 0; i < C::NBAR; ++i) mbar_init(&bars[i], i >= kPerWarp && i < kPerWarp + 6 ? 4 : 1);
    fence_mbar_init();
  }
  __syncthreads();
  if (warp == 9) {
    tmem_alloc(&tmem_base_s, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  if (warp != 8) named_bar_sync(2, 352);   // the TMA producer starts loading while TMEM is being allocated
  tc_fence_after_sync();
  const uint32_t tmem = warp == 8 ? 0u : tmem_base_s;
  if (qf) bwd64_body<true, BF16, PAD, DUAL, DROP>(maps, pp, rt, work.unit, smem, tmem, w);
  else bwd64_body<false, BF16, PAD, DUAL, DROP>(maps, pp, rt, work.unit, smem, tmem, w);
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 9) tmem_dealloc(tmem, 512);
}

template <bool BF16, bool PAD, bool DUAL, bool DROP>
int launch_bwd64(const jvpfa_bwd_args& a, int* status, cudaStream_t stream, const LaunchMarks& marks) {
  float4* stats = reinterpret_cast<float4*>(static_cast<uint8_t*>(a.workspace) + kStatusBytes);
  marks.mark(0);
  const int rc = launch_preprocess<BF16>(a, stats, stream);
  if (rc != JVPFA_OK) return rc;
  BwdMaps maps;
  if (!maps.encode(a)) return JVPFA_ERR_LAUNCH;
  Bwd64Params pp{};
  BwdKParams& p = pp.k;
  p.H = a.H; p.N = a.N; p.D = a.D; p.causal = a.causal;
  p.s = a.sm_scale;
  p.c1 = a.sm_scale * 1.4426950408889634f;
  p.mv = make_mask_view(a.mask, a.mask_summary, a.B, a.H, a.N);
  p.stats = stats;
  p.out0 = a.dk; p.out1 = a.dtk; p.out2 = a.dv; p.out3 = a.dtv;
  pp.dq = a.dq; pp.dtq = a.dtq;
  p.status = status;
  p.budget_ns = wait_budget_ns();
  p.drop = make_dropout_params(a.dropout_p, a.dropout_seed);
  p.n_rt = (a.N + 127) / 128;
  p.n_units = a.B * a.H;
  p.unit_group = unit_group_size(p.n_units);
  auto kern = bwd64_sm100_kernel<BF16, PAD, DUAL, DROP>;
  static SmemOptIn opt_in;
  if (!opt_in.set(reinterpret_cast<const void*>(kern), Bwd64Cfg::smem_bytes())) return JVPFA_ERR_LAUNCH;
  marks.mark(1);
  kern<<<2u * p.n_rt * p.n_units, 384, Bwd64Cfg::smem_bytes(), stream>>>(maps, pp);
  for (int i = 2; i < 5; ++i) marks.mark(i);
  return cudaGetLastError() == cudaSuccess ? JVPFA_OK : JVPFA_ERR_LAUNCH;
}

template <bool BF16>
int launch_bwd64_by_mode(const jvpfa_bwd_args& a, int* status, cudaStream_t stream, const LaunchMarks& marks) {
  auto go = [&](auto pad, auto dual) {
    constexpr bool P = decltype(pad)::value, DU = decltype(dual)::value;
    return a.dropout_p > 0.f ? launch_bwd64<BF16, P, DU, true>(a, status, stream, marks) : launch_bwd64<BF16, P, DU, false>(a, status, stream, marks);
  };
  auto by_pad = [&](auto dual) { return a.D == 64 ? go(std::false_type{}, dual) : go(std::true_type{}, dual); };
  return a.tq != nullptr ? by_pad(std::true_type{}) : by_pad(std::false_type{});
}

}  // namespace
}  // namespace jvpfa
