// tcgen05 forward kernel for inputs that need no rotation in shared memory: q and k are either not
// rotated at all or are the rotated copies a streaming pass left behind (swa_fwd_rot).  Geometry (strips, quarters,
// slots): swa_tc_strip.cuh.
//
//   warp 0        TMA producer: K / V blocks, quarters of query rows
//   warp 1        SCORE issuer: S = Q K^T (+ the window mask as 32 extra contraction columns)
//   warp 2        PV issuer:    O_g += P V with P read from tensor memory
//   warp 3        window-mask units of every streamed block
//   warps 4-11    two softmax groups on alternate blocks, one thread per query row each, each with its own
//                 running maximum / sum and its own accumulator O_g
//   warps 12-15   EPILOGUE, one warp per slot: the two groups' partial results of a quarter are merged (in an order fixed by
//                 the blocks' positions in the grid), normalised and stored
//
// One warp issuing every MMA ran a dependent scalar instruction stream of about 2000 cycles per block while the
// tensor pipe needs less than half of that, and an epilogue inside the softmax groups idled both at every item
// boundary; hence two issuers (the order a single issuer gave for free becomes the barrier s_free) and epilogue warps.
// Measured and dropped: two threads per query row, each on half of every block's columns with the row maximum
// exchanged through shared memory (the softmax phase of a block halves, but both groups then work on the SAME
// block and the blocks of an item become strictly sequential: 1.47 ms per launch against 1.17 ms); rotating the
// query tile in this kernel as well (about 400 dependent instructions per row on the critical path, 1.1 ms per launch
// at the default workload, against 0.1 ms for a streaming pass over q).
//
// All waits are bounded by polls, a second or (the producer's) half of one each (umma.cuh).  A warp whose wait gave up leaves its loop; the others run into
// their own limit, unless they have all they wait for.  At the end any of them raises the CTA's flag: what is in flight is given
// time to land, TMEM is freed and the status word records it.
#pragma once

#include "swa_tc_fwd.cuh"
#include "swa_tc_strip.cuh"

namespace swa {
namespace tc {

constexpr int kFwdRecs = kMaskRing + 4;   // block records (swa_tc_strip.cuh); at most four score buffers

struct Fwd2Shared {
  uint64_t q_full[2], q_empty[2];
  uint64_t k_full[kMaxStages], k_empty[kMaxStages], v_full[kMaxStages], v_empty[kMaxStages], rec_ready[kFwdRecs], kx_free[kMaskRing];
  uint64_t s_full[4], p_full[4], s_free[4], pv_done[2];
  // Per group and slot: the group's part of the quarter in it is complete / has been read.  Both count only the quarters that the
  // group has a part in -- one that lies in a single block is one group's alone -- and whoever waits for them keeps a parity bit of its own for
  // each and turns it over at every wait.  With a parity from the uses of the slot, uses that the group is not part of go by without a
  // wait, the barrier may be two phases behind at the next one, and the wait passes (tests/test_strip_handover.py walks the plans).
  uint64_t o_full[2][4], o_free[2][4];
  // [quarter parity][slot]: running maximum and sum handed over, per group; read.  The softmax groups run up to nsb blocks ahead of
  // the PV MMAs -- with small windows that is several quarters of a slot -- so a barrier per slot alone could complete twice
  // before the epilogue warp looks.  A group that has no part in a quarter skips a wait for ml_empty too.  The next one is no phase short
  // because the PV MMAs of a quarter that lies in a single block wait for both groups' o_free: the slot's quarter before the skipped
  // one, four blocks or more before the group's present one, has then been accumulated, which the one before it in the
  // ring has been read for.
  uint64_t ml_full[2][4][2], ml_empty[2][4];
  float ml[2][4][2][2][32];             // [quarter parity][slot][group][maximum | sum][row]
  uint32_t rec[kFwdRecs];
  ItemStart start;
  uint32_t tmem_base;
  int abort_flag;
};

// ONE: heads of at most 64 (one 64-column chunk per tensor); OWNP: P has columns of its own behind the scores.
template <bool BF16, bool ONE, bool OWNP>
__global__ void __launch_bounds__(kFwdThreads, 1)
fwd2_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
            const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_o,
            const __grid_constant__ KParams p, const __grid_constant__ View4 o, float* lse) {
  using namespace ptx;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);   // an offset: the compiler keeps seeing shared memory
  const Plan& pl = p.pl;
  const int N = pl.N, qch = ONE ? 1 : p.qch, vch = ONE ? 1 : p.vch;
  const uint32_t blk_bytes = (uint32_t)N * 128u;               // one 64-wide chunk of a streamed block
  const uint32_t q_bytes = qch * 16384u;
  const uint32_t k_stage = blk_bytes * qch, v_stage = blk_bytes * vch;
  const uint32_t o_cols = vch * 64u;                           // TMEM columns of one O accumulator
  const int nsb = pl.nsb;                                        // score buffers = look-ahead of the score MMAs
  // A stage of keys and values is free once the values have been accumulated -- which is also when the score buffer is free that the
  // third block on takes.  Where shared memory holds three stages (wide heads) that block's load would start when its MMAs could: keys and
  // values then have rings of their own, and keys are free once they have been scored (31 x 31 window, d = 128, 4 slices: 292 -> 240 us).
  // Not where the keys are the smaller part (15 x 15, d = 64 and d_v = 128, 32 slices: one ring 236.6 us, two 238.7).
  const bool split = !ONE && qch > 1 && pl.stages <= 3;
  // Score buffer b at column s_stride * b, O_g behind the buffers.  P gets columns of its own behind the scores when tensor
  // memory allows (p_off = N), so that the scores survive until it is certain that they need not be read again; else P is
  // written over them.
  const uint32_t s_stride = pl.s_stride, p_off = OWNP ? N : 0;
  const uint32_t o_base = nsb * s_stride;
  const uint32_t ub = unit_bytes(pl);
  uint8_t* q_smem = smem;                                        // two buffers
  uint8_t* stg_smem = q_smem + 2 * q_bytes;                     // output staging, pl.stg chunks per epilogue warp
  uint8_t* k_smem = stg_smem + 4 * pl.stg * kStageChunk;
  uint8_t* v_smem = k_smem + pl.stages * k_stage;
  uint8_t* kr_smem = v_smem + pl.stages * v_stage;              // window mask: row units of the mask ring,
  uint8_t* kc_smem = kr_smem + kMaskRing * ub * (pl.TH >> 3);   // ... column units,
  uint8_t* qx_smem = kc_smem + kMaskRing * ub * (pl.TW >> 3);  // ... indicator units of the query rows
  Fwd2Shared* sh = reinterpret_cast<Fwd2Shared*>(qx_smem + kIndicatorBytes);
  uint8_t* row_parts = reinterpret_cast<uint8_t*>(sh) + ((sizeof(Fwd2Shared) + 15) & ~size_t(15));

  const int warp = threadIdx.x >> 5;

  constexpr int n_bars = offsetof(Fwd2Shared, ml) / 8, warps4 = offsetof(Fwd2Shared, p_full) / 8;   // p_full: one arrival per warp
  for (int i = threadIdx.x; i < n_bars; i += kFwdThreads)
    mbar_init(reinterpret_cast<uint64_t*>(sh) + i, i >= warps4 && i < warps4 + 4 ? 4 : 1);
  if (threadIdx.x == 0) {
    sh->abort_flag = 0;
    item_start(p, &sh->start);
  }
  fence_barrier_init();
  if (warp == 1) {
    tmem_alloc(&sh->tmem_base, kFwdTmemCols);
    tmem_relinquish();
  }
  build_row_parts<BF16>(row_parts, threadIdx.x, kFwdThreads, p);
  if (threadIdx.x < 128) {
    write_indicator_units<BF16>(qx_smem, threadIdx.x, p);
  }
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_enter();                                                   // not before the allocation: a successor on this SM must not be first
  pdl_wait();                                                    // from here on: global memory
  const uint32_t tmem = sh->tmem_base;

  bool ok = true;   // warp-uniform: false once a wait has given up
  auto wait_spin = [&](uint64_t* bar, uint32_t parity) {
    ok &= __all_sync(0xffffffffu, mbar_wait_polls<0>(smem_u32(bar), parity)) != 0;
  };
  auto wait_park = [&](uint64_t* bar, uint32_t parity) {
    ok &= __all_sync(0xffffffffu, mbar_wait_polls<100>(smem_u32(bar), parity)) != 0;
  };
  const int n_mine = sh->start.count;

  // Registers follow the work: producer / issuer / mask warpgroup 104, softmax 120, epilogue 168:
  // (104 + 2 * 120 + 168) * 128 = 64 Ki.
  if (warp >= 4 && warp < 12) {
    setmaxnreg_dec<120>();
    // ------------------------------------------------------------------ softmax, one thread per query row and group
    const int lane = threadIdx.x & 31;
    const int g = (warp - 4) >> 2;                // group: takes the blocks whose stream position has parity g
    const int quarter = warp & 3;                 // TMEM lane quarter this warp may touch
    const int m = quarter * 32 + lane;
    const float none_thresh = -0.5f * p.mask_a * p.mask_b;     // a row maximum below this: every entry masked
    const uint32_t lane_base = tmem + ((uint32_t)(quarter * 32) << 16);
    const uint32_t o_tm = lane_base + o_base + g * o_cols;
    const float c2 = p.scale_log2;
    const int ng = N >> 4;                        // 16-column granules of a row
    uint32_t n_own = 0;                           // blocks this group has done
    int rs = g, rpar = 0;                         // ring entry of this group's next record, its barrier's parity
    int sbuf = g % nsb, spar = 0;                 // score buffer of that block, the same
    int tn = 0;
    float m_used = -INFINITY, l = 0.f;
#pragma unroll 1
    for (;; ++n_own) {
      // what does not depend on the scores comes before the wait for them
      wait_spin(&sh->rec_ready[rs], rpar);
      if (!ok) break;
      const uint32_t rec = sh->rec[rs] >> quarter;
      if (sh->rec[rs] & kRecEnd) break;
      const uint32_t s_tm = lane_base + sbuf * s_stride;
      trace_ev(p, 2 + g, tn, m == 0, 0 * 16 + rs);
      wait_spin(&sh->s_full[sbuf], spar);
      if (!ok) break;
      trace_ev(p, 2 + g, tn, m == 0, 1 * 16 + rs);
      // a quarter that takes no part in the block: its rows of P are never read (umma_ts_slots)
      if (rec >> kRecAct & 1u) {
        const bool first = rec >> kRecGroupFirst & 1u;        // this group's first block of the quarter
        if (first) { m_used = -INFINITY; l = 0.f; }
        tc_fence_after();
        uint32_t r[16];
        float mx = -INFINITY, bl;
        // The row maximum is taken before the exponentials in every block when P overwrites the scores, else only in a group's
        // first block of a quarter: the others use the running maximum and see afterwards whether it still serves: a row
        // whose maximum has grown by more than 2^8 is done again, which is rare.  (A load of 16 columns takes 14 cycles.)
        bool exact = !OWNP || first;
        tmem_ld16(s_tm, r);
        if (exact) {
          float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll 1
          for (int i = 0; i < ng; i += 2) {
            uint32_t t[16];
            if (i + 1 < ng) tmem_ld16(s_tm + 16 * (i + 1), t);
            tmem_wait_ld();
#pragma unroll
            for (int e = 0; e < 8; ++e) mx4[e & 3] = fmaxf(mx4[e & 3], fmaxf(__uint_as_float(r[2 * e]), __uint_as_float(r[2 * e + 1])));
            if (i + 1 < ng) {
              if (i + 2 < ng) tmem_ld16(s_tm + 16 * (i + 2), r);
#pragma unroll
              for (int e = 0; e < 8; ++e) mx4[e & 3] = fmaxf(mx4[e & 3], fmaxf(__uint_as_float(t[2 * e]), __uint_as_float(t[2 * e + 1])));
            }
          }
          mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
          tmem_ld16(s_tm, r);                             // first 16 columns, in flight during the bookkeeping
        }
#pragma unroll 1
        while (true) {
          if (exact) {
            if (mx < none_thresh) mx = -INFINITY;
            // running max with lazy rescale: keep scaling by m_used until the true max exceeds it by 2^8
            bool need = false;
            float m_new = m_used;
            if (mx > m_used) {
              if (m_used == -INFINITY) m_used = mx;       // nothing accumulated yet for this row
              else if ((mx - m_used) * c2 > kRescaleThreshold) { need = true; m_new = mx; }
            }
            if (__any_sync(0xffffffffu, need) && !first) {
              // O_g must be at rest: wait for the PV MMA of this group's previous block, then scale the row
              wait_spin(&sh->pv_done[g], (n_own - 1) & 1);
              if (ok) {
                tc_fence_after();
                const float alpha = need ? exp2f((m_used - m_new) * c2) : 1.f;
                tmem_wait_ld();
#pragma unroll 1
                for (int c = 0; c < (int)o_cols; c += 16) {
                  uint32_t t[16];
                  tmem_ld16(o_tm + c, t);
                  tmem_wait_ld();
#pragma unroll
                  for (int e = 0; e < 16; ++e) t[e] = __float_as_uint(__uint_as_float(t[e]) * alpha);
                  tmem_st16(o_tm + c, t);
                }
                if (need) { m_used = m_new; l *= alpha; }
              }
            }
          }
          const float mc = (m_used == -INFINITY) ? 0.f : m_used * c2;
          const uint64_t c22 = f2_pack(c2, c2), nmc2 = f2_pack(-mc, -mc);
          // P = exp2(S*c - m), its row sum, (OWNP) the row maximum of S*c - m; packed, two columns of P per word
          uint64_t ls[2] = {0ull, 0ull};
          float mx2[2] = {-INFINITY, -INFINITY};
#pragma unroll 1
          for (int i = 0; i < ng; ++i) {
            uint64_t e[8];
            uint32_t w[8];
            tmem_wait_ld();
#pragma unroll
            for (int h = 0; h < 8; ++h) e[h] = f2_fma(f2_pack(__uint_as_float(r[2 * h]), __uint_as_float(r[2 * h + 1])), c22, nmc2);
            if (i + 1 < ng) tmem_ld16(s_tm + 16 * (i + 1), r);
#pragma unroll
            for (int h = 0; h < 8; ++h) {
              const float2 x = f2_unpack(e[h]);
              if constexpr (OWNP) mx2[h & 1] = fmaxf(mx2[h & 1], fmaxf(x.x, x.y));
              const float p0 = exp2f(x.x), p1 = exp2f(x.y);
              ls[h & 1] = f2_add(ls[h & 1], f2_pack(p0, p1));
              w[h] = pack2<BF16>(p0, p1);
            }
            tmem_st8(s_tm + p_off + 8 * i, w);
          }
          const float2 l2 = f2_unpack(f2_add(ls[0], ls[1]));
          bl = l2.x + l2.y;
          if (exact) break;
          // rows whose maximum passes the threshold (or that had none yet) are done again with the true one
          const float emx = fmaxf(mx2[0], mx2[1]);
          const bool again = m_used == -INFINITY ? emx > none_thresh * c2 : emx > kRescaleThreshold;
          if (!__any_sync(0xffffffffu, again)) break;
          mx = again ? (emx + mc) / c2 : m_used;
          exact = true;
          tmem_ld16(s_tm, r);
        }
        l += bl;
        const bool last = rec >> kRecGroupLast & 1u;
        const int qp = rec >> kRecUse & 1u;
        if (last) {                             // hand maximum and sum to the epilogue warp
          wait_spin(&sh->ml_empty[qp][quarter], (rec >> kRecUse2 & 1u) ^ 1u);
          sh->ml[qp][quarter][g][0][lane] = m_used;
          sh->ml[qp][quarter][g][1][lane] = l;
        }
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (last && lane == 0) mbar_arrive(&sh->ml_full[qp][quarter][g]);
      }
      if (lane == 0) mbar_arrive(&sh->p_full[sbuf]);
      trace_ev(p, 2 + g, tn, m == 0, 2 * 16 + rs);
      sbuf += 2;                                  // two positions on in the ring of nsb buffers
      if (sbuf >= nsb) { sbuf -= nsb; spar ^= 1; }
      rs += 2;
      if (rs >= kFwdRecs) { rs -= kFwdRecs; rpar ^= 1; }
    }
  } else if (warp < 4) {
    setmaxnreg_dec<104>();
    if (warp == 0) {
      // ------------------------------------------------------------------ TMA producer
      const LoadArgs f{q_smem, q_bytes, k_smem, v_smem, k_stage, v_stage, blk_bytes, sh->q_full, sh->q_empty,
                       sh->k_full, sh->k_empty, split ? sh->v_full : nullptr, sh->v_empty, &sh->start, &tm_q, nullptr, &tm_k, &tm_v};
      load_warp<ONE, false>(p, f, ok);
    } else if (warp == 1) {
      // ------------------------------------------------------------------ score issuer
      const uint32_t fmt = BF16 ? 1u : 0u;
      const uint32_t idesc_s = instr_desc(fmt, 128, N, 0, 0);
      const uint32_t hi_sw = smem_desc_hi(1024, true), hi_ns = smem_desc_hi(kUnitSbo, false);
      const uint64_t q_desc0 = smem_desc_from(smem_u32(q_smem), 16, hi_sw), k_desc0 = smem_desc_from(smem_u32(k_smem), 16, hi_sw),
                     qx_desc0 = smem_desc_from(smem_u32(qx_smem), kIndicatorUnit, hi_ns);
      const uint32_t k_stage16 = k_stage >> 4, blk16 = blk_bytes >> 4;
      const uint32_t kr0 = smem_u32(kr_smem), kc0 = smem_u32(kc_smem), kz0 = smem_u32(qx_smem);
      int stage = 0, stage_par = 0, buf = 0, buf_par = 1, xb = 1, x_par = 1;   // query buffer in use; parity of its "full" phase
      int mslot = 0, rs = 0, rpar = 0;
      const int stages = pl.stages;
      // units of a ring entry: 0 and 1 of the first step, 2 and (unused) 3 of the second, from where and how far to the next entry
      const uint32_t row_step = ub * (pl.TH >> 3), col_step = ub * (pl.TW >> 3);
      const bool tw8 = pl.TW == 8;
      const uint32_t el = elect_one();
      int tn = 0;
#pragma unroll 1
      while (true) {
        trace_ev(p, 1, tn, (threadIdx.x & 31) == 0, 2 * 16 + rs);
        wait_spin(&sh->rec_ready[rs], rpar);          // the block's window-mask units are written
        const uint32_t rec = sh->rec[rs];
        if (!ok || (rec & kRecEnd)) break;
        if (rec & kRecEnters) {                       // a quarter enters: the next version of the query rows
          xb ^= 1;
          if (xb == 0) x_par ^= 1;
          wait_spin(&sh->q_full[xb], x_par);
        }
        wait_spin(&sh->k_full[stage], stage_par);    // the block has landed
        // the buffer is free once the PV MMA of the block that used it last has completed
        wait_spin(&sh->s_free[buf], buf_par);
        if (!ok) break;
        tc_fence_after();
        const uint32_t sd = tmem + buf * s_stride;
        // window mask, indicator x penalty: row units, column units, the unused unit
        const uint32_t yc = kc0 + mslot * col_step;
        const uint32_t u0 = kr0 + mslot * row_step, u1 = tw8 ? u0 + ub : yc, u2 = tw8 ? yc : yc + ub;
        umma_ss_el(el, sd, qx_desc0, smem_desc_from(u0, u1 - u0, hi_ns), idesc_s, 0u);
        umma_ss_el(el, sd, qx_desc0 + 256, smem_desc_from(u2, kz0 - u2, hi_ns), idesc_s, 1u);
        const uint64_t qd = q_desc0 + (uint64_t)(xb * (q_bytes >> 4)), kd = k_desc0 + (uint64_t)(stage * k_stage16);
#pragma unroll
        for (int k = 0; k < 4; ++k) umma_ss_el(el, sd, qd + 2 * k, kd + 2 * k, idesc_s, 1u);
        if (qch > 1) {
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_ss_el(el, sd, qd + 1024 + 2 * k, kd + blk16 + 2 * k, idesc_s, 1u);
        }
        umma_commit_el(el, &sh->s_full[buf]);
        if (split) umma_commit_el(el, &sh->k_empty[stage]);
        umma_commit_el(el, &sh->kx_free[mslot]);                     // its mask units may be overwritten
        if (rec & kRecLeaves) umma_commit_el(el, &sh->q_empty[xb]);   // last read of this version
        trace_ev(p, 1, tn, (threadIdx.x & 31) == 0, 3 * 16 + rs);
        if (++stage == stages) { stage = 0; stage_par ^= 1; }
        if (++mslot == kMaskRing) mslot = 0;
        if (++buf == nsb) { buf = 0; buf_par ^= 1; }
        if (++rs == kFwdRecs) { rs = 0; rpar ^= 1; }
      }
    } else if (warp == 2) {
      // ------------------------------------------------------------------ PV issuer: O_g += P V, P from tensor memory
      const uint32_t fmt = BF16 ? 1u : 0u;
      const uint32_t idesc_pv = instr_desc(fmt, 128, o_cols, 0, 1);
      const uint32_t hi_sw = smem_desc_hi(1024, true);
      const uint64_t v_desc0 = smem_desc_from(smem_u32(v_smem), blk_bytes, hi_sw);
      const uint32_t v_stage16 = v_stage >> 4;
      const int stages = pl.stages;
      const int nks = N >> 4;
      int stage = 0, stage_par = 0, buf = 0, buf_par = 0, grp = 0, rs = 0, rpar = 0;
      uint32_t free_par = 0xffu;                           // parity of the next wait for o_free, bit 4 * group + slot
      const uint32_t el = elect_one();
      int tn = 0;
#pragma unroll 1
      while (true) {
        trace_ev(p, 6, tn, (threadIdx.x & 31) == 0, 0 * 16 + rs);
        // everything that does not depend on P first: what follows the wait for it is the chain of a score buffer
        wait_spin(&sh->rec_ready[rs], rpar);
        const uint32_t rec = sh->rec[rs];
        if (!ok || (rec & kRecEnd)) break;
        const uint32_t act = rec >> kRecAct & 15u, fresh = act & rec >> kRecGroupFirst;   // first block of these quarters for this group's O_g
        const uint32_t alone = rec >> kRecFresh & rec >> kRecEnds & 15u;    // quarters of this block only: the other group's as well (ml_empty)
#pragma unroll 1
        for (uint32_t h = fresh | alone << 4; h; h &= h - 1) {              // the accumulators' last quarter has been read
          const int e = (__ffs(h) - 1) ^ 4 * grp;
          wait_spin(&sh->o_free[0][e], free_par >> e & 1u);
        }
        free_par ^= fresh << (4 * grp);
        if (split) wait_spin(&sh->v_full[stage], stage_par);
        wait_spin(&sh->p_full[buf], buf_par);
        if (!ok) break;
        trace_ev(p, 6, tn, (threadIdx.x & 31) == 0, 4 * 16 + rs);
        tc_fence_after();
        accumulate_block(el, tmem + o_base + grp * o_cols, tmem + buf * s_stride + p_off, v_desc0 + (uint64_t)(stage * v_stage16), idesc_pv, nks,
                         8, act, fresh);
        umma_commit_el(el, &sh->s_free[buf]);
        umma_commit_el(el, split ? &sh->v_empty[stage] : &sh->k_empty[stage]);
        umma_commit_el(el, &sh->pv_done[grp]);
#pragma unroll 1
        for (uint32_t h = act & rec >> kRecGroupLast; h; h &= h - 1) umma_commit_el(el, &sh->o_full[grp][__ffs(h) - 1]);
        trace_ev(p, 6, tn, (threadIdx.x & 31) == 0, 1 * 16 + rs);
        grp ^= 1;
        if (++stage == stages) { stage = 0; stage_par ^= 1; }
        if (++buf == nsb) { buf = 0; buf_par ^= 1; }
        if (++rs == kFwdRecs) { rs = 0; rpar ^= 1; }
      }
    } else {
      // ------------------------------------------------------------------ window mask
      const MaskArgs f{kr_smem, kc_smem, sh->kx_free, sh->rec, sh->rec_ready, kFwdRecs, nullptr, nullptr, nullptr, row_parts, &sh->start};
      mask_warp<BF16, false>(p, f, ok, wait_park);
    }
  } else {
    setmaxnreg_inc<168>();
    // ------------------------------------------------------------------ epilogue, one warp per slot, one thread per row
    const int slot = warp & 3, lane = threadIdx.x & 31;
    const uint32_t lane_base = tmem + ((uint32_t)(slot * 32) << 16);
    const float c2 = p.scale_log2;
    const int own_r = lane >> pl.tw_log, own_c = lane & (pl.TW - 1);
    uint8_t* const stg = stg_smem + slot * pl.stg * kStageChunk;
    const uint32_t row0 = smem_u32(stg) + lane * 128, swz_x = (uint32_t)(lane & 7) << 4;
    int tn = 0;
    int o_par = 0, ml_par = 0;                      // barrier parities (o: bit per group; ml: per quarter parity and group)
    uint32_t gb = 0, q0 = 0;
    ItemWalk w(sh->start);
#pragma unroll 1
    for (int it = 0; ok && it < n_mine; ++it, w.next(p)) {
      const StripItem si = strip_item(p, w);
#pragma unroll 1
      for (int i = (slot - (int)q0) & 3; i < si.nq; i += 4) {
        // The groups' partial results are merged in the order in which they become complete, which the blocks' positions in the grid
        // decide: the result of a row does not depend on the work that preceded it.  The one that is complete a block earlier is
        // read -- and its accumulator handed on -- then: where quarters follow each other block by block the next block wants it.
        const int qr = si.r0 + i * pl.R4, b_lo = quarter_first(p, si, i), b_hi = quarter_last(p, si, i);
        const int g2 = (int)((gb + (uint32_t)b_hi) & 1u), g1 = g2 ^ 1;      // the group of the last block, the other one
        const bool both = b_hi > b_lo;
        const int qp = (int)((q0 + i) >> 2) & 1;
        float m_1 = -INFINITY, l_1 = 0.f;
        trace_ev(p, 5, tn, slot == 0 && lane == 0, 0 * 16 + (i & 15));
        const uint32_t o_2 = lane_base + o_base + g2 * o_cols, o_1 = lane_base + o_base + (both ? g1 : g2) * o_cols;
        [[maybe_unused]] uint32_t x[ONE ? 64 : 1];
        if (both) {
          wait_park(&sh->ml_full[qp][slot][g1], (ml_par >> (2 * qp + g1)) & 1);
          ml_par ^= 1 << (2 * qp + g1);
          m_1 = sh->ml[qp][slot][g1][0][lane];
          l_1 = sh->ml[qp][slot][g1][1][lane];
          wait_spin(&sh->o_full[g1][slot], o_par >> g1 & 1);
          o_par ^= 1 << g1;
        }
        if (!ok) break;
        tc_fence_after();
        if constexpr (ONE) {
          if (both) {
            tmem_ld32(o_1, x);
            tmem_ld32(o_1 + 32, x + 32);
            tmem_wait_ld();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh->o_free[g1][slot]);
          } else {
#pragma unroll
            for (int e = 0; e < 64; ++e) x[e] = 0u;
          }
        }
        wait_park(&sh->ml_full[qp][slot][g2], (ml_par >> (2 * qp + g2)) & 1);
        ml_par ^= 1 << (2 * qp + g2);
        const float m_2 = sh->ml[qp][slot][g2][0][lane], l_2 = sh->ml[qp][slot][g2][1][lane];
        __syncwarp();
        if (ok && lane == 0) mbar_arrive(&sh->ml_empty[qp][slot]);
        const float mm = fmaxf(m_1, m_2);
        const float w_1 = (m_1 == -INFINITY) ? 0.f : exp2f((m_1 - mm) * c2);
        const float w_2 = (m_2 == -INFINITY) ? 0.f : exp2f((m_2 - mm) * c2);
        const float lt = fmaf(l_2, w_2, l_1 * w_1);
        const float inv = 1.f / lt;
        const float f_1 = w_1 * inv, f_2 = w_2 * inv;
        wait_spin(&sh->o_full[g2][slot], o_par >> g2 & 1);
        o_par ^= 1 << g2;
        if (!ok) break;
        trace_ev(p, 5, tn, slot == 0 && lane == 0, 1 * 16 + (i & 15));
        tc_fence_after();
        // Heads of at most 64 leave through the staging by TMA; wider ones, which need the shared memory for larger blocks, are
        // stored by the threads that hold the rows.
        const int tr = qr + own_r, tx = si.x0 + own_c;
        const bool t_in = tr < p.t_h && tx < p.Wtok;
        const int64_t tok = (int64_t)tr * p.Wtok + tx;
        using T = typename std::conditional<BF16, __nv_bfloat16, __half>::type;
        [[maybe_unused]] T* const orow = (T*)o.ptr + w.bi * o.s0 + w.hi * o.s1 + tok * o.s2;
        if constexpr (ONE) {
          uint32_t y[64];
          tmem_ld32(o_2, y);
          tmem_ld32(o_2 + 32, y + 32);
          tmem_wait_ld();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&sh->o_free[g2][slot]);
          trace_ev(p, 5, tn, slot == 0 && lane == 0, 2 * 16 + (i & 15));
          if (lane == 0) tma_store_wait_read();          // the previous quarter's rows have left the staging
          __syncwarp();
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            uint32_t wd[4];
#pragma unroll
            for (int h = 0; h < 4; ++h) {
              const int e = 8 * u + 2 * h;
              wd[h] = pack2<BF16>(fmaf(__uint_as_float(y[e]), f_2, __uint_as_float(x[e]) * f_1),
                                  fmaf(__uint_as_float(y[e + 1]), f_2, __uint_as_float(x[e + 1]) * f_1));
            }
            sts128(row0 + (((uint32_t)u << 4) ^ swz_x), wd[0], wd[1], wd[2], wd[3]);
          }
        } else {
          // (a group without blocks has weight 0 and an accumulator that may hold anything: the other one is read twice)
#pragma unroll 1
          for (int m = 0; m < 2 * vch; ++m) {              // 32 columns
            uint32_t a[32], b[32];
            tmem_ld32(o_1 + 32 * m, a);
            tmem_ld32(o_2 + 32 * m, b);
            tmem_wait_ld();
            if (m == 2 * vch - 1) {                        // the last column has been read
              tc_fence_before();
              __syncwarp();
              if (lane == g2 || (both && lane == g1)) mbar_arrive(&sh->o_free[lane][slot]);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              uint32_t wd[4];
#pragma unroll
              for (int h = 0; h < 4; ++h) {
                const int e = 8 * u + 2 * h;
                wd[h] = pack2<BF16>(fmaf(__uint_as_float(b[e]), f_2, __uint_as_float(a[e]) * f_1),
                                    fmaf(__uint_as_float(b[e + 1]), f_2, __uint_as_float(a[e + 1]) * f_1));
              }
              if (t_in && 32 * m + 8 * u < p.dv) *reinterpret_cast<uint4*>(orow + 32 * m + 8 * u) = make_uint4(wd[0], wd[1], wd[2], wd[3]);
            }
          }
        }
        if constexpr (ONE) {
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            tma_store_5d(&tm_o, stg, 0, si.x0, qr, w.hi, w.bi);
            tma_store_commit();
          }
        }
        if (t_in) lse[(int64_t)(w.bi * p.H + w.hi) * p.t_h * p.Wtok + tok] = mm * c2 + log2f(lt);
        trace_ev(p, 5, tn, slot == 0 && lane == 0, 3 * 16 + (i & 15));
      }
      gb += si.nblk;
      q0 += si.nq;
    }
    if (lane == 0) tma_store_wait_all();
  }

  // ------------------------------------------------------------------ teardown
  if (!ok) sh->abort_flag = 1;
  tc_fence_before();
  __syncthreads();
  if (*(volatile int*)&sh->abort_flag) {
    // let whatever is still in flight (TMA, MMA) land before shared memory and TMEM are released
#pragma unroll 1
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
    if (threadIdx.x == 0) report_abort(p.status, 6, 0);
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, kFwdTmemCols);
  }
}

}  // namespace tc
}  // namespace swa
