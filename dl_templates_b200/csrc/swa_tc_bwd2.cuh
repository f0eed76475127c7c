// tcgen05 backward kernels for inputs that need no rotation in shared memory: q and k are either
// not rotated at all or are the rotated copies an earlier kernel left behind (NE > 0: the gradients
// are rotated back to the un-rotated tensors in the epilogue).  Geometry (strips, quarters, slots): swa_tc_strip.cuh.
//
//   warp 0        TMA producer: streamed blocks, quarters of the resident side
//   warp 1        SCORE issuer:  S = X_qk Y_qk^T (+ mask), dP = X_v Y_v^T into the block's buffers
//   warp 2        ACCUMULATE issuer: dV += P^T dO, dK += dS^T Q  resp.  dQ += dS K, A operand in tensor memory
//   warp 3        window-mask units and lse / delta of every streamed block
//   warps 4-11    two compute groups, one thread per resident row each, on either half of every block's columns
//   warps 12-15   EPILOGUE, one warp per slot: accumulators -> registers -> inverse rotation -> global
//
// Why two issuers and epilogue warps: one warp that issues every MMA of the kernel runs a dependent scalar instruction
// stream of about 2000 cycles per block (waits, descriptor arithmetic, commits) next to busy compute warps, while the
// tensor pipe needs about 850 cycles for the same block; and an epilogue inside the compute groups idles both of them.
// The order the single issuer gave for free ("the accumulating MMAs of the block that used this buffer last were issued
// before") is one more barrier, s_free, that the accumulate issuer commits and the score issuer waits for.
//
// All waits are bounded by polls, a second or (the producer's) half of one each (umma.cuh).  A warp whose wait gave up leaves its loop; the others run into
// their own limit, unless they have all they wait for.  At the end any of them raises the CTA's flag: what is in flight is given
// time to land, TMEM is freed and the status word records it.
#pragma once

#include "swa_tc_bwd.cuh"
#include "swa_tc_strip.cuh"

namespace swa {
namespace tc {

constexpr int kBwdRecs = kMaskRing + 3;   // block records (swa_tc_strip.cuh); at most three score buffers
// Shared memory for the softmax statistics: dK/dV [record][-lse | -delta][128] of the streamed queries, behind the indicator units;
// dQ [use parity][slot][-lse | -delta][32] of the resident ones, in the place of the fourth of them.  (In 2 KB of their own they cost dQ
// plans of tall windows their block size: 256 x 256, 57 x 31 window, d = 128, 6 slices, blocks of 48 tokens 952 us, of 80 669.)
__host__ __device__ constexpr uint32_t bwd_vec_bytes(bool dkdv) { return dkdv ? kBwdRecs * 1024u : 0u; }
static_assert(kIndicatorUnit >= 2 * 4 * 2 * 32 * sizeof(float), "lse / delta of the dQ kernel");

struct Bwd2Shared {
  uint64_t x_full[2], x_empty[2];
  uint64_t y_full[kMaxStages], y_empty[kMaxStages], rec_ready[kBwdRecs], yx_free[kMaskRing];
  uint64_t sd_full[3], ds_full[3], s_free[3];   // per score buffer: S and dP are there; P / dS are; they have been accumulated
  // per slot: the quarter in it is complete; its dV / its dQ, dK accumulators have been read
  uint64_t acc_full[4], v_free[4], qk_free[4];
  uint64_t xvec_full[2][4];            // dQ: lse / delta of a quarter are written
  uint32_t rec[kBwdRecs];
  ItemStart start;
  uint32_t tmem_base;
  int abort_flag;
};

// NE: width of the inverse rotation of dQ / dK in the epilogue (n_rdim / 8; 0 = none); ONE: heads of at most 64
// (one 64-column chunk per tensor).
template <bool BF16, bool DKDV, int NE, bool ONE>
__global__ void __launch_bounds__(kBwdThreads, 1)
bwd2_kernel(const __grid_constant__ CUtensorMap tm_xqk, const __grid_constant__ CUtensorMap tm_xv,
            const __grid_constant__ CUtensorMap tm_yqk, const __grid_constant__ CUtensorMap tm_yv,
            const __grid_constant__ CUtensorMap tm_oqk, const __grid_constant__ CUtensorMap tm_ov, const __grid_constant__ KParams p,
            const float* lse, const float* delta) {
  using namespace ptx;
  constexpr int R = NE > 0 ? 8 * NE : 8;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);   // an offset: the compiler keeps seeing shared memory
  const Plan& pl = p.pl;
  const int N = pl.N, nxb = pl.nxb, qch = ONE ? 1 : p.qch, vch = ONE ? 1 : p.vch;
  const int nsb = pl.nsb;                                        // score buffers; dP has two, used in turn
  const uint32_t blk_bytes = (uint32_t)N * 128u;               // one 64-wide chunk of a streamed block
  const uint32_t x_bytes = qch * 16384u + vch * 16384u;
  const uint32_t yqk_stage = blk_bytes * qch, yv_stage = blk_bytes * vch;
  const uint32_t ub = unit_bytes(pl);
  uint8_t* x_smem = smem;                                        // nxb buffers of (qk chunks, v chunks)
  uint8_t* stg_smem = x_smem + nxb * x_bytes;                   // output staging, pl.stg chunks per epilogue warp
  uint8_t* yqk_smem = stg_smem + 4 * pl.stg * kStageChunk;
  uint8_t* yv_smem = yqk_smem + pl.stages * yqk_stage;
  uint8_t* yr_smem = yv_smem + pl.stages * yv_stage;            // window mask: row units of the mask ring,
  uint8_t* yc_smem = yr_smem + kMaskRing * ub * (pl.TH >> 3);   // ... column units,
  uint8_t* xx_smem = yc_smem + kMaskRing * ub * (pl.TW >> 3);  // ... indicator units of the resident rows
  constexpr int xx_units = DKDV ? 4 : 3;
  float* vec_smem = reinterpret_cast<float*>(xx_smem + xx_units * kIndicatorUnit);
  Bwd2Shared* sh = reinterpret_cast<Bwd2Shared*>(xx_smem + kIndicatorBytes + bwd_vec_bytes(DKDV));
  uint8_t* row_parts = reinterpret_cast<uint8_t*>(sh) + ((sizeof(Bwd2Shared) + 15) & ~size_t(15));
  // Tensor memory: score buffer b at column N b, the two dP buffers behind them, then the accumulators.  P and dS replace the scores,
  // 16 columns by 16 -- in dK/dV P in the first eight, dS in the others, so that a dP buffer is free once it has been read and the next
  // block but one's dP need not wait for this one's accumulating MMAs.  With a third score buffer, where there is room, neither need
  // its scores (31 x 31 window, d = 128, 4 slices, when it was built: dK/dV, with three, 498 -> 434 us; dQ, with two, 326 -> 309).
  const uint32_t dp0 = nsb * N, acc_qk = dp0 + 2 * N, acc_v = acc_qk + qch * 64;

  const int warp = threadIdx.x >> 5;

  constexpr int n_bars = offsetof(Bwd2Shared, rec) / 8, warps4 = offsetof(Bwd2Shared, ds_full) / 8;   // ds_full: one arrival per compute warp
  for (int i = threadIdx.x; i < n_bars; i += kBwdThreads) mbar_init(reinterpret_cast<uint64_t*>(sh) + i, i >= warps4 && i < warps4 + 3 ? 8 : 1);
  if (threadIdx.x == 0) {
    sh->abort_flag = 0;
    item_start(p, &sh->start);
  }
  fence_barrier_init();
  if (warp == 1) {
    tmem_alloc(&sh->tmem_base, kBwdTmemCols);
    tmem_relinquish();
  }
  build_row_parts<BF16>(row_parts, threadIdx.x, kBwdThreads, p);
  if (threadIdx.x < 128) {
    write_indicator_units<BF16, xx_units>(xx_smem, threadIdx.x, p);
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

  // Registers follow the work: producer / issuer / mask warpgroup 104, compute 120, epilogue 168:
  // (104 + 2 * 120 + 168) * 128 = 64 Ki.
  if (warp >= 4 && warp < 12) {
    setmaxnreg_dec<120>();
    // ------------------------------------------------------------------ P / dS, one thread per resident row and group
    const int lane = threadIdx.x & 31;
    const int g = (warp - 4) >> 2;
    const int quarter = warp & 3;
    const int m = quarter * 32 + lane;
    const uint32_t lane_base = tmem + ((uint32_t)(quarter * 32) << 16);
    const uint64_t c22 = f2_pack(p.scale_log2, p.scale_log2);
    const int ng = N >> 4;
    const int n1 = (ng + 1) >> 1;                  // first half: n1 steps of 16 columns
    int buf = 0, buf_par = 0, rs = 0, rpar = 0;    // score buffer and record of the next block, their barriers' parities
    uint32_t dp = dp0;                             // its dP buffer
    int tn = 0;
    bool second = g != 0;
    float my_nlse = 0.f, my_ndelta = 0.f;          // dQ: of this thread's query
#pragma unroll 1
    while (true) {
      // what does not depend on the scores comes before the wait for them
      trace_ev(p, 2 + g, tn, m == 0, 0 * 16 + rs);
      wait_spin(&sh->rec_ready[rs], rpar);
      const uint32_t rec = sh->rec[rs];
      if (!ok || (rec & kRecEnd)) break;
      // a quarter that takes no part in the block: its rows of P and dS are never read (umma_ts_slots)
      const bool mine = rec >> (kRecAct + quarter) & 1u;
      if (!DKDV && (rec >> (kRecFresh + quarter) & 1u)) {
        const int use = rec >> (kRecUse + quarter) & 1;
        wait_spin(&sh->xvec_full[use][quarter], rec >> (kRecUse2 + quarter) & 1u);
        const float* xv = vec_smem + (use * 4 + quarter) * 64 + lane;
        my_nlse = xv[0];
        my_ndelta = xv[32];
      }
      wait_spin(&sh->sd_full[buf], buf_par);
      if (!ok) break;
      trace_ev(p, 2 + g, tn, m == 0, 1 * 16 + rs);
      if (mine) {
        const uint32_t s_tm = lane_base + buf * N, d_tm = lane_base + dp;
        [[maybe_unused]] const float* vec = vec_smem + rs * 256;
        tc_fence_after();
        // this group's half of the columns, 16 at a time
        const int c_hi = second ? N : 16 * n1;
#pragma unroll 1
        for (int c = second ? 16 * n1 : 0; c < c_hi; c += 16) {
          uint32_t s[16], d[16];
          tmem_ld16(s_tm + c, s);
          tmem_ld16(d_tm + c, d);
          uint32_t w[DKDV ? 16 : 8];
          uint64_t nl[8], ndl[8];                          // -lse, -delta of the columns
#pragma unroll
          for (int h = 0; h < 4; ++h) {
            if constexpr (DKDV) {
              const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(vec + c + 4 * h), b = *reinterpret_cast<const ulonglong2*>(vec + 128 + c + 4 * h);
              nl[2 * h] = a.x; nl[2 * h + 1] = a.y;
              ndl[2 * h] = b.x; ndl[2 * h + 1] = b.y;
            } else {
              nl[2 * h] = nl[2 * h + 1] = f2_pack(my_nlse, my_nlse);
              ndl[2 * h] = ndl[2 * h + 1] = f2_pack(my_ndelta, my_ndelta);
            }
          }
          tmem_wait_ld();
#pragma unroll
          for (int h = 0; h < 8; ++h) {
            const float2 x = f2_unpack(f2_fma(f2_pack(__uint_as_float(s[2 * h]), __uint_as_float(s[2 * h + 1])), c22, nl[h]));
            const float p0 = exp2f(x.x), p1 = exp2f(x.y);
            const uint64_t u = f2_add(f2_pack(__uint_as_float(d[2 * h]), __uint_as_float(d[2 * h + 1])), ndl[h]);
            const float2 ds = f2_unpack(f2_mul(f2_pack(p0, p1), u));
            w[DKDV ? 8 + h : h] = pack2<BF16>(ds.x, ds.y);
            if constexpr (DKDV) w[h] = pack2<BF16>(p0, p1);
          }
          if constexpr (DKDV) tmem_st16(s_tm + c, w);
          else tmem_st8(s_tm + c, w);
        }
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
      }
      if (lane == 0) mbar_arrive(&sh->ds_full[buf]);
      trace_ev(p, 2 + g, tn, m == 0, 2 * 16 + rs);
      second = !second;                            // the groups take turns with the larger half
      dp ^= dp0 ^ (dp0 + N);
      if (++buf == nsb) { buf = 0; buf_par ^= 1; }
      if (++rs == kBwdRecs) { rs = 0; rpar ^= 1; }
    }
  } else if (warp < 4) {
    setmaxnreg_dec<104>();
    if (warp == 0) {
      // ------------------------------------------------------------------ TMA producer
      const LoadArgs f{x_smem, x_bytes, yqk_smem, yv_smem, yqk_stage, yv_stage, blk_bytes, sh->x_full, sh->x_empty,
                       sh->y_full, sh->y_empty, nullptr, nullptr, &sh->start, &tm_xqk, &tm_xv, &tm_yqk, &tm_yv};
      load_warp<ONE, true>(p, f, ok);
    } else if (warp == 1) {
      // ------------------------------------------------------------------ score issuer: S (+ mask) and dP of every block
      const uint32_t fmt = BF16 ? 1u : 0u;
      const uint32_t idesc_s = instr_desc(fmt, 128, N, 0, 0);                 // both operands K-major
      const uint32_t hi_sw = smem_desc_hi(1024, true), hi_ns = smem_desc_hi(kUnitSbo, false);
      const uint64_t x_desc0 = smem_desc_from(smem_u32(x_smem), 16, hi_sw),
                     yqk_desc0 = smem_desc_from(smem_u32(yqk_smem), 16, hi_sw), yv_desc0 = smem_desc_from(smem_u32(yv_smem), 16, hi_sw),
                     xx_desc0 = smem_desc_from(smem_u32(xx_smem), kIndicatorUnit, hi_ns);
      const uint32_t yqk16 = yqk_stage >> 4, yv16 = yv_stage >> 4, blk16 = blk_bytes >> 4, x16 = x_bytes >> 4;
      const uint32_t yr0 = smem_u32(yr_smem), yc0 = smem_u32(yc_smem);
      [[maybe_unused]] const uint32_t yz0 = smem_u32(xx_smem);
      int stage = 0, stage_par = 0, buf = 0, buf_par = 1, xb = nxb - 1, x_par = 1;   // resident buffer in use; parity of its "full" phase
      int rbuf = 0, rbuf_par = 0, started = 0;   // score buffer of the block that read this block's dP buffer last; blocks so far, up to 2
      uint32_t dp = dp0;
      int mslot = 0, rs = 0, rpar = 0;
      const int stages = pl.stages;
      // units of a ring entry: 0 and 1 of the first step, 2 and (unused) 3 of the second (dQ: 1 and 2), from where and how far to the next entry
      const uint32_t row_step = ub * (pl.TH >> 3), col_step = ub * (pl.TW >> 3);
      const bool tw8 = pl.TW == 8;
      const uint32_t el = elect_one();
      int tn = 0;
      const bool tl = (threadIdx.x & 31) == 0;
#pragma unroll 1
      while (true) {
        trace_ev(p, 1, tn, tl, 2 * 16 + rs);
        wait_spin(&sh->rec_ready[rs], rpar);         // the block's mask units (and lse / delta) are written
        const uint32_t rec = sh->rec[rs];
        if (!ok || (rec & kRecEnd)) break;
        if (rec & kRecEnters) {                      // a quarter enters: the next version of the resident rows
          if (++xb == nxb) { xb = 0; x_par ^= 1; }
          wait_spin(&sh->x_full[xb], x_par);
        }
        wait_spin(&sh->y_full[stage], stage_par);    // the block has landed
        // the dP buffer is free once the compute groups are done with the block but one before
        if (started == 2) {
          wait_spin(&sh->ds_full[rbuf], rbuf_par);
          if (++rbuf == nsb) { rbuf = 0; rbuf_par ^= 1; }
        } else {
          ++started;
        }
        if (!ok) break;
        tc_fence_after();
        const uint32_t s_tm = tmem + buf * N, d_tm = tmem + dp;
        const uint64_t xd = x_desc0 + (uint64_t)(xb * x16), yd = yqk_desc0 + (uint64_t)(stage * yqk16);
        const uint64_t xv = xd + (uint64_t)(qch * 1024), yv = yv_desc0 + (uint64_t)(stage * yv16);   // the v chunks
#pragma unroll
        for (int k = 0; k < 4; ++k) umma_ss_el(el, d_tm, xv + 2 * k, yv + 2 * k, idesc_s, k ? 1u : 0u);
        if (vch > 1) {
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_ss_el(el, d_tm, xv + 1024 + 2 * k, yv + blk16 + 2 * k, idesc_s, 1u);
        }
        // the score buffer is free once the accumulating MMAs of the block that used it last have completed
        wait_spin(&sh->s_free[buf], buf_par);
        if (!ok) break;
        tc_fence_after();
        // window mask, indicator x penalty: row units, column units, the unused unit
        const uint32_t yc = yc0 + mslot * col_step;
        const uint32_t u0 = yr0 + mslot * row_step, u1 = tw8 ? u0 + ub : yc, u2 = tw8 ? yc : yc + ub;
        umma_ss_el(el, s_tm, xx_desc0, smem_desc_from(u0, u1 - u0, hi_ns), idesc_s, 0u);
        if constexpr (DKDV) umma_ss_el(el, s_tm, xx_desc0 + 256, smem_desc_from(u2, yz0 - u2, hi_ns), idesc_s, 1u);
        else umma_ss_el(el, s_tm, xx_desc0 + 128, smem_desc_from(u1, u2 - u1, hi_ns), idesc_s, 1u);
#pragma unroll
        for (int k = 0; k < 4; ++k) umma_ss_el(el, s_tm, xd + 2 * k, yd + 2 * k, idesc_s, 1u);
        if (qch > 1) {
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_ss_el(el, s_tm, xd + 1024 + 2 * k, yd + blk16 + 2 * k, idesc_s, 1u);
        }
        umma_commit_el(el, &sh->sd_full[buf]);
        umma_commit_el(el, &sh->yx_free[mslot]);                     // its mask units may be overwritten
        if (rec & kRecLeaves) umma_commit_el(el, &sh->x_empty[xb]);   // last read of this version
        trace_ev(p, 1, tn, tl, 3 * 16 + rs);
        dp ^= dp0 ^ (dp0 + N);
        if (++buf == nsb) { buf = 0; buf_par ^= 1; }
        if (++stage == stages) { stage = 0; stage_par ^= 1; }
        if (++mslot == kMaskRing) mslot = 0;
        if (++rs == kBwdRecs) { rs = 0; rpar ^= 1; }
      }
    } else if (warp == 2) {
      // ------------------------------------------------------------------ accumulate issuer: A operands come from tensor memory
      const uint32_t fmt = BF16 ? 1u : 0u;
      const uint32_t idesc_qk = instr_desc(fmt, 128, qch * 64, 0, 1);       // dQ / dK: B = streamed qk tile, MN-major
      const uint32_t idesc_v = instr_desc(fmt, 128, vch * 64, 0, 1);        // dV: B = streamed dO tile, MN-major
      const uint32_t hi_sw = smem_desc_hi(1024, true);
      const uint64_t yqk_mn0 = smem_desc_from(smem_u32(yqk_smem), blk_bytes, hi_sw), yv_mn0 = smem_desc_from(smem_u32(yv_smem), blk_bytes, hi_sw);
      const uint32_t yqk16 = yqk_stage >> 4, yv16 = yv_stage >> 4;
      const int stages = pl.stages;
      const int nks = N >> 4;
      int stage = 0, buf = 0, buf_par = 0, rs = 0, rpar = 0;
      const uint32_t el = elect_one();
      int tn = 0;
      const bool tl = (threadIdx.x & 31) == 0;
#pragma unroll 1
      while (true) {
        trace_ev(p, 6, tn, tl, 0 * 16 + rs);
        wait_spin(&sh->rec_ready[rs], rpar);
        const uint32_t rec = sh->rec[rs];
        if (!ok || (rec & kRecEnd)) break;
        const uint32_t act = rec >> kRecAct & 15u, fresh = rec >> kRecFresh & 15u;
        wait_spin(&sh->ds_full[buf], buf_par);
        trace_ev(p, 6, tn, tl, 3 * 16 + rs);
        // dV += P^T dO and dK += dS^T Q, resp. dQ += dS K
#pragma unroll 1
        for (int t = DKDV ? 0 : 1; t < 2; ++t) {
          // the accumulators' last quarter has been read (heads of at most 64: dV and dK at once; 251.9 -> 245.0 us, dK/dV, 64 slices)
#pragma unroll 1
          for (uint32_t h = ONE && DKDV && t ? 0u : fresh; h; h &= h - 1) {
            const int e = __ffs(h) - 1;
            wait_spin((t ? sh->qk_free : sh->v_free) + e, (rec >> (kRecUse + e) & 1u) ^ 1u);
          }
          if (!ok) break;
          tc_fence_after();
          if (act)
            accumulate_block(el, tmem + (t ? acc_qk : acc_v), tmem + buf * N + (DKDV && t ? 8 : 0),
                             t ? yqk_mn0 + (uint64_t)(stage * yqk16) : yv_mn0 + (uint64_t)(stage * yv16), t ? idesc_qk : idesc_v, nks, 16,
                             act, fresh);
        }
        if (!ok) break;
        umma_commit_el(el, &sh->s_free[buf]);
        umma_commit_el(el, &sh->y_empty[stage]);
#pragma unroll 1
        for (uint32_t h = rec >> kRecEnds & 15u; h; h &= h - 1) umma_commit_el(el, &sh->acc_full[__ffs(h) - 1]);
        trace_ev(p, 6, tn, tl, 1 * 16 + rs);
        if (++stage == stages) stage = 0;
        if (++buf == nsb) { buf = 0; buf_par ^= 1; }
        if (++rs == kBwdRecs) { rs = 0; rpar ^= 1; }
      }
    } else {
      // ------------------------------------------------------------------ window mask, lse / delta
      const MaskArgs f{yr_smem, yc_smem, sh->yx_free, sh->rec, sh->rec_ready, kBwdRecs, vec_smem, lse, delta, row_parts, &sh->start};
      mask_warp<BF16, DKDV>(p, f, ok, wait_park);
    }
  } else {
    setmaxnreg_inc<168>();
    // ------------------------------------------------------------------ epilogue, one warp per slot, one thread per row
    const int slot = warp & 3, lane = threadIdx.x & 31;
    const uint32_t lane_base = tmem + ((uint32_t)(slot * 32) << 16);
    const bool rope_on = NE > 0 && p.rope.idx != nullptr;
    const int own_r = lane >> pl.tw_log, own_c = lane & (pl.TW - 1);
    const int vn = DKDV ? vch : 0, nch = vn + qch;             // 64-column chunks: dV, then dQ / dK
    uint8_t* const stg = stg_smem + slot * pl.stg * kStageChunk;
    const uint32_t row0 = smem_u32(stg) + lane * 128, swz_x = (uint32_t)(lane & 7) << 4;
    // Half m of 64-column chunk c: scaled, rotated back and packed into the staging.  Four groups of 8 columns, g0 paired with
    // g2 and g1 with g3: the rotated dims [0, 4R) are row-angle pairs (i, i + R) in [0, 2R) and column-angle pairs in
    // [2R, 4R), so with R = 32 a half takes two groups of either half of the chunk, with R = 16 its own 32 columns, and R = 8
    // pairs neighbouring groups.
    auto put_half = [&](uint32_t* x, int m, int c, float mul, bool rot, int irow, int icol, uint32_t row) {
      float4 cs[8];
      int pos0 = -1, pos1 = -1;                    // table rows of pairs 0-7 and 8-15 of this half; < 0: not rotated
      if constexpr (NE > 0) {
        if (rot && c < (NE == 4 ? 2 : 1) && (NE > 1 || m == 0)) {
          pos0 = (NE == 4 ? c : NE == 2 ? m : 0) ? icol : irow;
          pos1 = NE == 1 ? icol : pos0;
        }
        const int i0 = NE == 4 ? 16 * m : 0;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int pos = e < 4 ? pos0 : pos1, pair = i0 + (NE == 1 ? 2 * (e & 3) : 2 * e);
          const bool colk = NE == 4 ? c != 0 : NE == 2 ? m != 0 : e >= 4;
          cs[e] = make_float4(1.f, 0.f, 1.f, 0.f);
          if (pos >= 0) {
            cs[e] = *reinterpret_cast<const float4*>((colk ? p.rope.col_cs : p.rope.row_cs) + ((int64_t)pos * R + pair) * 2);
          }
        }
      }
      constexpr int PR = NE == 1 ? 8 : 16;         // distance of a pair in x
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int j0 = NE == 1 ? (e >> 2) * 16 + (e & 3) * 2 : 2 * e;
        const float a0 = __uint_as_float(x[j0]) * mul, b0 = __uint_as_float(x[j0 + PR]) * mul;
        const float a1 = __uint_as_float(x[j0 + 1]) * mul, b1 = __uint_as_float(x[j0 + 1 + PR]) * mul;
        if constexpr (NE > 0) {
          x[j0 >> 1] = pack2<BF16>(a0 * cs[e].x + b0 * cs[e].y, a1 * cs[e].z + b1 * cs[e].w);
          cs[e].x = __uint_as_float(pack2<BF16>(b0 * cs[e].x - a0 * cs[e].y, b1 * cs[e].z - a1 * cs[e].w));
        } else {
          x[j0 >> 1] = pack2<BF16>(a0, a1);
          cs[e].x = __uint_as_float(pack2<BF16>(b0, b1));
        }
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) {                // 16-byte group e of the half
        uint32_t wd[4];
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          const int k = 4 * e + h, col = 2 * k;    // word k = columns col, col + 1 of x
          const bool second = (col / PR) & 1;      // of a pair
          const int pe = NE == 1 ? (col / 16) * 4 + (col % 8) / 2 : (col % 16) / 2;
          wd[h] = second ? __float_as_uint(cs[pe].x) : x[(NE == 1 ? (pe >> 2) * 16 + (pe & 3) * 2 : 2 * pe) >> 1];
        }
        const int g8 = NE == 4 ? (e >> 1) * 4 + 2 * m + (e & 1) : 4 * m + e;   // its place among the chunk's eight
        sts128(row + (((uint32_t)g8 << 4) ^ swz_x), wd[0], wd[1], wd[2], wd[3]);
      }
    };
    int tn = 0;
    int use = 0;                                   // how often the slot has been used
    const int n_mine = sh->start.count;
    QuarterWalk qw(p, sh->start, slot);
    // dQ: -lse and -delta of the slot's next quarter, one ahead of the accumulators
    auto fetch = [&](int u) {
      if (DKDV || !qw.more) return;
      const int tr = qw.s.r0 + qw.i * pl.R4 + own_r, tx = qw.s.x0 + own_c;
      float a = -INFINITY, b = 0.f;
      if (tr < p.t_h && tx < p.Wtok) {
        const int64_t at = ((int64_t)(qw.w.bi * p.H + qw.w.hi) * p.t_h + tr) * p.Wtok + tx;
        a = -lse[at];
        b = -delta[at];
      }
      float* xv = vec_smem + ((u & 1) * 4 + slot) * 64 + lane;
      xv[0] = a;
      xv[32] = b;
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh->xvec_full[u & 1][slot]);
    };
    fetch(0);
#pragma unroll 1
    while (qw.more) {
        const int qr = qw.s.r0 + qw.i * pl.R4, x0 = qw.s.x0, hi = qw.w.hi, bi = qw.w.bi;
        qw.next(p, n_mine, slot);
        fetch(use + 1);
        int irow = -1, icol = -1;
        if constexpr (NE > 0) {
          const int tr = qr + own_r, tx = x0 + own_c;
          if (rope_on && tr < p.t_h && tx < p.Wtok) decode_idx(p.rope.idx[(int64_t)tr * p.Wtok + tx], p.rope.max_h, p.rope.max_w, irow, icol);
        }
        trace_ev(p, 5, tn, slot == 0 && lane == 0, 0 * 16 + (use & 15));
        wait_park(&sh->acc_full[slot], use & 1);
        ++use;
        trace_ev(p, 5, tn, slot == 0 && lane == 0, 1 * 16 + (use & 15));
        if (!ok) break;
        tc_fence_after();
        if constexpr (ONE) {
          // Heads of at most 64: the accumulators are read at once and handed on before anything else is done with them --
          // where quarters follow each other block by block, the next block's MMAs wait for that.
          uint32_t a[DKDV ? 64 : 1], x[64];
          if constexpr (DKDV) {
            tmem_ld32(lane_base + acc_v, a);
            tmem_ld32(lane_base + acc_v + 32, a + 32);
          }
          tmem_ld32(lane_base + acc_qk, x);
          tmem_ld32(lane_base + acc_qk + 32, x + 32);
          tmem_wait_ld();
          tc_fence_before();
          if (lane == 0) tma_store_wait_read();          // the previous quarter's rows have left the staging
          __syncwarp();
          if (lane == 0) {
            if constexpr (DKDV) mbar_arrive(&sh->v_free[slot]);
            mbar_arrive(&sh->qk_free[slot]);
          }
          trace_ev(p, 5, tn, slot == 0 && lane == 0, 2 * 16 + (use & 15));
          if constexpr (DKDV) {
#pragma unroll
            for (int u = 0; u < 8; ++u) {
              uint32_t wd[4];
#pragma unroll
              for (int e = 0; e < 4; ++e) wd[e] = pack2<BF16>(__uint_as_float(a[8 * u + 2 * e]), __uint_as_float(a[8 * u + 2 * e + 1]));
              sts128(row0 + (((uint32_t)u << 4) ^ swz_x), wd[0], wd[1], wd[2], wd[3]);
            }
          }
          const uint32_t row = row0 + (DKDV ? kStageChunk : 0u);
          put_half(x, 0, 0, p.sm_scale, rope_on, irow, icol, row);
          put_half(x + 32, 1, 0, p.sm_scale, rope_on, irow, icol, row);
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            if constexpr (DKDV) tma_store_5d(&tm_ov, stg, 0, x0, qr, hi, bi);
            tma_store_5d(&tm_oqk, stg + (DKDV ? kStageChunk : 0u), 0, x0, qr, hi, bi);
            tma_store_commit();
          }
        } else {
          if (lane == 0) tma_store_wait_read();
          __syncwarp();
          int sc = 0;
#pragma unroll 1
          for (int ch = 0; ch < nch; ++ch) {
            const bool is_v = ch < vn;
            const int c = is_v ? ch : ch - vn;
            const uint32_t acc = lane_base + (is_v ? acc_v : acc_qk) + 64 * c;
#pragma unroll 1
            for (int m = 0; m < 2; ++m) {
              uint32_t x[32];
              if constexpr (NE == 4) {
                tmem_ld16(acc + 16 * m, x);
                tmem_ld16(acc + 32 + 16 * m, x + 16);
              } else {
                tmem_ld32(acc + 32 * m, x);
              }
              tmem_wait_ld();
              if (m == 1 && (ch == vn - 1 || ch == nch - 1)) {   // the last column of dV / of dQ, dK has been read
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(is_v ? &sh->v_free[slot] : &sh->qk_free[slot]);
              }
              put_half(x, m, c, is_v ? 1.f : p.sm_scale, rope_on && !is_v, irow, icol, row0 + sc * kStageChunk);
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              tma_store_5d(is_v ? &tm_ov : &tm_oqk, stg + sc * kStageChunk, 64 * c, x0, qr, hi, bi);
              tma_store_commit();
            }
            if (++sc == pl.stg && ch + 1 < nch) {
              sc = 0;
              if (lane == 0) tma_store_wait_read();
              __syncwarp();
            }
          }
        }
        trace_ev(p, 5, tn, slot == 0 && lane == 0, 3 * 16 + (use & 15));
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
    if (threadIdx.x == 0) report_abort(p.status, DKDV ? 5 : 4, 0);
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, kBwdTmemCols);
  }
}

}  // namespace tc
}  // namespace swa
