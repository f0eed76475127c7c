// Geometry of the kernels that rotate no streamed row (swa_tc_fwd2.cuh, swa_tc_bwd2.cuh).
//
// A work item is a CHUNK of a strip: TW token columns wide, nq "quarters" of R4 = 32 / TW grid rows high.  The 128 rows
// of the MMA hold four quarters at a time, one per SLOT (32 tensor-memory lanes, the lanes one warp of a warpgroup may
// touch), and the streamed tokens -- KR grid rows x KW token columns per block -- are walked ONCE per chunk from top to
// bottom.  Quarter i takes part in the blocks [first(i), last(i)] that hold a row of its window; when its last block has
// been accumulated it leaves its slot and quarter i + 4 takes it over, so the resident rows slide down the strip with
// the blocks.  A fixed 128-token tile instead meets every block of its halo with all four quarters although a quarter sees
// little more than half of them (16 x 8 tile, 13 x 13 window: 7 blocks of 80 tokens per 128 rows, 16 of the 28
// quarter-blocks useful); sliding needs 4 blocks per 128 rows, all of them useful, and 4/7 of the loads and MMAs.
// Sliding works while first(i + 4) > last(i) (13 rows of window at TW = 8); the planner checks that, and gives larger
// windows chunks of four quarters, where nothing slides.
//
// Slots are taken in turn by the quarters of the whole stream of items (a running counter modulo 4), so consecutive items
// overlap: the first quarters of the next item are loaded and scored while the last ones of this item are stored.
// Accumulating MMAs write only the lanes of quarters that take part in the block (umma_ts_slots): a quarter that is
// complete rests untouched until it has been read, however late that is, and a new quarter's first MMA overwrites.
//
// What bounds these kernels is how long each role takes for a block, one after the other along the chain of a score buffer --
// score MMAs, tensor memory to registers, exponentials, back, accumulating MMAs -- and beside it: at the 13 x 13 window with d = 64
// a block of 128 rows x 80 columns takes 1500 to 1900 cycles, of which the MMAs need 520 to 930 and the exponentials 640 (16 a
// clock and SM); masking, loading and issuing warps were each busy for most of the rest, as a satisfied wait alone costs 80
// cycles and an MMA issued under a branch twice one issued by a converged warp (umma.cuh).  Hence block records instead of
// six walks over items and quarters, written eight blocks at a time, a load order without polling, and scores of the next blocks
// that wait for as little as possible (swa_tc_bwd2.cuh).  128 x 128 grid, 13 x 13 window, d = 64, 64 slices, bf16: forward / dQ /
// dK/dV 240 / 273 / 318 us before, 204 / 191 / 243 now; 256 x 256, 31 x 31, d = 128, 4 slices: 329 / 366 / 577, 239 / 306 / 439 (CUDA events,
// 1965 MHz, kernels one at a time with pauses).
//
// Backward both compute groups work on every block, each on half of its columns (whole steps of 16; they take turns with
// the larger half): one group walking 80 columns alone took 1.85 ms per dK/dV launch at 256 slices, two sharing them 1.61 (first
// strip kernels).  Forward, with two to four score buffers (two where d_v > 64 and a block has more than 85 columns), the groups
// alternate blocks (0.94 against 1.03 ms).
//
// Rows of the grid: block j of an item covers the rows h0 + band * KR .. with h0 = -wr (mod KR) in every item (chunk heights
// are multiples of KR), so the blocks a row meets, and with them the order of every sum, depend neither on the chunk height
// nor on where in the batch the row lies.
#pragma once

#include "swa_tc_common.cuh"

namespace swa {
namespace tc {

// The work items of a CTA, blockIdx.x, blockIdx.x + gridDim.x, ..., walked by addition: the host gives the steps, one thread
// the start.  (Six roles decomposing every item by division were a third of the kernels' code.)
struct ItemStart {
  int tx, cy, hi, bi, count;
};
struct ItemWalk {
  int tx, cy, hi, bi;
  __device__ __forceinline__ explicit ItemWalk(const ItemStart& s) : tx(s.tx), cy(s.cy), hi(s.hi), bi(s.bi) {}
  __device__ __forceinline__ void next(const KParams& p) {
    tx += p.step_tx;
    cy += p.step_cy;
    hi += p.step_hi;
    bi += p.step_bi;
    if (tx >= p.pl.n_tiles_x) { tx -= p.pl.n_tiles_x; ++cy; }
    if (cy >= p.pl.n_tiles_y) { cy -= p.pl.n_tiles_y; ++hi; }
    if (hi >= p.H) { hi -= p.H; ++bi; }
  }
};
__device__ __forceinline__ void item_start(const KParams& p, ItemStart* s) {
  const int item = blockIdx.x, per_head = p.pl.n_tiles_x * p.pl.n_tiles_y, bh = item / per_head, t = item - bh * per_head;
  s->cy = t / p.pl.n_tiles_x;
  s->tx = t - s->cy * p.pl.n_tiles_x;
  s->bi = bh / p.H;
  s->hi = bh - s->bi * p.H;
  s->count = (p.n_items - item + (int)gridDim.x - 1) / (int)gridDim.x;
}

struct StripItem {
  int r0, x0;        // first resident row, first token column of the strip
  int h0;            // first streamed row (may lie outside the grid: zero-filled and masked)
  int nq, nblk;      // quarters, streamed blocks
  int off;           // r0 - wr - h0
};

__device__ __forceinline__ int div_kr(const Plan& pl, int x) { return (int)(((uint32_t)x * (uint32_t)pl.kr_inv) >> 16); }

__device__ __forceinline__ StripItem strip_item(const KParams& p, const ItemWalk& w) {
  const Plan& pl = p.pl;
  StripItem s;
  s.r0 = w.cy * pl.chunk_rows;
  s.x0 = w.tx << pl.tw_log;
  s.nq = min(pl.nq, (p.t_h - s.r0 + pl.R4 - 1) >> (5 - pl.tw_log));
  s.h0 = s.r0 - p.wr + pl.KR * div_kr(pl, max(0, p.wr - s.r0));
  s.off = s.r0 - p.wr - s.h0;
  const int last = min(s.r0 + s.nq * pl.R4 - 1 + p.wr, p.t_h - 1);
  s.nblk = (div_kr(pl, last - s.h0) + 1) * pl.ncb;
  return s;
}
// First streamed token column of the strip (may lie outside the grid).
__device__ __forceinline__ int strip_hx0(const KParams& p, int x0) {
  const int c = p.div_b ? (int)__umulhi((uint32_t)x0, p.div_b) : x0;
  return (c - p.wc) * p.b;
}

// First and last block of the item that hold a row of quarter i's window.
struct QuarterBlocks {
  int R4, kr_inv, ncb, reach;    // reach: R4 - 1 + 2 wr
  __device__ __forceinline__ explicit QuarterBlocks(const KParams& p)
      : R4(p.pl.R4), kr_inv(p.pl.kr_inv), ncb(p.pl.ncb), reach(p.pl.R4 - 1 + 2 * p.wr) {}
  __device__ __forceinline__ int band(int x) const { return (int)(((uint32_t)x * (uint32_t)kr_inv) >> 16) * ncb; }
  __device__ __forceinline__ int first(const StripItem& s, int i) const { return band(max(i * R4 + s.off, 0)); }
  __device__ __forceinline__ int last(const StripItem& s, int i, int end) const {   // end: the grid's last row, from the first streamed one
    return band(min(i * R4 + s.off + reach, end)) + ncb - 1;
  }
};
__device__ __forceinline__ int quarter_first(const KParams& p, const StripItem& s, int i) { return QuarterBlocks(p).first(s, i); }
__device__ __forceinline__ int quarter_last(const KParams& p, const StripItem& s, int i) { return QuarterBlocks(p).last(s, i, p.t_h - 1 - s.h0); }

// What the roles do with a block is put together once, by the masking warp, in one word: the roles that run block by block are
// loops over these records and know nothing of items and quarters.
// A ring of kMaskRing + (score buffers) records: a record is overwritten once the score MMAs of the block kMaskRing before the
// new one are complete, which needed the buffer, and so the accumulating MMAs, of the block whose record it is.
// Two kRecEnd records follow the last block (the forward kernel's groups read every second one).
enum : uint32_t {
  kRecAct = 0,              // 4 bits each, per slot: its quarter takes part in the block,
  kRecFresh = 4,            // ... starts with it,
  kRecEnds = 8,             // ... is complete with it;
  kRecGroupFirst = 12,      // ... starts with it or the block before (the first for one of two groups on alternate blocks),
  kRecGroupLast = 16,       // ... is complete with it or the next;
  kRecUse = 20,             // bit 0 and
  kRecUse2 = 24,            // ... bit 1 of how often the slot had been used before its quarter
  kRecEnters = 0x10000000u,  // a quarter enters: the next version of the resident rows
  kRecLeaves = 0x20000000u,  // the last block that reads this version
  kRecEnd = 0x40000000u,    // no block: the stream has ended
};

// The quarters of one slot in the order of the stream.
struct QuarterWalk {
  ItemWalk w;
  StripItem s;
  int it, i;                // item, quarter in the item
  uint32_t q0;              // quarters before the item
  bool more;
  __device__ __forceinline__ QuarterWalk(const KParams& p, const ItemStart& st, int slot) : w(st), it(0), i(slot), q0(0), more(true) {
    s = strip_item(p, w);
    settle(p, st.count, slot);
  }
  __device__ __forceinline__ void next(const KParams& p, int count, int slot) {
    i += 4;
    settle(p, count, slot);
  }
  __device__ __forceinline__ void settle(const KParams& p, int count, int slot) {
#pragma unroll 1
    while (i >= s.nq && more) {
      q0 += s.nq;
      more = ++it < count;
      w.next(p);
      s = strip_item(p, w);
      i = (slot - (int)q0) & 3;
    }
  }
};

// ---- window mask --------------------------------------------------------------------------------------------------
// As in swa_tc_common.cuh: the score MMA contracts over 32 more columns, the resident row carries an indicator in the
// column of its ring row (slot * R4 + row in the quarter) and of its token column, a streamed token a penalty in every
// column it may not interact with.  Every 8 of those columns (a "unit", 16 bytes of a row) are a tile of their own,
// rows one after the other (8-row core matrices 128 bytes apart), so that what changes at different times lies apart:
// the row units with the blocks, the column units with the strips.  The fourth unit is unused: the resident rows' is zero, and the
// streamed side is pointed at their units (any finite numbers behind the others in memory).  The dQ kernel has its lse / delta in that
// unit's place and contracts the middle one of the three twice instead, which adds nothing to allowed pairs and one penalty more to
// others.
constexpr uint32_t kUnitSbo = 128;
constexpr uint32_t kIndicatorUnit = 128 * 16, kIndicatorBytes = 4 * kIndicatorUnit;
constexpr int kMaskRing = 4;      // blocks whose units are held; evenly sliding quarters repeat them every four blocks
__device__ __forceinline__ uint32_t unit_bytes(const Plan& pl) { return (uint32_t)pl.N * 16u; }

// Indicator units of the resident rows (128 rows each), the same for every item.
template <bool BF16, int UNITS = 4>
__device__ __forceinline__ void write_indicator_units(uint8_t* xx, int row, const KParams& p) {
  const int hot_r = row >> p.pl.tw_log, hot_c = p.pl.TH + (row & (p.pl.TW - 1));
  const uint16_t one = (uint16_t)(pack2<BF16>(p.mask_a, 0.f) & 0xffffu);
#pragma unroll 1
  for (int e = 0; e < 8 * UNITS; ++e)
    reinterpret_cast<uint16_t*>(xx + (e >> 3) * kIndicatorUnit + row * 16)[e & 7] = (e == hot_r || e == hot_c) ? one : (uint16_t)0;
}

// The row part of a streamed token depends on which quarter holds each slot: it is put together per block from the entries
// of a table, one per distance between the token's row and a quarter's first row.
__host__ __device__ __forceinline__ uint32_t row_parts_bytes(int wr, int R4) {
  return ((uint32_t)(2 * wr + R4 + 1) * R4 * 2u + 15u) & ~15u;
}
template <bool BF16>
__device__ __forceinline__ void build_row_parts(uint8_t* tab, int t, int nthreads, const KParams& p) {
  const uint32_t nb = pack2<BF16>(-p.mask_b, 0.f);
  const int sh = 5 - p.pl.tw_log, n = 2 * p.wr + p.pl.R4;      // entry n: nothing allowed
#pragma unroll 1
  for (int i = t; i < ((n + 1) << sh); i += nthreads) {
    const int d = (i >> sh) - p.wr, rr = i & (p.pl.R4 - 1);      // distance row - first row of the quarter; row in the quarter
    const bool ok = (i >> sh) < n && d - p.wr <= rr && rr <= d + p.wr;
    reinterpret_cast<uint16_t*>(tab)[i] = ok ? (uint16_t)0 : (uint16_t)nb;
  }
}

// ---- accumulating MMAs ------------------------------------------------------------------------------------------------
// D (+)= A B over nks steps of 16 streamed tokens, rows of the quarters that take part (`act`) only; the first step overwrites
// the rows of quarters that start with this block (`fresh`).  A's steps lie `step` columns apart.
__device__ __forceinline__ void accumulate_block(uint32_t el, uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, int nks, uint32_t step,
                                                 uint32_t act, uint32_t fresh) {
  using namespace ptx;
  if (fresh) umma_ts_slots(el, d, a, b, idesc, 0u, SlotMask(fresh));
  if (act & ~fresh) umma_ts_slots(el, d, a, b, idesc, 1u, SlotMask(act & ~fresh));
  const SlotMask m(act);
#pragma unroll 1
  for (int ks = 1; ks < nks; ++ks) {
    a += step;
    b += 128;
    umma_ts_slots(el, d, a, b, idesc, 1u, m);
  }
}

// ---- loads ----------------------------------------------------------------------------------------------------------
// The producer warp fills the ring of streamed blocks and the buffers of resident rows.  A resident buffer holds four quarters;
// it changes when a quarter slides in, so the blocks alternate between nxb buffers ("versions") and a buffer is brought up to
// date -- the slots whose quarter has changed since it was last loaded -- when the score MMAs of its previous version are done.
// With two buffers a quarter crosses L2 twice (it is fetched into L2 one quarter ahead), and its load has one whole block's time
// to arrive.
// Blocks and versions are loaded in one fixed order: the version nxb - 1 after the one that block n starts, right before block
// n + stages - 2.  Its buffer is read last by the score MMAs of block n - 1; the stage of the block loaded before it by the
// accumulating MMAs of block n - 3, which are complete by then, and the stage of the one after it by those of block n - 2: neither
// waits long for the other, and what a wait needs has been loaded before.  (Looking at both rings in turn took 2000 cycles per
// block with the walk that goes with it, more than the other roles needed.)
struct LoadArgs {
  uint8_t* x_smem;              // nxb buffers of qk chunks, then v chunks (128 rows of 128 bytes each)
  uint32_t x_bytes;
  uint8_t *yqk_smem, *yv_smem;  // streamed blocks
  uint32_t yqk_stage, yv_stage, blk_bytes;
  uint64_t *x_full, *x_empty, *y_full, *y_empty;
  uint64_t *yv_full, *yv_empty; // null, or those of the v chunks, which then have a ring of their own
  const ItemStart* start;
  const CUtensorMap *xqk, *xv, *yqk, *yv;   // (the forward kernel has no second resident tensor: XV)
};

template <bool ONE, bool XV>
__device__ __forceinline__ void load_warp(const KParams& p, const LoadArgs& f, bool& ok) {
  using namespace ptx;
  const Plan& pl = p.pl;
  const int count = f.start->count, qch = ONE ? 1 : p.qch, vch = ONE ? 1 : p.vch;
  const int KR = pl.KR, KW = pl.KW, ncb = pl.ncb, stages = pl.stages, nxb = pl.nxb;
  const uint32_t y_bytes = f.yqk_stage + f.yv_stage, yqk_stage = f.yqk_stage, yv_stage = f.yv_stage, blk_bytes = f.blk_bytes,
                 x_bytes = f.x_bytes;
  QuarterBlocks qb(p);
  const uint32_t el = elect_one();
  int tn = 0;
  int stage = 0, stage_par = 1, xb = 0, x_par = 1;
  uint32_t q0 = 0;
  ItemWalk wy(*f.start), wx(*f.start);
  StripItem sy = strip_item(p, wy), sx = sy;
  int jy = 0, yrow = sy.h0, ycol = strip_hx0(p, sy.x0), cblk = 0, ity = 0, ny = 0;   // next streamed block; blocks loaded
  int jx = 0, itx = 0, hi = 0, from = 0, bx = 0;   // block the next version is for, in its item; quarters in so far, and before the last version; blocks before the item
  // a ring of their own: the v chunks are loaded two blocks behind
  const bool split = !ONE && !XV && f.yv_full != nullptr;
  struct At { int col, row, hi, bi; };
  At v1{}, v2{};                                   // the last two blocks
  int vstage = 0, vstage_par = 1;
  auto load_v = [&](const At& b, int st, uint32_t bar) {
    uint32_t to = smem_u32(f.yv_smem) + st * yv_stage;
#pragma unroll 1
    for (int c = 0; c < vch; ++c, to += blk_bytes) tma_load_5d_el(el, to, f.yv, bar, c * 64, b.col, b.row, b.hi, b.bi);
  };
  auto load_behind = [&](const At& b) {
    ok = __all_sync(0xffffffffu, mbar_wait_polls<kSleepPoll>(smem_u32(f.yv_empty + vstage), vstage_par));
    if (!ok) return;
    mbar_expect_tx_el(el, smem_u32(f.yv_full + vstage), yv_stage);
    load_v(b, vstage, smem_u32(f.yv_full + vstage));
    if (++vstage == stages) { vstage = 0; vstage_par ^= 1; }
  };
  int due = 0;                                     // the next version is loaded once so many blocks are
#pragma unroll 1
  while (ity < count || itx < count) {
    if (itx < count && (ny >= due || ity == count)) {
      trace_ev(p, 0, tn, el, 0 * 16 + xb);
      ok = __all_sync(0xffffffffu, mbar_wait_polls<kSleepPoll>(smem_u32(f.x_empty + xb), x_par));
      trace_ev(p, 0, tn, el, 1 * 16 + xb);
      if (!ok) break;
      // The quarters that enter: the first four with the item, the others with the first block that needs them.  This buffer
      // (of two) lacks those that entered with the version before, too.
      int i = nxb == 1 ? hi : from;
      from = hi;
      const int had = bx + jx;                     // block this version is for
#pragma unroll 1
      do {
        ++hi;
        jx = hi < sx.nq ? hi < 4 ? 0 : qb.first(sx, hi) : 1 << 30;
      } while (jx <= had - bx);
      i = max(i, hi - 4);
      const uint32_t dst = smem_u32(f.x_smem + xb * x_bytes), bar = smem_u32(f.x_full + xb);
      mbar_expect_tx_el(el, bar, (uint32_t)(hi - i) * (x_bytes >> 2));
      int row = sx.r0 + i * qb.R4;
#pragma unroll 1
      for (; i < hi; ++i, row += qb.R4) {
        uint32_t to = dst + ((q0 + i) & 3u) * 4096u;
#pragma unroll 1
        for (int c = 0; c < qch; ++c, to += 16384) tma_load_5d_el(el, to, f.xqk, bar, c * 64, sx.x0, row, wx.hi, wx.bi);
        if constexpr (XV) {
#pragma unroll 1
          for (int c = 0; c < vch; ++c, to += 16384) tma_load_5d_el(el, to, f.xv, bar, c * 64, sx.x0, row, wx.hi, wx.bi);
        }
      }
      if (hi < sx.nq) {                            // the next quarter on its way into L2
#pragma unroll 1
        for (int c = 0; c < qch; ++c) tma_prefetch_5d_el(el, f.xqk, c * 64, sx.x0, row, wx.hi, wx.bi);
        if constexpr (XV) {
#pragma unroll 1
          for (int c = 0; c < vch; ++c) tma_prefetch_5d_el(el, f.xv, c * 64, sx.x0, row, wx.hi, wx.bi);
        }
      } else {
        jx = hi = from = 0;
        q0 += sx.nq;
        bx += sx.nblk;
        wx.next(p);
        sx = strip_item(p, wx);
        ++itx;
      }
      if (++xb == nxb) { xb = 0; x_par ^= 1; }
      // (deep rings: one block earlier, since score MMAs then run further ahead of the accumulating ones: 201.9 -> 199.5 us, forward, 64 slices
      // of 128 x 128 x 64; with three stages, 31 x 31 and d = 128, it would cost 3 %)
      due = (nxb == 1 ? bx + jx : had) + stages - (stages >= 6 ? 3 : 2);
    } else {
      trace_ev(p, 0, tn, el, 2 * 16 + stage);
      ok = __all_sync(0xffffffffu, mbar_wait_polls<kSleepPoll>(smem_u32(f.y_empty + stage), stage_par));
      trace_ev(p, 0, tn, el, 3 * 16 + stage);
      if (!ok) break;
      const uint32_t bar = smem_u32(f.y_full + stage);
      mbar_expect_tx_el(el, bar, split ? yqk_stage : y_bytes);
      uint32_t to = smem_u32(f.yqk_smem) + stage * yqk_stage;
#pragma unroll 1
      for (int c = 0; c < qch; ++c, to += blk_bytes) tma_load_5d_el(el, to, f.yqk, bar, c * 64, ycol, yrow, wy.hi, wy.bi);
      const At now{ycol, yrow, wy.hi, wy.bi};
      if (split) {
        if (ny >= 2) load_behind(v2);
        if (!ok) break;
        v2 = v1;
        v1 = now;
      } else {
        load_v(now, stage, bar);
      }
      ++ny;
      if (++stage == stages) { stage = 0; stage_par ^= 1; }
      ycol += KW;
      if (++cblk == ncb) { cblk = 0; ycol -= KW * ncb; yrow += KR; }
      if (++jy == sy.nblk) {
        jy = 0;
        wy.next(p);
        sy = strip_item(p, wy);
        yrow = sy.h0;
        ycol = strip_hx0(p, sy.x0);
        ++ity;
      }
    }
  }
  if (split && ok && ny >= 2) load_behind(v2);
  if (split && ok) load_behind(v1);
}

// ---- the masking warp ---------------------------------------------------------------------------------------------
// One warp writes the record, the mask units (VEC: and -lse / -delta) of every streamed block.  What they are is worked out for eight
// blocks of an item at a time, by four lanes each: block by block the masking warp was busy for nearly the whole time of a block
// and bounded the forward kernel (cells of 16 tokens, head dim 32: 40.8 -> 36.9 us).  A ring entry whose units already
// are what the block needs is left alone: while quarters slide evenly the row units repeat with the period of their ring, and the
// strips that the grid does not clip share their column units.
struct MaskArgs {
  uint8_t *yr_smem, *yc_smem;   // row and column units of every ring entry
  uint64_t* yx_free;
  uint32_t* rec;                // ring of n_rec records
  uint64_t* rec_ready;          // a block's record, mask units and vec slot are written
  int n_rec;
  float* vec_smem;              // VEC: [record][-lse | -delta][128]
  const float *lse, *delta;
  const uint8_t* row_parts;
  const ItemStart* start;
};

// Eight 16-bit penalties (`nb2`: two of them), one for every set bit of the low eight.
__device__ __forceinline__ uint4 penalties(uint32_t bits, uint32_t nb2) {
  uint32_t w[4];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const uint32_t x = (((bits >> (4 * k) & 15u) * 0x00204081u) & 0x01010101u) << 7;      // bit t -> the top bit of byte t, whose sign fills two bytes
    asm("prmt.b32 %0, %1, %1, 0x9988;" : "=r"(w[2 * k]) : "r"(x));
    asm("prmt.b32 %0, %1, %1, 0xbbaa;" : "=r"(w[2 * k + 1]) : "r"(x));
  }
  return make_uint4(w[0] & nb2, w[1] & nb2, w[2] & nb2, w[3] & nb2);
}

template <bool BF16, bool VEC, typename Wait>
__device__ __forceinline__ void mask_warp(const KParams& p, const MaskArgs& f, bool& ok, Wait&& wait) {
  using namespace ptx;
  const Plan& pl = p.pl;
  const int lane = threadIdx.x & 31, slot = lane & 3, N = pl.N;
  const int t_h = p.t_h, Wtok = p.Wtok, wr = p.wr, KR = pl.KR, KW = pl.KW, ncb = pl.ncb;
  const int r4_log = 5 - pl.tw_log;
  const uint32_t nb2 = pack2<BF16>(-p.mask_b, -p.mask_b);
  QuarterBlocks qb(p);
  const uint32_t ub = unit_bytes(pl), row_stage = ub * (uint32_t)(pl.TH >> 3), col_units = ub * (uint32_t)(pl.TW >> 3);
  int jr[4], jc[4], to[4];                         // block row and column of this lane's (up to four) streamed tokens, their offsets
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int n = lane + 32 * e, r = (int)((uint32_t)(n * pl.kw_inv) >> 16);
    jr[e] = n < N ? r : 1 << 30;                   // no such token: below every grid
    jc[e] = n - r * KW;
    to[e] = n < N ? r * Wtok + jc[e] : 0;
  }
  int tn = 0;
  int stage = 0, stage_par = 1, rs = 0;            // ring entries of units and of records
  uint32_t q0 = 0;                                 // quarters before the item
  int old_row = 1 << 31, old_col = -1;             // lane 16 + 4 t + e: what the units of the t'th of the last four blocks are for
  ItemWalk w(*f.start);
  const int count = f.start->count, none = 2 * wr + qb.R4;
  constexpr int kNever = 1 << 30;
#pragma unroll 1
  for (int it = 0; it < count; ++it, w.next(p)) {
    const StripItem s = strip_item(p, w);
    const int hx0 = strip_hx0(p, s.x0), end = t_h - 1 - s.h0;
    const int64_t slice = (int64_t)(w.bi * p.H + w.hi) * t_h * Wtok;
#pragma unroll 1
    for (int j0 = 0; j0 < s.nblk; j0 += 8) {
      // Lane 4 t + e: slot e in the item's block j0 + t.  Its quarter i is the first of the slot that is not over by then.
      const int j = j0 + (lane >> 2), band = ncb == 1 ? j : j / ncb, cblk = j - band * ncb;
      const int over = band * KR - s.off - qb.reach, lo = over <= 0 ? 0 : (over + qb.R4 - 1) >> r4_log;
      const int i = lo + ((slot - (int)q0 - lo) & 3);
      const int first = i < s.nq ? qb.first(s, i) : kNever, last = i < s.nq ? qb.last(s, i, end) : kNever,
                next_first = i + 4 < s.nq ? qb.first(s, i + 4) : kNever;
      // (The first four quarters of an item enter with it.)
      uint32_t rec = (q0 + i & 4u) << (kRecUse - 2) | (q0 + i & 8u) << (kRecUse2 - 3);
      if (first <= j)
        rec |= 1u << kRecAct | (uint32_t)(first == j) << kRecFresh | (uint32_t)(last == j) << kRecEnds |
               (uint32_t)(j - first < 2) << kRecGroupFirst | (uint32_t)(last - j < 2) << kRecGroupLast;
      rec <<= slot;
      if (j == 0 || (i >= 4 && first == j)) rec |= kRecEnters;
      if (j == s.nblk - 1 || (i >= 4 && first == j + 1) || next_first == j + 1) rec |= kRecLeaves;
      rec |= __shfl_xor_sync(0xffffffffu, rec, 1);
      rec |= __shfl_xor_sync(0xffffffffu, rec, 2);
      // Row units: the distance of the block's first row from the quarter (beyond the window: all alike), the rows that the grid
      // cuts off.  Column units: where the block lies relative to the strip, the columns that the grid cuts off.
      const int y0 = s.h0 + band * KR, c0 = hx0 + cblk * KW, at = y0 + wr - (s.r0 + i * qb.R4);
      const int want_row = min(max(at, -KR), none) & 0xffff | max(0, -y0) << 16 | min(KR, max(0, t_h - y0)) << 24;
      const int want_col = (c0 - s.x0) << 20 | cblk << 16 | min(max(0, -c0), 255) << 8 | min(max(0, Wtok - c0), 255);
      const int row4 = __shfl_sync(0xffffffffu, want_row, lane & 15), col4 = __shfl_sync(0xffffffffu, want_col, lane & 15);
      const int row4o = __shfl_sync(0xffffffffu, old_row, lane | 16), col4o = __shfl_sync(0xffffffffu, old_col, lane | 16);
      uint32_t new_row = __ballot_sync(0xffffffffu, want_row != (lane < 16 ? row4o : row4)),
               new_col = __ballot_sync(0xffffffffu, want_col != (lane < 16 ? col4o : col4));
      const int nb = min(8, s.nblk - j0);
      {
        const int k = nb - 4 + ((lane >> 2) & 3), src = 4 * (k < 0 ? k + 8 : k) + slot;
        const int a = __shfl_sync(0xffffffffu, want_row, src), b = __shfl_sync(0xffffffffu, old_row, src);
        const int c = __shfl_sync(0xffffffffu, want_col, src), d = __shfl_sync(0xffffffffu, old_col, src);
        old_row = k < 0 ? b : a;
        old_col = k < 0 ? d : c;
      }
      [[maybe_unused]] float nl[4], dl[4];
      auto fetch = [&](int t) {                    // lse and delta of block t's tokens
        if constexpr (VEC) {
          const int y = __shfl_sync(0xffffffffu, y0, 4 * t), c = __shfl_sync(0xffffffffu, c0, 4 * t);
          const int64_t tok = slice + (int64_t)y * Wtok + c;
          const float *l0 = f.lse + tok, *d0 = f.delta + tok;
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const bool in = (uint32_t)(y + jr[e]) < (uint32_t)t_h && (uint32_t)(c + jc[e]) < (uint32_t)Wtok;
            nl[e] = ld_if(l0 + to[e], in, INFINITY);
            dl[e] = ld_if(d0 + to[e], in, 0.f);
          }
        }
      };
      fetch(0);
#pragma unroll 1
      for (int t = 0; t < nb; ++t, new_row >>= 4, new_col >>= 4) {
        trace_ev(p, 4, tn, lane == 0, 0 * 16 + rs);
        wait(f.yx_free + stage, stage_par);
        trace_ev(p, 4, tn, lane == 0, 1 * 16 + rs);
        if (!ok) return;
        if (new_col & 15u) {
          const int c = __shfl_sync(0xffffffffu, c0, 4 * t);
          uint8_t* col = f.yc_smem + stage * col_units;
#pragma unroll 1
          for (int n = lane; n < N; n += 32) {
            const int yx = c + n - (int)((uint32_t)(n * pl.kw_inv) >> 16) * KW;
            uint32_t seen = 0u;                            // bit t: tile column t may interact with the token
            if ((uint32_t)yx < (uint32_t)Wtok) {
              const int yc = p.div_b ? (int)__umulhi((uint32_t)yx, p.div_b) : yx;
              const int l = min(max((yc - p.wc) * p.b - s.x0, 0), 16), h = min(max((yc + p.wc + 1) * p.b - s.x0, 0), 16);
              seen = (1u << h) - (1u << min(l, h));
            }
#pragma unroll 1
            for (int u = 0; u < (pl.TW >> 3); ++u) *reinterpret_cast<uint4*>(col + u * ub + n * 16) = penalties(~(seen >> (8 * u)), nb2);
          }
          fence_proxy_async_smem();
        }
        if (new_row & 15u) {
          uint8_t* tile = f.yr_smem + stage * row_stage;
          const int y = __shfl_sync(0xffffffffu, y0, 4 * t), at0 = __shfl_sync(0xffffffffu, at, 4 * t), at1 = __shfl_sync(0xffffffffu, at, 4 * t + 1),
                    at2 = __shfl_sync(0xffffffffu, at, 4 * t + 2), at3 = __shfl_sync(0xffffffffu, at, 4 * t + 3);
          // All table entries of this lane's tokens before the first store: token by token this took most of the time of a block where the
          // pattern does not repeat with the ring (15 x 15 window, d = 64, d_v = 128, 32 slices: forward kernel 235 -> 221 us, and with the
          // column units from bits instead of comparisons 213).
          auto entry = [&](int a, int e) {
            const int d = a + jr[e];
            return (uint32_t)(y + jr[e]) < (uint32_t)t_h && (uint32_t)d <= (uint32_t)none ? d : none;
          };
          if (pl.TW == 8) {
            const uint2* u = reinterpret_cast<const uint2*>(f.row_parts);
            // (In dK/dV, whose warp holds lse and delta as well, in two halves: at once its kernels for wide heads spill.  dK/dV, 56 x 56, 7 x 7
            // window, 96 slices 71.4 -> 70.8 us, 45 x 77, 9 x 9, 24 slices 28.2 -> 27.7; d_v = 128 as above, by its registers alone, 305 -> 302.
            // In halves in the forward kernel, 128 x 128, 13 x 13, 64 slices: 204 -> 208.5.)
            const int d4[4] = {at0, at1, at2, at3};
            constexpr int kUnits = VEC ? 1 : 2;
#pragma unroll
            for (int h = 0; h < 2; h += kUnits) {
              uint2 a[kUnits][4], b[kUnits][4];
#pragma unroll
              for (int e = 0; e < 4; ++e)
#pragma unroll
                for (int k = 0; k < kUnits; ++k) {
                  a[k][e] = u[entry(d4[2 * (h + k)], e)];
                  b[k][e] = u[entry(d4[2 * (h + k) + 1], e)];
                }
#pragma unroll
              for (int e = 0; e < 4; ++e)
                if (lane + 32 * e < N)
#pragma unroll
                  for (int k = 0; k < kUnits; ++k)
                    *reinterpret_cast<uint4*>(tile + (h + k) * ub + (lane + 32 * e) * 16) = make_uint4(a[k][e].x, a[k][e].y, b[k][e].x, b[k][e].y);
            }
          } else {
            const uint32_t* u = reinterpret_cast<const uint32_t*>(f.row_parts);
            uint4 a[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) a[e] = make_uint4(u[entry(at0, e)], u[entry(at1, e)], u[entry(at2, e)], u[entry(at3, e)]);
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (lane + 32 * e < N) *reinterpret_cast<uint4*>(tile + (lane + 32 * e) * 16) = a[e];
          }
          fence_proxy_async_smem();
        }
        if constexpr (VEC) {
          float* v = f.vec_smem + rs * 256 + lane;
#pragma unroll
          for (int e = 0; e < 4; ++e) {            // (rows beyond N: written, never read)
            v[32 * e] = -nl[e];
            v[128 + 32 * e] = -dl[e];
          }
        }
        if (lane == 4 * t) f.rec[rs] = rec;
        __syncwarp();
        if (lane == 4 * t) mbar_arrive(f.rec_ready + rs);
        trace_ev(p, 4, tn, lane == 0, 2 * 16 + rs);
        if (++stage == kMaskRing) { stage = 0; stage_par ^= 1; }
        if (++rs == f.n_rec) rs = 0;
        if (t + 1 < nb) fetch(t + 1);
      }
    }
    q0 += s.nq;
  }
#pragma unroll 1
  for (int e = 0; e < 2; ++e) {
    wait(f.yx_free + stage, stage_par);
    if (!ok) return;
    if (lane == 0) {
      f.rec[rs] = kRecEnd;
      mbar_arrive(f.rec_ready + rs);
    }
    if (++stage == kMaskRing) { stage = 0; stage_par ^= 1; }
    if (++rs == f.n_rec) rs = 0;
  }
}

// ---- epilogue staging ---------------------------------------------------------------------------------------------
// A finished quarter leaves the accumulators as 64-column chunks of 32 rows in shared memory (128-byte swizzle) and goes to
// global memory by TMA, which clips the rows and columns beyond the tensor: whole lines are written, the warp does no
// address arithmetic, and the slot is free for the next quarter once the last column has been read.
constexpr uint32_t kStageChunk = 32 * 128;

}  // namespace tc
}  // namespace swa
