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
// What bounds these kernels is the latency of the chain of a buffer pair -- score MMAs, tensor memory to registers,
// exponentials, back, next MMAs -- and, next to it, the exponentials (16 a clock and SM: 640 cycles for 128 rows x 80
// columns; the MMAs of such a block take 530 to 1000).  Backward, with two buffer pairs, both compute groups work on every
// block, each on half of its columns (whole steps of 16; they take turns with the larger half): one group walking 80 columns
// alone took 1.85 ms per dK/dV launch at the 128 x 128 grid with a 13 x 13 window, d = 64 and 256 slices, two sharing
// them 1.61.  Forward, with three or four score buffers, the groups alternate blocks (0.94 against 1.03 ms).
// There the sliding strips run 0.93 / 1.09 / 1.25 ms (forward / dQ / dK/dV) against 1.17 / 1.31 / 2.16 for fixed tiles.
//
// Six roles fetch their code anew for every block: the kernels are kept near 50 KB (at 90 KB, with unrolled polling loops
// and divisions, everything ran at half the speed).
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
__device__ __forceinline__ int quarter_first(const KParams& p, const StripItem& s, int i) {
  return div_kr(p.pl, max(i * p.pl.R4 + s.off, 0)) * p.pl.ncb;
}
__device__ __forceinline__ int quarter_last(const KParams& p, const StripItem& s, int i) {
  return div_kr(p.pl, min(i * p.pl.R4 + s.off + p.pl.R4 - 1 + 2 * p.wr, p.t_h - 1 - s.h0)) * p.pl.ncb + p.pl.ncb - 1;
}

// The quarters that take part in the blocks of an item, block by block (roles that issue MMAs).
struct QuarterCursor {
  int lo, hi;               // quarters lo .. hi - 1 take part
  int next_first, lo_last;  // first block of quarter hi, last block of quarter lo
  uint32_t act;             // slots that take part
  __device__ __forceinline__ void begin(const KParams& p, const StripItem& s) {
    lo = hi = 0;
    act = 0u;
    next_first = 0;
    lo_last = quarter_last(p, s, 0);
  }
};

// ---- window mask --------------------------------------------------------------------------------------------------
// As in swa_tc_common.cuh: the score MMA contracts over 32 more columns, the resident row carries an indicator in the
// column of its ring row (slot * R4 + row in the quarter) and of its token column, a streamed token a penalty in every
// column it may not interact with.  Every 8 of those columns (a "unit", 16 bytes of a row) are a tile of their own,
// rows one after the other (8-row core matrices 128 bytes apart), so that what changes at different times lies apart:
// the row units with the blocks, the column units with the strips, the unused unit never.
constexpr uint32_t kUnitSbo = 128;
constexpr int kMaskRing = 4;      // blocks whose units are held; evenly sliding quarters repeat them every four blocks
__device__ __forceinline__ uint32_t unit_bytes(const Plan& pl) { return (uint32_t)pl.N * 16u; }

// Indicator units of the resident rows (4 x 128 rows), the same for every item.
template <bool BF16>
__device__ __forceinline__ void write_indicator_units(uint8_t* xx, int row, const KParams& p) {
  const int hot_r = row >> p.pl.tw_log, hot_c = p.pl.TH + (row & (p.pl.TW - 1));
  const uint16_t one = (uint16_t)(pack2<BF16>(p.mask_a, 0.f) & 0xffffu);
#pragma unroll 1
  for (int e = 0; e < 32; ++e)
    reinterpret_cast<uint16_t*>(xx + (e >> 3) * 2048 + row * 16)[e & 7] = (e == hot_r || e == hot_c) ? one : (uint16_t)0;
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
// the rows of quarters that start with this block (`fresh`).  From step n1 on A lies `gap` columns further.  One elected thread.
__device__ __forceinline__ void accumulate_block(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, int nks, int n1, uint32_t gap,
                                                 uint32_t act, uint32_t fresh) {
  using namespace ptx;
  const SlotMask m(act);
  if (fresh) {
    umma_ts_slots(d, a, b, idesc, 0u, SlotMask(fresh));
    act &= ~fresh;
  }
  if (act) umma_ts_slots(d, a, b, idesc, 1u, SlotMask(act));
#pragma unroll 1
  for (int ks = 1; ks < nks; ++ks) {
    a += 8;
    b += 128;
    if (ks == n1) a += gap;
    umma_ts_slots(d, a, b, idesc, 1u, m);
  }
}

// ---- loads ----------------------------------------------------------------------------------------------------------
// The producer warp fills the ring of streamed blocks and the buffers of resident rows, whichever has room first.  A
// resident buffer holds four quarters; it changes when a quarter slides in, so the blocks alternate between nxb buffers
// ("versions") and a buffer is brought up to date -- the slots whose quarter has changed since it was last loaded -- as soon as
// the score MMAs of its previous version are done.  With two buffers a quarter crosses L2 twice (it is fetched into L2 one
// quarter ahead), and its load has one whole block's time to arrive.
// Whether a barrier's phase has completed is voted on: two lanes that test it while it completes may see different answers, and
// the walk's state and elect_one must not part ways.
struct LoadArgs {
  uint8_t* x_smem;              // nxb buffers of qk chunks, then v chunks (128 rows of 128 bytes each)
  uint32_t x_bytes, xqk_bytes;
  uint8_t *yqk_smem, *yv_smem;  // streamed blocks
  uint32_t yqk_stage, yv_stage, blk_bytes;
  uint64_t *x_full, *x_empty, *y_full, *y_empty;
  const ItemStart* start;
  const CUtensorMap *xqk, *xv, *yqk, *yv;   // xv: null in the forward kernel (no second resident tensor)
};

constexpr uint32_t kLoadPolls = 1u << 23;   // rounds that found no room in a row: 64 ns or more each, 0.5 s and up

__device__ __forceinline__ void load_warp(const KParams& p, const LoadArgs& f, bool& ok) {
  using namespace ptx;
  const Plan& pl = p.pl;
  const int count = f.start->count;
  int stage = 0, stage_par = 1, xb = 0, x_par = 1;
  bool ring_full = false, x_ring_full = false;
  uint32_t q0 = 0, stale0 = 0, stale1 = 0, m = 0, polls = 0;
  ItemWalk wy(*f.start), wx(*f.start);
  StripItem sy = strip_item(p, wy), sx = sy;
  int jy = 0, yrow = sy.h0, ycol = strip_hx0(p, sy.x0), cblk = 0, ity = 0;   // next streamed block
  int jx = 0, itx = 0, hi = 0;                                               // block the next version is for; quarters in so far
#pragma unroll 1
  while (ok && (ity < count || itx < count)) {
    bool idle = true;
    if (ity < count && (!ring_full || __all_sync(0xffffffffu, mbar_test(smem_u32(f.y_empty + stage), stage_par)))) {
      idle = false;
      if (elect_one()) {
        uint64_t* bar = f.y_full + stage;
        mbar_arrive_expect_tx(bar, f.yqk_stage + f.yv_stage);
#pragma unroll 1
        for (int c = 0; c < p.qch; ++c) tma_load_5d(f.yqk_smem + stage * f.yqk_stage + c * f.blk_bytes, f.yqk, bar, c * 64, ycol, yrow, wy.hi, wy.bi);
#pragma unroll 1
        for (int c = 0; c < p.vch; ++c) tma_load_5d(f.yv_smem + stage * f.yv_stage + c * f.blk_bytes, f.yv, bar, c * 64, ycol, yrow, wy.hi, wy.bi);
      }
      __syncwarp();
      if (++stage == pl.stages) { stage = 0; stage_par ^= 1; ring_full = true; }
      ycol += pl.KW;
      if (++cblk == pl.ncb) { cblk = 0; ycol -= pl.KW * pl.ncb; yrow += pl.KR; }
      if (++jy == sy.nblk) {
        jy = 0;
        wy.next(p);
        sy = strip_item(p, wy);
        yrow = sy.h0;
        ycol = strip_hx0(p, sy.x0);
        ++ity;
      }
    }
    if (itx < count && (!x_ring_full || __all_sync(0xffffffffu, mbar_test(smem_u32(f.x_empty + xb), x_par)))) {
      idle = false;
      if (jx == 0) stale0 = stale1 = 0;
      // the quarters that enter: the first four with the item, the others with the first block that needs them
      int lo = hi;
      m = 0;
#pragma unroll 1
      do m |= 1u << ((q0 + hi++) & 3u);
      while (hi < sx.nq && (hi < 4 || quarter_first(p, sx, hi) <= jx));
      stale0 |= m;
      stale1 |= m;
      m = xb ? stale1 : stale0;
      if (xb) stale1 = 0; else stale0 = 0;
      if (elect_one()) {
        uint8_t* dst = f.x_smem + xb * f.x_bytes;
        uint64_t* bar = f.x_full + xb;
        mbar_arrive_expect_tx(bar, __popc(m) * (f.x_bytes >> 2));
        lo = max(hi - 4, 0);                       // a slot of m holds one of the last four quarters
#pragma unroll 1
        for (int i = lo; i < hi; ++i) {
          const int e = (q0 + i) & 3, row = sx.r0 + i * pl.R4;
          if (!(m >> e & 1u)) continue;
#pragma unroll 1
          for (int c = 0; c < p.qch; ++c) tma_load_5d(dst + c * 16384 + e * 4096, f.xqk, bar, c * 64, sx.x0, row, wx.hi, wx.bi);
          if (f.xv != nullptr) {
#pragma unroll 1
            for (int c = 0; c < p.vch; ++c) tma_load_5d(dst + f.xqk_bytes + c * 16384 + e * 4096, f.xv, bar, c * 64, sx.x0, row, wx.hi, wx.bi);
          }
        }
        if (hi < sx.nq) {                          // the next quarter on its way into L2
          const int row = sx.r0 + hi * pl.R4;
#pragma unroll 1
          for (int c = 0; c < p.qch; ++c) tma_prefetch_5d(f.xqk, c * 64, sx.x0, row, wx.hi, wx.bi);
          if (f.xv != nullptr) {
#pragma unroll 1
            for (int c = 0; c < p.vch; ++c) tma_prefetch_5d(f.xv, c * 64, sx.x0, row, wx.hi, wx.bi);
          }
        }
      }
      __syncwarp();
      if (++xb == pl.nxb) { xb = 0; x_par ^= 1; x_ring_full = true; }
      if (hi < sx.nq) {
        jx = quarter_first(p, sx, hi);
      } else {
        jx = 0;
        hi = 0;
        q0 += sx.nq;
        wx.next(p);
        sx = strip_item(p, wx);
        ++itx;
      }
    }
    polls = idle ? polls + 1 : 0;
    if (idle) __nanosleep(32);
    if (polls == kLoadPolls) ok = false;
  }
}

// ---- the masking warp ---------------------------------------------------------------------------------------------
// One warp writes the mask units (VEC: and -lse / delta) of every streamed block.  A ring entry whose units already are what the
// block needs is left alone: while quarters slide evenly the row units repeat with the period of their ring, and the strips
// that the grid does not clip share their column units.
struct MaskArgs {
  uint8_t *yr_smem, *yc_smem;   // row and column units of every ring entry
  uint64_t *yx_free, *y_ready;
  float* vec_smem;              // VEC: [slot][-lse | -delta][128]
  int vslots;
  uint64_t* vec_ready;
  const float *lse, *delta;
  const uint8_t* row_parts;
  const ItemStart* start;
};

template <bool BF16, bool VEC, typename Wait>
__device__ __forceinline__ void mask_warp(const KParams& p, const MaskArgs& f, bool& ok, Wait&& wait) {
  using namespace ptx;
  const Plan& pl = p.pl;
  const int lane = threadIdx.x & 31, N = pl.N;
  const uint32_t ub = unit_bytes(pl), row_stage = ub * (uint32_t)(pl.TH >> 3), col_units = ub * (uint32_t)(pl.TW >> 3);
  int jrc[4];                                      // block column | block row << 8 of this lane's (up to four) streamed tokens
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int n = lane + 32 * e, r = (int)((uint32_t)(n * pl.kw_inv) >> 16);
    jrc[e] = n < N ? r << 8 | (n - r * pl.KW) : 1 << 30;                        // no such token: below every grid
  }
  int stage = 0, stage_par = 1, vslot = 0;
  bool ring_full = false;
  uint32_t q0 = 0;
  int xr = 0;                                      // lane s < 4: first grid row of the quarter in slot s
  uint64_t row_sig = ~0ull;                        // lane l: what the row units of stage l are for
  uint64_t col_sig = ~0ull;                        // ... and its column units
  ItemWalk w(*f.start);
  const int count = f.start->count, none = 2 * p.wr + pl.R4;
#pragma unroll 1
  for (int it = 0; it < count; ++it, w.next(p)) {
    const StripItem s = strip_item(p, w);
    const int hx0 = strip_hx0(p, s.x0);
    int hi = 0, next_first = 0, y0 = s.h0, cblk = 0;
    const int64_t slice = (int64_t)(w.bi * p.H + w.hi) * p.t_h * p.Wtok;
#pragma unroll 1
    for (int j = 0; j < s.nblk; ++j) {
      float nl[4], dl[4];
      if constexpr (VEC) {                         // (used after the wait below, which covers their latency)
        const int c0 = hx0 + cblk * pl.KW;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int y = y0 + (jrc[e] >> 8), c = c0 + (jrc[e] & 255);
          nl[e] = INFINITY;
          dl[e] = 0.f;
          if ((uint32_t)y < (uint32_t)p.t_h && (uint32_t)c < (uint32_t)p.Wtok) {
            const int64_t at = slice + y * p.Wtok + c;
            nl[e] = f.lse[at];
            dl[e] = f.delta[at];
          }
        }
      }
#pragma unroll 1
      while (hi < s.nq && (hi < 4 || next_first <= j)) {       // the first four quarters enter with the item
        if (lane == ((q0 + hi) & 3)) xr = s.r0 + hi * pl.R4;
        next_first = quarter_first(p, s, ++hi);
      }
      if (ring_full) wait(f.yx_free + stage, stage_par);
      if (ok) {
        // Column units: which tile columns a token column may interact with depends on where the block lies relative to the
        // strip, and on what the grid clips.
        const int c0 = hx0 + cblk * pl.KW;
        const uint64_t want_col = (uint64_t)(uint32_t)(c0 - s.x0) << 32 | (uint32_t)cblk << 24 | (uint32_t)min(max(0, -c0), 255) << 12 |
                                  (uint32_t)min(max(0, p.Wtok - c0), 255);
        if (__shfl_sync(0xffffffffu, col_sig, stage) != want_col) {
          if (lane == stage) col_sig = want_col;
          uint8_t* col = f.yc_smem + stage * col_units;
#pragma unroll 1
          for (int n = lane; n < N; n += 32) {
            const int yx = c0 + n - (int)((uint32_t)(n * pl.kw_inv) >> 16) * pl.KW;
            int lo = 1, hi_ = 0;
            if ((uint32_t)yx < (uint32_t)p.Wtok) {
              const int yc = p.div_b ? (int)__umulhi((uint32_t)yx, p.div_b) : yx;
              lo = (yc - p.wc) * p.b - s.x0;                         // allowed tile columns, inclusive
              hi_ = (yc + p.wc + 1) * p.b - s.x0 - 1;
            }
#pragma unroll 1
            for (int u = 0; u < (pl.TW >> 3); ++u)
              *reinterpret_cast<uint4*>(col + u * ub + n * 16) = penalty_unit<BF16>(lo - 8 * u, hi_ - 8 * u, -p.mask_b);
          }
        }
        // distance of the block's first row from every slot's quarter (beyond the window: all alike), rows inside the grid
        uint32_t at0[4], sig = 0;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          at0[e] = (uint32_t)(y0 + p.wr - __shfl_sync(0xffffffffu, xr, e));
          const int d = min(max((int)at0[e], -pl.KR), none);
          sig = sig << 8 | (uint32_t)(d + 16);             // -16 <= d <= 2 * 64 + 4
        }
        const uint32_t clip = (uint32_t)max(0, -y0) << 8 | (uint32_t)min(pl.KR, max(0, p.t_h - y0));
        const uint64_t want = (uint64_t)clip << 32 | sig;
        if (__shfl_sync(0xffffffffu, row_sig, stage) != want) {
          if (lane == stage) row_sig = want;
          uint8_t* tile = f.yr_smem + stage * row_stage;
#pragma unroll 1
          for (int n = lane; n < N; n += 32) {
            const int r = (int)((uint32_t)(n * pl.kw_inv) >> 16);
            const bool in = (uint32_t)(y0 + r) < (uint32_t)p.t_h;
            uint32_t at[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              at[e] = at0[e] + r;
              if (!in || at[e] > (uint32_t)none) at[e] = none;
            }
            if (pl.TW == 8) {
              const uint2* t = reinterpret_cast<const uint2*>(f.row_parts);
              const uint2 a = t[at[0]], b = t[at[1]], c = t[at[2]], d = t[at[3]];
              *reinterpret_cast<uint4*>(tile + n * 16) = make_uint4(a.x, a.y, b.x, b.y);
              *reinterpret_cast<uint4*>(tile + ub + n * 16) = make_uint4(c.x, c.y, d.x, d.y);
            } else {
              const uint32_t* t = reinterpret_cast<const uint32_t*>(f.row_parts);
              *reinterpret_cast<uint4*>(tile + n * 16) = make_uint4(t[at[0]], t[at[1]], t[at[2]], t[at[3]]);
            }
          }
        }
        if constexpr (VEC) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {            // (rows beyond N: written, never read)
            f.vec_smem[vslot * 256 + lane + 32 * e] = -nl[e];
            f.vec_smem[vslot * 256 + 128 + lane + 32 * e] = -dl[e];
          }
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(f.y_ready + stage);
          if constexpr (VEC) mbar_arrive(f.vec_ready + vslot);
        }
      }
      if (++stage == kMaskRing) { stage = 0; stage_par ^= 1; ring_full = true; }
      if (VEC && ++vslot == f.vslots) vslot = 0;
      if (++cblk == pl.ncb) { cblk = 0; y0 += pl.KR; }
    }
    q0 += s.nq;
  }
}

// ---- epilogue staging ---------------------------------------------------------------------------------------------
// A finished quarter leaves the accumulators as 64-column chunks of 32 rows in shared memory (128-byte swizzle) and goes to
// global memory by TMA, which clips the rows and columns beyond the tensor: whole lines are written, the warp does no
// address arithmetic, and the slot is free for the next quarter once the last column has been read.
constexpr uint32_t kStageChunk = 32 * 128;

}  // namespace tc
}  // namespace swa
