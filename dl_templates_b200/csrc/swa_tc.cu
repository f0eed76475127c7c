// Host side of the tcgen05 kernels: shape qualification, tile planning, TMA tensor
// maps and launches.
#include <cudaTypedefs.h>

#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <tuple>
#include <type_traits>
#include <vector>

#include "swa_tc.cuh"
#include "swa_tc_bwd.cuh"
#include "swa_tc_bwd2.cuh"
#include "swa_tc_fwd.cuh"
#include "swa_tc_fwd2.cuh"

namespace swa {
namespace tc {

namespace {

thread_local char g_tc_err[256] = "";
constexpr uint32_t kSmemLimit = 227 * 1024;

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  });
  return fn;
}

// 5-D map over a [B, H, N, d] tensor seen as (d, token column, grid row, head, batch); box =
// (64 elements, box_cols, box_rows, 1, 1), 128-byte swizzle, zero fill outside the tensor.
bool make_map(CUtensorMap* m, const swa_tensor_t* t, const swa_geom_t* g, int d, int box_cols, int box_rows) {
  auto fn = encode_fn();
  if (!fn) {
    snprintf(g_tc_err, sizeof(g_tc_err), "cuTensorMapEncodeTiled entry point not available");
    return false;
  }
  const uint64_t Wtok = (uint64_t)g->t_width * g->b_size;
  cuuint64_t dims[5] = {(cuuint64_t)d, Wtok, (cuuint64_t)g->t_height, (cuuint64_t)g->H, (cuuint64_t)g->B};
  cuuint64_t strides[4] = {(cuuint64_t)t->stride[2] * 2, (cuuint64_t)t->stride[2] * 2 * Wtok,
                           (cuuint64_t)t->stride[1] * 2, (cuuint64_t)t->stride[0] * 2};
  // a dimension of extent 1 may carry any stride; give it a legal one
  for (int i = 0; i < 4; ++i)
    if (dims[i + 1] == 1 && (strides[i] == 0 || strides[i] % 16)) strides[i] = 16;
  cuuint32_t box[5] = {64u, (cuuint32_t)box_cols, (cuuint32_t)box_rows, 1u, 1u};
  cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  const CUtensorMapDataType dt = g->dtype == SWA_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  CUresult r = fn(m, dt, 5, t->ptr, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    snprintf(g_tc_err, sizeof(g_tc_err), "cuTensorMapEncodeTiled failed (%d)", (int)r);
    return false;
  }
  return true;
}

// Experiment knobs (environment variables), read ONCE per process -- a launch must not pay for a dozen getenv
// calls -- and again only when refresh_env() is called (tests that vary them do).  -1 / 0 = not set.
struct Knobs {
  int nmax, nxb, kr, kw, stages, nsb, th_all, th[3], trace_it;
  bool no_tabs, disable, verbose, trace;
};
std::mutex g_plan_mu;                 // guards the plan cache and the reading of the knobs
std::atomic<const Knobs*> g_knobs{nullptr};      // (a snapshot is never freed: refresh_env is a diagnostic)

int env_raw(const char* name, int dflt) {
  const char* v = getenv(name);
  return v ? atoi(v) : dflt;
}
void read_knobs_locked() {
  Knobs k;
  k.nmax = env_raw("SWA_TC_NMAX", 0);
  k.nxb = env_raw("SWA_TC_NXB", 0);
  k.kr = env_raw("SWA_TC_KR", 0);
  k.kw = env_raw("SWA_TC_KW", 0);
  k.stages = env_raw("SWA_TC_STAGES", 0);
  k.nsb = env_raw("SWA_TC_NSB", 0);
  k.th_all = env_raw("SWA_TC_TH", 0);
  k.th[0] = env_raw("SWA_TC_TH_FWD", 0);
  k.th[1] = env_raw("SWA_TC_TH_DQ", 0);
  k.th[2] = env_raw("SWA_TC_TH_DKDV", 0);
  k.trace_it = env_raw("SWA_TC_TRACE_IT", 1);
  k.no_tabs = getenv("SWA_TC_NO_TABS") != nullptr;
  k.disable = getenv("SWA_TC_DISABLE") != nullptr;
  k.verbose = getenv("SWA_TC_VERBOSE") != nullptr;
  k.trace = getenv("SWA_TC_TRACE") != nullptr;
  g_knobs.store(new Knobs(k), std::memory_order_release);
}
const Knobs& knobs() {
  const Knobs* k = g_knobs.load(std::memory_order_acquire);
  if (k) return *k;
  std::lock_guard<std::mutex> lock(g_plan_mu);
  if (!g_knobs.load()) read_knobs_locked();
  return *g_knobs.load();
}

// Widest halo, in token columns, over all resident-tile columns; at most kHaloMost, more than any plan takes (a half-size may be
// any 32-bit number: in 32 bits the width of a huge one wrapped round to a narrow halo, and to a plan for that).
constexpr int kHaloMost = 1 << 20;
int halo_width(const swa_geom_t* g, int TW) {
  const int64_t Wtok = (int64_t)g->t_width * g->b_size, b = g->b_size, wc = g->col_size;
  int64_t best = 0;
  for (int64_t x0 = 0; x0 < Wtok; x0 += TW) {
    const int64_t lo = (x0 / b - wc) * b;
    const int64_t hi = ((x0 + TW - 1) / b + wc + 1) * b;
    best = hi - lo > best ? hi - lo : best;
  }
  return (int)std::min<int64_t>(best, kHaloMost);
}

// Choose the resident tile, the streamed-block shape and the pipeline depths.  Tile shapes tried: 16 x 8 first -- a warp's 32 rows then span
// 4 grid rows and skip 3 of the 7 streamed blocks of a 13-row window -- then 8 x 16.
//   tensor memory (512 columns): forward  score buffers at 128-column strides (packed when they do not fit) + two O accumulators;
//                                backward nsb pairs (S, dP) of 2N columns + the accumulators
//   shared memory:               nxb resident-tile buffers + indicator rows + stages x (block + penalty rows [+ lse, delta])
// (Kernels with streamed rotation; those without: make_strip_shape below.)
bool make_plan_shape(const swa_geom_t* g, int which, int TH, int TW, uint32_t tab_bytes, Plan* out, long* cost_out = nullptr) {
  Plan pl{};
  pl.ncb = 1;
  pl.tab_bytes = tab_bytes;
  pl.TH = TH;
  pl.TW = TW;
  const int hw = halo_width(g, pl.TW);
  if (hw > kPenCols) return false;     // these kernels keep a whole halo row per block row
  const int halo_rows = pl.TH + 2 * g->row_size;
  const int qch = (g->d_qk + 63) / 64, vch = (g->d_v + 63) / 64;
  const uint32_t x_bytes = (which == 0 ? qch : qch + vch) * 16384u;
  const uint32_t row_bytes = (qch + vch) * 128u + kXRowBytes;
  const uint32_t stage_extra = which == 0 ? 0u : 1024u;       // lse / delta slots of a streamed block
  const int acc_cols = which == 0 ? 0 : (which == 1 ? 64 * qch : 64 * (qch + vch));
  const int min_stages = 3;
  // alignment pad of the swizzled tiles + the kernel's barrier / exchange / penalty-table block behind the ring
  const uint32_t kSmemSlack = 1024u + (((which == 0 ? (uint32_t)sizeof(FwdShared) : (uint32_t)sizeof(BwdShared)) + 15u) & ~15u);
  {
    // backward: two (S, dP) pairs of 2N columns next to the accumulators (N = 64 always fits: 256 + 256 columns)
    const int nsb = 2;
    int nmax = which == 0 ? 128 : (512 - acc_cols) / (2 * nsb);
    nmax = nmax > 128 ? 128 : nmax;
    const Knobs kn = knobs();
    if (kn.nmax) nmax = kn.nmax;
    for (int nxb = which == 0 ? 2 : (kn.nxb ? kn.nxb : 2); nxb >= (which == 0 ? 2 : 1); --nxb) {
      const uint32_t fixed = nxb * x_bytes + 128u * kXRowBytes + tab_bytes;
      long best_cost = -1;
      for (int KW = hw; KW <= kPenCols; ++KW)
        for (int KR = 1; KR <= 16; ++KR) {
          const int N = KW * KR;
          if (N > nmax || N % 16) continue;
          if (fixed + min_stages * ((uint32_t)N * row_bytes + stage_extra) + kSmemSlack > kSmemLimit) continue;
          const long nblk = (halo_rows + KR - 1) / KR;
          const long cost = nblk * N * 16 + nblk * 400;  // executed columns + a per-block overhead
          if (best_cost < 0 || cost < best_cost) {
            best_cost = cost;
            pl.KR = KR; pl.KW = KW; pl.N = N;
          }
        }
      if (best_cost < 0) continue;
      if (kn.kr) {
        pl.KR = kn.kr;
        if (kn.kw) pl.KW = kn.kw;
        pl.N = pl.KR * pl.KW;
        pl.ncb = 1;
        // an override must still hold a whole halo row per block row and fit the penalty-table columns
        if (pl.KW < hw || pl.KW > kPenCols || pl.KR > 16) return false;
      }
      const uint32_t stage = (uint32_t)pl.N * row_bytes + stage_extra;
      const int Wtok = g->t_width * g->b_size;
      pl.n_tiles_x = (Wtok + pl.TW - 1) / pl.TW;
      pl.n_tiles_y = (g->t_height + pl.TH - 1) / pl.TH;
      pl.nxb = nxb;
      pl.stages = min_stages;
      while (pl.stages < kMaxStages && fixed + (pl.stages + 1) * stage + kSmemSlack <= kSmemLimit) ++pl.stages;
      if (kn.stages) pl.stages = kn.stages;
      pl.smem_bytes = fixed + pl.stages * stage + kSmemSlack;
      if (which == 0) {
        // forward: score buffers = look-ahead of the score MMAs: 3 next to the two accumulators, 4 (packed at N-column
        // strides) when tensor memory allows and the block ring is deep enough to feed them (measured)
        int n = pl.stages >= 6 ? 4 : 3;
        while (n > 2 && n * pl.N + 2 * 64 * vch > 512) --n;
        pl.nsb = kn.nsb ? kn.nsb : n;
      } else {
        pl.nsb = nsb;
      }
      *out = pl;
      if (cost_out) *cost_out = best_cost;
      // tensor-memory columns of the final plan (the environment overrides above included): a plan beyond the
      // 512-column allocation is refused here, never launched
      const uint32_t fwd_stride = (pl.N <= 128 && pl.nsb * 128 + 2 * 64 * vch <= 512) ? 128u : (uint32_t)pl.N;
      const uint32_t tmem_cols = which == 0 ? pl.nsb * fwd_stride + 2u * 64u * vch : 2u * nsb * pl.N + (uint32_t)acc_cols;
      return pl.smem_bytes <= kSmemLimit && pl.N % 16 == 0 && pl.N >= 16 && pl.N <= 256 && pl.N <= nmax && pl.stages >= 2 &&
             pl.stages <= kMaxStages && pl.nsb >= 2 && pl.nsb <= 4 && tmem_cols <= 512u;
    }
  }
  return false;
}

// Shared memory of the strip kernels beside resident rows, ring and tables: alignment pad of the swizzled tiles, barrier /
// exchange block, row parts of the window mask, dK/dV the lse / delta of streamed rows.
uint32_t strip_slack(const swa_geom_t* g, int which, int R4) {
  const uint32_t sh = which == 0 ? (uint32_t)sizeof(Fwd2Shared) : (uint32_t)sizeof(Bwd2Shared);
  return 1024u + ((sh + 15u) & ~15u) + row_parts_bytes(g->row_size, R4) + (which == 0 ? 0u : bwd_vec_bytes(which == 2));
}

// ... and the mask units: three per ring entry.  In dQ the room of one more is left free: with it one plan in seven would be another, with a
// second resident buffer or strips of the other width, and not all of them a faster one (188 x 100 grid, 9 x 61 window, d = 96, d_v = 32,
// 21 slices: 338 -> 370 us; 59 x 208, 3 x 61, d = 128, d_v = 64: 252 -> 209).
uint32_t mask_bytes(int N, int which) { return (uint32_t)N * 16u * (3u * kMaskRing + (which == 1 ? 1u : 0u)); }

// Blocks of a chunk of `nq` quarters whose first row is r0 (the kernels' strip_item).
int strip_blocks(const swa_geom_t* g, const Plan& pl, int r0, int nq) {
  const int q = std::min(nq, (g->t_height - r0 + pl.R4 - 1) / pl.R4);
  const int h0 = r0 - g->row_size + pl.KR * (std::max(0, g->row_size - r0) / pl.KR);
  const int last = std::min(r0 + q * pl.R4 - 1 + g->row_size, g->t_height - 1);
  return ((last - h0) / pl.KR + 1) * pl.ncb;
}

// Whether quarters can slide through the slots: quarter i + 4 must not meet a block before the last one of quarter i.
bool strip_slides(const swa_geom_t* g, int R4, int KR) {
  for (int i = 0; i < KR; ++i)
    if ((i * R4 + R4 - 1 + 2 * g->row_size) / KR >= (i + 4) * R4 / KR) return false;
  return true;
}

// Chunk height in quarters.  Sliding strips: the tallest chunk has the fewest blocks per row (2 wr rows of halo are met
// once per chunk), short ones spread a small problem over all SMs; the slowest SM's blocks decide, the taller of two equals.  The
// height is a multiple of the block height, so that no row's blocks depend on it.
// A call of a batch size not met before pays for this (three plans: 2 us at 24 x 24, 24 at 128 x 128 with one head, 470 at
// 4096 x 64; walking every item of every height took 28, 750 and 11100): heights are taken in the order of a bound -- their
// mean load, their largest item -- and the load of every CTA is put together only for those whose bound is not beyond the best
// load found.
void choose_chunk(const swa_geom_t* g, Plan* pl) {
  const int quarters = (g->t_height + pl->R4 - 1) / pl->R4;
  const int64_t strips = (int64_t)pl->n_tiles_x * g->B * g->H;
  if (!strip_slides(g, pl->R4, pl->KR)) {
    pl->nq = 4;
  } else {
    struct Height {
      double bound;
      int nq, lo, hi;                                        // chunks [lo, hi) meet their whole halo inside the grid: the same blocks
      int64_t mid;
      bool exact;
      bool operator<(const Height& o) const { return bound < o.bound || (bound == o.bound && nq > o.nq); }
    };
    const int sms = sm_count();
    int unit = 1;
    while (unit * pl->R4 % pl->KR) ++unit;
    const int most = std::max(1, 2048 / pl->R4);            // chunk rows the kernels' div_kr covers
    auto cost = [&](int nq, int c) { return (int64_t)strip_blocks(g, *pl, c * nq * pl->R4, nq) + 2; };
    std::vector<Height> heights;
    for (int nq = unit; ; nq += unit) {
      const bool whole = nq >= quarters;
      if (nq > most && !(whole && quarters <= most) && nq > unit) break;
      const int chunks = (quarters + nq - 1) / nq, rows = nq * pl->R4;
      Height h;
      h.nq = nq;
      h.lo = std::min(chunks, (g->row_size + rows - 1) / rows);
      h.hi = std::max(h.lo, (g->t_height - g->row_size) / rows);
      h.mid = h.hi > h.lo ? cost(nq, h.lo) : 0;
      int64_t total = (h.hi - h.lo) * h.mid, largest = h.mid;
      for (int c = 0; c < chunks; ++c) {
        if (c == h.lo) c = h.hi;
        if (c >= chunks) break;
        const int64_t x = cost(nq, c);
        total += x;
        largest = std::max(largest, x);
      }
      const int64_t items = strips * chunks;
      h.exact = items <= sms || items > 8 * sms;
      h.bound = items > 8 * sms ? (double)total * strips / sms + 0.5 * strip_blocks(g, *pl, 0, nq)
                                : (double)std::max(largest, items <= sms ? 0 : (total * strips + sms - 1) / sms);
      heights.push_back(h);
      if (whole) break;
    }
    std::sort(heights.begin(), heights.end());
    double best = -1.;
    std::vector<int64_t> cta(sms);
    for (const Height& h : heights) {
      if (best >= 0. && (h.bound > best || (h.bound == best && h.nq < pl->nq))) {
        if (h.bound > best) break;
        continue;
      }
      double load = h.bound;
      if (!h.exact) {
        const int chunks = (quarters + h.nq - 1) / h.nq, items = (int)(strips * chunks), each = items / sms, more = items % sms;
        for (int i = 0; i < sms; ++i) cta[i] = (each + (i < more ? 1 : 0)) * h.mid;
        for (int c = 0; c < chunks; ++c) {                     // what the chunks at the edges have less
          if (c == h.lo) c = h.hi;
          if (c >= chunks) break;
          const int64_t x = cost(h.nq, c) - h.mid;
          for (int i = c * pl->n_tiles_x; i < items; i += chunks * pl->n_tiles_x) {
            int at = i % sms;
            for (int tx = 0; tx < pl->n_tiles_x; ++tx) {
              cta[at] += x;
              if (++at == sms) at = 0;
            }
          }
        }
        load = (double)*std::max_element(cta.begin(), cta.end());
      }
      if (best < 0. || load < best || (load == best && h.nq > pl->nq)) {
        best = load;
        pl->nq = h.nq;
      }
    }
  }
  pl->n_tiles_y = (quarters + pl->nq - 1) / pl->nq;
  pl->chunk_rows = pl->nq * pl->R4;
}

// Plan of the kernels without streamed rotation for strips TW token columns wide (swa_tc_strip.cuh).  Halos wider than any
// block are walked in `ncb` column blocks per row band.
bool make_strip_shape(const swa_geom_t* g, int which, int TW, Plan* out) {
  Plan pl{};
  pl.TW = TW;
  pl.TH = 128 / TW;
  pl.R4 = 32 / TW;
  const int hw = halo_width(g, TW);
  const int qch = (g->d_qk + 63) / 64, vch = (g->d_v + 63) / 64;
  const uint32_t x_bytes = (which == 0 ? qch : qch + vch) * 16384u;
  const uint32_t row_bytes = (qch + vch) * 128u;
  const int out_chunks = which == 0 ? vch : which == 1 ? qch : qch + vch;
  const int acc_cols = which == 0 ? 2 * 64 * vch : (which == 1 ? 64 * qch : 64 * (qch + vch));
  const int min_stages = 3;
  const uint32_t slack = strip_slack(g, which, pl.R4);
  const Knobs kn = knobs();
  int nmax = which == 0 ? 128 : std::min(128, (512 - acc_cols) / 4);
  if (kn.nmax) nmax = kn.nmax;
  pl.n_tiles_x = (g->t_width * g->b_size + TW - 1) / TW;
  const int quarters = (g->t_height + pl.R4 - 1) / pl.R4;
  // output staging for a whole quarter; for wide heads, whose quarters never follow each other block by block, one chunk (the
  // forward kernel: none)
  pl.stg = which == 0 ? (qch == 1 && vch == 1) : qch == 1 && vch == 1 ? out_chunks : 1;
  const uint32_t fixed = kIndicatorBytes + 4u * pl.stg * kStageChunk + slack;
  long best_cost = -1;
  for (int ncb = 1; ncb <= 16 && best_cost < 0; ++ncb)
    for (int KW = (hw + ncb - 1) / ncb; KW <= 128 && (ncb == 1 || KW * (ncb - 1) < hw); ++KW)
      for (int KR = 1; KR <= 16; ++KR) {
        const int N = KW * KR;
        if (N > nmax || N % 16 || N < 32) continue;            // (both compute groups need columns)
        const bool slides = strip_slides(g, pl.R4, KR);
        Plan c = pl;
        c.KR = KR; c.KW = KW; c.N = N; c.ncb = ncb;
        long blocks = 0, items = 1;                            // per strip of the whole grid height
        if (slides) {
          blocks = strip_blocks(g, c, 0, quarters);
        } else {
          items = (quarters + 3) / 4;
          for (int q = 0; q < quarters; q += 4) blocks += strip_blocks(g, c, q * pl.R4, 4);
        }
        // One resident buffer leaves room for larger blocks, but nothing overlaps the load of an item's resident rows (about
        // 3000 cycles, the time of 250 columns); sliding strips need two.
        for (int nxb = kn.nxb && which ? kn.nxb : 2; nxb >= (kn.nxb || slides || which == 0 ? 2 : 1) && nxb >= 1; --nxb) {
          if (fixed + nxb * x_bytes + min_stages * (uint32_t)N * row_bytes + mask_bytes(N, which) > kSmemLimit) continue;
          // executed columns + what a block costs beside them: backward as much as a hundred columns, forward forty.  (Fitted on kernels
          // whose blocks took a quarter longer; the number of score buffers, two or three, is not in it.  On the present ones, 49 plans of 17
          // geometries against those of the other strip width and of smaller blocks and either resident buffer count: the fastest
          // or within 3 % of it in 44, 5 to 8 % off in five -- 60 x 60, 7 x 7, d = 128, all three kernels; 100 x 75, 5 x 5, forward; 80 x 80,
          // 13 x 13, d = 128 / 64, dK/dV.)
          const long cost = (blocks * (N + (which == 0 ? 40 : 100)) + (nxb == 1 ? items * 250 : 0)) * pl.n_tiles_x;
          if (best_cost < 0 || cost < best_cost) {
            best_cost = cost;
            pl.KR = KR; pl.KW = KW; pl.N = N; pl.ncb = ncb; pl.nxb = nxb;
          }
        }
      }
  if (best_cost < 0) return false;
  if (kn.kr) {
    pl.KR = kn.kr;
    if (kn.kw) pl.KW = kn.kw;
    pl.N = pl.KR * pl.KW;
    pl.ncb = 1;
    if (pl.KW < hw || pl.KW > 128 || pl.KR > 16) return false;      // an override must still hold a whole halo row
    pl.nxb = 2;
  }
  const uint32_t stage = (uint32_t)pl.N * row_bytes, rest = fixed + pl.nxb * x_bytes + mask_bytes(pl.N, which);
  pl.kr_inv = (65536 + pl.KR - 1) / pl.KR;
  pl.kw_inv = (65536 + pl.KW - 1) / pl.KW;
  pl.tw_log = TW == 8 ? 3 : 4;
  pl.stages = min_stages;
  while (pl.stages < kMaxStages && rest + (pl.stages + 1) * stage <= kSmemLimit) ++pl.stages;
  if (kn.stages) pl.stages = kn.stages;
  pl.smem_bytes = rest + pl.stages * stage;
  // backward: a third score buffer where tensor memory has room beside the two of dP (swa_tc_bwd2.cuh)
  pl.nsb = which && 5 * pl.N + acc_cols <= 512 ? 3 : 2;
  if (which == 0) {
    // score buffers = look-ahead of the score MMAs: 3, or 4 when the block ring is deep enough to feed them (measured); with
    // columns of their own for P if that leaves three (swa_tc_fwd2.cuh), else P over the scores
    const int most = kn.nsb ? kn.nsb : pl.stages >= 6 ? 4 : 3, room = 512 - acc_cols;
    pl.p_off = std::max(3, kn.nsb) * (pl.N + pl.N / 2) <= room ? pl.N : 0;
    const int per = pl.N + pl.p_off / 2;
    pl.nsb = std::max(kn.nsb ? kn.nsb : 2, std::min(most, room / per));
    pl.s_stride = per <= 128 && pl.nsb * 128 <= room ? 128 : per;
  }
  *out = pl;
  // tensor-memory columns of the final plan (the environment overrides above included): a plan beyond the
  // 512-column allocation is refused here, never launched
  const uint32_t tmem_cols = (uint32_t)(which == 0 ? pl.nsb * pl.s_stride : (pl.nsb + 2) * pl.N) + (uint32_t)acc_cols;
  return pl.smem_bytes <= kSmemLimit && pl.N % 16 == 0 && pl.N >= 16 && pl.N <= 256 && pl.N <= nmax && pl.stages >= 2 &&
         pl.stages <= kMaxStages && pl.nsb >= 2 && pl.nsb <= 4 && tmem_cols <= 512u;
}

// Strip width by the time of a whole image (the choice, and with it the order of every sum, must not depend on the batch): its
// blocks, each its columns and what it costs beside them (as in make_strip_shape), and per item the load of its resident rows
// where one buffer holds them, here at half of what it weighs against a second buffer there: the next item's first blocks
// hide the rest.  At 250 columns, 131 x 24, window 11, d = 96 took strips of 8 backward (1165 us a training step of 128 slices
// against 949 with strips of 16), 128 x 128, window 15, d_v = 128 strips of 16 in dQ (151 against 135 us for 16 slices).
bool make_strip_plan(const swa_geom_t* g, int which, Plan* out) {
  const Knobs kn = knobs();
  const int th = kn.th[which] ? kn.th[which] : kn.th_all;
  const double beside = which == 0 ? 40. : 100.;
  double best = -1.;
  for (int TW : {8, 16}) {
    Plan pl;
    if ((th && th != 128 / TW) || !make_strip_shape(g, which, TW, &pl)) continue;
    const int quarters = (g->t_height + pl.R4 - 1) / pl.R4, step = strip_slides(g, pl.R4, pl.KR) ? quarters : 4;
    double cost = 0.;
    for (int q = 0; q < quarters; q += step) cost += strip_blocks(g, pl, q * pl.R4, step) * (pl.N + beside) + (pl.nxb == 1 ? 125. : 0.);
    cost *= pl.n_tiles_x;
    if (best < 0. || cost < best) {
      best = cost;
      *out = pl;
    }
  }
  return best >= 0.;
}

// Bytes of the cos/sin tables when they are small enough to be staged in shared memory, else 0.
uint32_t rope_table_bytes(const swa_rope_t* rope) {
  if (!rope || !rope->idx) return 0;
  const uint64_t b = (uint64_t)(rope->max_h + rope->max_w) * rope_tab_stride(rope->n_rdim);
  return b <= 48 * 1024 && !knobs().no_tabs ? (uint32_t)((b + 15) & ~15ull) : 0;
}

// Tile shape for one choice of staged-table bytes; *cost = the planner's block cost of the plan taken.
static bool make_plan_tab(const swa_geom_t* g, const swa_rope_t* rope, int which, uint32_t tab, Plan* out, long* cost) {
  const Knobs kn = knobs();
  const int th = kn.th[which] ? kn.th[which] : kn.th_all;
  if (th == 8) return make_plan_shape(g, which, 8, 16, tab, out, cost);
  if (th == 16) return make_plan_shape(g, which, 16, 8, tab, out, cost);
  if (which == 2) {
    // dK/dV (K tile resident, Q blocks streamed; its accumulators leave the narrowest blocks): the shape whose
    // blocks cost less by the planner's own measure -- 16 x 8 at the 13 x 13 window with d = 64, 8 x 16 once
    // d_v = 128 or the window grows (measured: 10 % and 13 % faster at 15 x 15 / d_v = 128 and 31 x 31 / d = 128).
    Plan a, b;
    long ca = 0, cb = 0;
    const bool oa = make_plan_shape(g, which, 16, 8, tab, &a, &ca), ob = make_plan_shape(g, which, 8, 16, tab, &b, &cb);
    if (!oa && !ob) return false;
    const bool take_a = oa && (!ob || ca <= cb);
    *out = take_a ? a : b;
    *cost = take_a ? ca : cb;
    return true;
  }
  // measured at the 13 x 13 window: 16 x 8 wins (80-token blocks, every block row shared by two rotating threads),
  // except for the dQ kernel when at most 32 of 64 q/k dims are rotated (measured 12 % faster at d_v = 128
  // with a 15 x 15 window and 3 % at the 13 x 13 window; at d_qk = 128 the 16 x 8 tile stays 27 % ahead)
  const bool wide_first = which == 1 && rope->n_rdim <= 8 && g->d_qk == 64;
  return wide_first ? (make_plan_shape(g, which, 8, 16, tab, out, cost) || make_plan_shape(g, which, 16, 8, tab, out, cost))
                    : (make_plan_shape(g, which, 16, 8, tab, out, cost) || make_plan_shape(g, which, 8, 16, tab, out, cost));
}

// The cos/sin tables are staged in shared memory when that does not cost block size: a plan with the tables is
// taken only if its blocks are as cheap as those of the plan without them (40 KB of tables beside d = 128 tiles
// would force 48-token instead of 80-token blocks, measured 1.5x slower in the forward kernel).
// Plans are cached: the search below is a few thousand candidate shapes, repeated for the three kernels of every
// step with the same geometry.  Key = everything the planner reads.
using PlanKey = std::tuple<int, int, int, int, int, int, int, int, int, int, int, int, int>;
std::map<PlanKey, std::pair<bool, Plan>> g_plan_cache;

// `items`: batch x heads, which only the strips' chunk height depends on (0: everything else of a plan).
PlanKey plan_key(const swa_geom_t* g, const swa_rope_t* rope, int which, bool v2, int items = 0) {
  const bool has = rope && rope->idx;
  return PlanKey(which + (v2 ? 3 : 0), g->t_height, g->t_width, g->b_size, g->row_size, g->col_size, g->d_qk, g->d_v,
                 has ? rope->n_rdim : 0, has ? rope->max_h : 0, has ? rope->max_w : 0, g->dtype == SWA_BF16 ? 1 : 0, items);
}
bool cache_lookup(const PlanKey& k, bool* ok, Plan* out) {
  std::lock_guard<std::mutex> lock(g_plan_mu);
  auto it = g_plan_cache.find(k);
  if (it == g_plan_cache.end()) return false;
  *ok = it->second.first;
  *out = it->second.second;
  return true;
}
void cache_store(const PlanKey& k, bool ok, const Plan& pl) {
  std::lock_guard<std::mutex> lock(g_plan_mu);
  if (g_plan_cache.size() > 4096) g_plan_cache.clear();
  g_plan_cache[k] = std::make_pair(ok, pl);
}

bool make_plan_uncached(const swa_geom_t* g, const swa_rope_t* rope, int which, Plan* out) {
  const uint32_t tab = rope_table_bytes(rope);
  Plan with, without;
  long cw = 0, cn = 0;
  const bool ok_n = make_plan_tab(g, rope, which, 0, &without, &cn);
  if (tab && make_plan_tab(g, rope, which, tab, &with, &cw) && (!ok_n || cw <= cn)) {
    *out = with;
    return true;
  }
  if (ok_n) *out = without;
  return ok_n;
}

bool make_plan(const swa_geom_t* g, const swa_rope_t* rope, int which, Plan* out) {
  const PlanKey key = plan_key(g, rope, which, false);
  bool ok = false;
  if (cache_lookup(key, &ok, out)) return ok;
  Plan pl{};
  ok = make_plan_uncached(g, rope, which, &pl);
  cache_store(key, ok, pl);
  if (ok) *out = pl;
  return ok;
}

// Indicator value a and penalty b (powers of two, exact in fp16 and bf16) of the window mask that
// rides on the score MMA: a*b*scale*log2(e) >= 4000, so exp2 of a masked score is exactly 0.
bool mask_constants(float sm_scale, float* a, float* b) {
  const float need = 4000.f / (sm_scale * kLog2e);
  float bb = 16384.f, aa = 1.f;
  while (aa * bb < need && aa < 16384.f) aa *= 2.f;
  *a = aa;
  *b = bb;
  return aa * bb >= need;
}

// Plan of the kernels that rotate no streamed row (rotation handed on between the kernels, or no RoPE).
bool make_plan_prerot(const swa_geom_t* g, int which, Plan* out) {
  // a step asks for the same three plans a dozen times: the last one of each kind, per thread, needs no lock
  struct Last { PlanKey key; bool ok; Plan pl; const Knobs* epoch; };
  static thread_local Last last[3] = {};
  const Knobs* epoch = &knobs();
  const PlanKey key = plan_key(g, nullptr, which, true, g->B * g->H);
  Last& l = last[which];
  if (l.epoch == epoch && l.key == key) {
    if (l.ok) *out = l.pl;
    return l.ok;
  }
  bool ok = false;
  Plan pl{};
  if (!cache_lookup(key, &ok, &pl)) {
    const PlanKey shape = plan_key(g, nullptr, which, true);
    if (!cache_lookup(shape, &ok, &pl)) {
      ok = make_strip_plan(g, which, &pl);
      cache_store(shape, ok, pl);
    }
    if (ok) choose_chunk(g, &pl);
    cache_store(key, ok, pl);
  }
  l = Last{key, ok, pl, epoch};
  if (ok) *out = pl;
  return ok;
}

KParams make_params(const swa_geom_t* g, const swa_rope_t* rope, const Plan& pl, int32_t* status) {
  KParams p;
  p.t_h = g->t_height;
  p.Wtok = g->t_width * g->b_size;
  p.b = g->b_size;
  p.wr = g->row_size;
  p.wc = g->col_size;
  p.H = g->H;
  p.qch = (g->d_qk + 63) / 64;
  p.vch = (g->d_v + 63) / 64;
  p.dqk = g->d_qk;
  p.dv = g->d_v;
  p.sm_scale = g->sm_scale;
  p.scale_log2 = g->sm_scale * kLog2e;
  mask_constants(g->sm_scale, &p.mask_a, &p.mask_b);
  p.pl = pl;
  p.rope = make_rope(rope);
  p.n_items = pl.n_tiles_x * pl.n_tiles_y * g->B * g->H;
  p.div_b = g->b_size == 1 ? 0u : (uint32_t)((0x100000000ull + g->b_size - 1) / g->b_size);
  {
    int step = std::min(p.n_items, sm_count());                // one CTA per SM
    p.step_tx = step % pl.n_tiles_x;
    step /= pl.n_tiles_x;
    p.step_cy = step % pl.n_tiles_y;
    step /= pl.n_tiles_y;
    p.step_hi = step % g->H;
    p.step_bi = step / g->H;
  }
  p.status = status;
  // the Python layer hands a 4 KiB status buffer: words 0-3 status, bytes 16.. = 4 roles x 32 clock samples
  const Knobs kn = knobs();
  p.trace = (status != nullptr && kn.trace) ? reinterpret_cast<long long*>(status + 4) : nullptr;
  p.trace_it = kn.trace_it;
  return p;
}

// What a tensor map of these kernels can describe: unit last stride, 16-byte aligned base and rows, and strictly
// positive strides (a batch or head dimension broadcast with stride 0 cannot be encoded; extents of 1 are
// given a legal stride when the map is built).  `B`, `H` = extents of the first two dimensions.
bool tensor_ok(const swa_tensor_t* t, int B, int H) {
  return t->stride[3] == 1 && ((uintptr_t)t->ptr % 16) == 0 && t->stride[0] % 8 == 0 && t->stride[1] % 8 == 0 &&
         t->stride[2] % 8 == 0 && t->stride[2] > 0 && (B == 1 || t->stride[0] > 0) && (H == 1 || t->stride[1] > 0);
}

}  // namespace

const char* last_error() { return g_tc_err; }

int sm_count() {
  static std::atomic<int> cached[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  int n = cached[dev].load(std::memory_order_relaxed);
  if (n == 0) {
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    cached[dev].store(n, std::memory_order_relaxed);
  }
  return n;
}

void refresh_env() {
  std::lock_guard<std::mutex> lock(g_plan_mu);
  read_knobs_locked();
  g_plan_cache.clear();
}

const char* unsupported_reason(const swa_geom_t* g, const swa_rope_t* rope, const swa_tensor_t* const* tensors,
                               int n_tensors, int which, bool prerotated, bool any8) {
  if (knobs().disable) return "disabled by SWA_TC_DISABLE";
  if (g->dtype != SWA_F16 && g->dtype != SWA_BF16) return "fp32 runs on the SIMT kernels";
  // The kernels work on 64-element chunks of a row.  Those without streamed rotation also take head dims of 32 and
  // 96, and with any8 any multiple of 8 (a tensor map's rows and strides are counted in 16 bytes): the tensor map's innermost
  // extent is the real head dim, so TMA zero-fills the missing part of the last chunk
  // (zero columns of q, k leave every score unchanged, zero columns of v and dO give zero columns of O, dV that are
  // never stored), which costs MMA work on zeros but no HBM traffic and no padded copies.
  {
    const bool v2_dims = prerotated || !(rope && rope->idx);
    auto dim_ok = [&](int d) { return v2_dims && any8 ? (d >= 8 && d <= 128 && d % 8 == 0) : v2_dims ? (d >= 32 && d <= 128 && d % 32 == 0) : (d == 64 || d == 128); };
    if (!dim_ok(g->d_qk) || !dim_ok(g->d_v))
      return v2_dims && any8 ? "head dims must be multiples of 8 up to 128" : v2_dims ? "head dims must be 32, 64, 96 or 128" : "head dims must be 64 or 128 for the kernels that rotate streamed rows";
  }
  if (!(g->sm_scale > 0.f)) return "sm_scale must be positive";
  float ma, mb;
  if (!mask_constants(g->sm_scale, &ma, &mb)) return "sm_scale too small for the MMA-side window mask";
  if (rope && rope->idx && rope->n_rdim != 8 && rope->n_rdim != 16 && rope->n_rdim != 32)
    return "n_rdim must be 8, 16 or 32 (RoPE on 32, 64 or 128 dims)";
  if (rope && rope->idx && !(prerotated && which == 0) && (((uintptr_t)rope->row_cs | (uintptr_t)rope->col_cs) & 15))
    return "cos/sin tables must be 16-byte aligned";      // (the forward kernel of rotated copies reads none)
  if (g->row_size > 64) return "row window too tall for the penalty tables";
  if ((int64_t)g->t_height * g->t_width * g->b_size > (1 << 30)) return "grid too large";
  Plan pl;
  const bool v2 = prerotated || !(rope && rope->idx);
  if (!(v2 ? make_plan_prerot(g, which, &pl) : make_plan(g, rope, which, &pl)))
    return "no tile plan fits (window too wide for one streamed block of the kernels with streamed rotation)";
  for (int i = 0; i < n_tensors; ++i)
    if (!tensor_ok(tensors[i], g->B, g->H)) return "tensors need unit last stride, positive strides and 16-byte aligned rows";
  return nullptr;
}

bool describe_plan(const swa_geom_t* g, const swa_rope_t* rope, int which, int32_t* out) {
  // which 0..2: the kernel swa_fwd / swa_bwd_dq / swa_bwd_dkdv would run; 3..5: swa_fwd_rot / swa_bwd_dq_rot /
  // swa_bwd_dkdv_rot.  Without RoPE, and for 3..5, these are the kernels without streamed rotation.
  const bool prerot = which >= 3;
  const int kind = which % 3;
  const bool v2 = prerot || !(rope && rope->idx);
  Plan pl;
  if (!(v2 ? make_plan_prerot(g, kind, &pl) : make_plan(g, rope, kind, &pl))) return false;
  const uint32_t qch = (g->d_qk + 63) / 64, vch = (g->d_v + 63) / 64, N = pl.N;
  const uint32_t xrow = v2 ? 0u : kXRowBytes;                               // window-mask bytes per streamed token of a stage
  const uint32_t x_fixed = v2 ? kIndicatorBytes + 4u * pl.stg * kStageChunk + mask_bytes(pl.N, kind) + row_parts_bytes(g->row_size, pl.R4) : 128u * kXRowBytes;
  uint32_t used = 1023, tmem = 0;   // worst-case pad to the 1024-byte alignment of the swizzled tiles
  if (kind == 0) {
    used += 2 * qch * 16384u + x_fixed + pl.stages * N * ((qch + vch) * 128u + xrow);
    used += ((v2 ? (uint32_t)sizeof(Fwd2Shared) : (uint32_t)sizeof(FwdShared)) + 15u) & ~15u;
    const uint32_t o_cols = vch * 64u;
    const uint32_t stride = v2 ? (uint32_t)pl.s_stride : (N <= 128u && pl.nsb * 128u + 2 * o_cols <= 512u) ? 128u : N;
    tmem = pl.nsb * stride + 2 * o_cols;
    if (stride < N + (v2 ? pl.p_off / 2 : 0)) tmem = 1u << 30;   // a score buffer would not hold a block
  } else {
    used += pl.nxb * (qch + vch) * 16384u + x_fixed + pl.stages * (N * ((qch + vch) * 128u + xrow) + (v2 ? 0u : 1024u));
    used += (((v2 ? (uint32_t)sizeof(Bwd2Shared) : (uint32_t)sizeof(BwdShared)) + 15u) & ~15u) + (v2 ? bwd_vec_bytes(kind == 2) : 0u);
    tmem = (v2 ? pl.nsb + 2 : 4) * N + 64u * qch + (kind == 2 ? 64u * vch : 0u);
  }
  used += pl.tab_bytes;
  const int32_t v[12] = {pl.TH, pl.TW, pl.KR, pl.KW, pl.N, pl.stages, kind == 0 || v2 ? pl.nsb : 2, kind == 0 ? 2 : pl.nxb,
                         (int32_t)pl.tab_bytes, (int32_t)pl.smem_bytes, (int32_t)used, (int32_t)tmem};
  for (int i = 0; i < 12; ++i) out[i] = v[i];
  return true;
}

int launch_fwd(const swa_geom_t* g, const swa_rope_t* rope, const swa_tensor_t* q, const swa_tensor_t* k,
               const swa_tensor_t* v, const swa_tensor_t* o, float* lse, int32_t* status, cudaStream_t st) {
  if (!(rope && rope->idx)) return launch_fwd2(g, q, k, v, o, lse, status, st);
  Plan pl;
  if (!make_plan(g, rope, 0, &pl)) {
    snprintf(g_tc_err, sizeof(g_tc_err), "no tile plan");
    return -1;
  }
  CUtensorMap tq, tk, tv;
  if (!make_map(&tq, q, g, g->d_qk, pl.TW, pl.TH) || !make_map(&tk, k, g, g->d_qk, pl.KW, pl.KR) ||
      !make_map(&tv, v, g, g->d_v, pl.KW, pl.KR))
    return -1;
  const KParams p = make_params(g, rope, pl, status);
  // persistent: one CTA per SM, each walks the items blockIdx.x, blockIdx.x + gridDim.x, ...
  const int n_items = pl.n_tiles_x * pl.n_tiles_y * g->B * g->H;
  const int sms = sm_count();
  dim3 grid(n_items < sms ? n_items : sms), block(kFwdThreads);
  using FwdKernel = void (*)(const CUtensorMap, const CUtensorMap, const CUtensorMap, KParams, View4, float*);
  // the RoPE table width is a template parameter of the kernel (index: n_rdim / 8; calls without rotation went to launch_fwd2),
  // and so is whether the cos/sin tables are staged in shared memory
  static const FwdKernel fwd_table[2][2][5] = {
      {{nullptr, fwd_kernel<false, 1, false>, fwd_kernel<false, 2, false>, nullptr, fwd_kernel<false, 4, false>},
       {nullptr, fwd_kernel<false, 1, true>, fwd_kernel<false, 2, true>, nullptr, fwd_kernel<false, 4, true>}},
      {{nullptr, fwd_kernel<true, 1, false>, fwd_kernel<true, 2, false>, nullptr, fwd_kernel<true, 4, false>},
       {nullptr, fwd_kernel<true, 1, true>, fwd_kernel<true, 2, true>, nullptr, fwd_kernel<true, 4, true>}}};
  const int ni = rope->n_rdim / 8;
  FwdKernel kern = fwd_table[g->dtype == SWA_BF16 ? 1 : 0][pl.tab_bytes ? 1 : 0][ni];
  if (kern == nullptr) {
    snprintf(g_tc_err, sizeof(g_tc_err), "n_rdim %d has no tensor-core kernel", rope ? rope->n_rdim : 0);
    return -1;
  }
  cudaError_t e = allow_smem((const void*)kern);
  if (e != cudaSuccess) {
    snprintf(g_tc_err, sizeof(g_tc_err), "cudaFuncSetAttribute(%u bytes): %s", pl.smem_bytes, cudaGetErrorString(e));
    return -1;
  }
  if (knobs().verbose)
    fprintf(stderr, "[swa2d] fwd plan: tile %dx%d, block %dx%d (N=%d), stages %d, tables %u, smem %u, %d items on %u CTAs\n",
            pl.TH, pl.TW, pl.KR, pl.KW, pl.N, pl.stages, pl.tab_bytes, pl.smem_bytes, n_items, grid.x);
  kern<<<grid, block, pl.smem_bytes, st>>>(tq, tk, tv, p, make_view(o), lse);
  return 0;
}

int launch_fwd2(const swa_geom_t* g, const swa_tensor_t* q, const swa_tensor_t* k, const swa_tensor_t* v,
                const swa_tensor_t* o, float* lse, int32_t* status, cudaStream_t st) {
  Plan pl;
  if (!make_plan_prerot(g, 0, &pl)) {      // nothing is rotated: the plan of the problem without RoPE
    snprintf(g_tc_err, sizeof(g_tc_err), "no tile plan");
    return -1;
  }
  CUtensorMap tq, tk, tv, to;
  if (!make_map(&tq, q, g, g->d_qk, pl.TW, pl.R4) || !make_map(&tk, k, g, g->d_qk, pl.KW, pl.KR) ||
      !make_map(&tv, v, g, g->d_v, pl.KW, pl.KR) || !make_map(&to, o, g, g->d_v, pl.TW, pl.R4))
    return -1;
  const KParams p = make_params(g, nullptr, pl, status);
  const int sms = sm_count();
  dim3 grid(p.n_items < sms ? p.n_items : sms), block(kFwdThreads);   // persistent: one CTA per SM walks the items
  const bool one = p.qch == 1 && p.vch == 1;
  using FwdKernel = void (*)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const CUtensorMap, const KParams, const View4, float*);
  static const FwdKernel table[2][2][2] = {   // [dtype][heads of at most 64][P in columns of its own]
      {{fwd2_kernel<false, false, false>, fwd2_kernel<false, false, true>}, {fwd2_kernel<false, true, false>, fwd2_kernel<false, true, true>}},
      {{fwd2_kernel<true, false, false>, fwd2_kernel<true, false, true>}, {fwd2_kernel<true, true, false>, fwd2_kernel<true, true, true>}}};
  const FwdKernel kern = table[g->dtype == SWA_BF16 ? 1 : 0][one ? 1 : 0][pl.p_off ? 1 : 0];
  cudaError_t e = allow_smem((const void*)kern);
  if (e != cudaSuccess) {
    snprintf(g_tc_err, sizeof(g_tc_err), "cudaFuncSetAttribute(%u bytes): %s", pl.smem_bytes, cudaGetErrorString(e));
    return -1;
  }
  if (knobs().verbose)
    fprintf(stderr, "[swa2d] fwd2 plan: tile %dx%d, block %dx%d (N=%d), stages %d, score buffers %d, %d quarters per chunk, smem %u, %d items on %u CTAs\n",
            pl.TH, pl.TW, pl.KR, pl.KW, pl.N, pl.stages, pl.nsb, pl.nq, pl.smem_bytes, p.n_items, grid.x);
  e = launch_pdl(kern, grid, block.x, pl.smem_bytes, st, tq, tk, tv, to, p, make_view(o), lse);
  if (e != cudaSuccess) snprintf(g_tc_err, sizeof(g_tc_err), "launch: %s", cudaGetErrorString(e));
  return e == cudaSuccess ? 0 : -1;
}

namespace {

// `prerotated`: q and k are the rotated copies the streaming pass of swa_fwd_rot made; the strip kernels rotate nothing
// they stream and only rotate dQ / dK back in the epilogue.
template <bool DKDV>
int launch_bwd(const swa_geom_t* g, const swa_rope_t* rope, bool prerotated, const swa_tensor_t* xqk, const swa_tensor_t* xv,
               const swa_tensor_t* yqk, const swa_tensor_t* yv, const float* lse, const float* delta,
               const swa_tensor_t* out_qk, const swa_tensor_t* out_v, int32_t* status, cudaStream_t st) {
  Plan pl;
  const bool v2 = prerotated || !(rope && rope->idx);      // the kernels without streamed rotation
  if (!(v2 ? make_plan_prerot(g, DKDV ? 2 : 1, &pl) : make_plan(g, rope, DKDV ? 2 : 1, &pl))) {
    snprintf(g_tc_err, sizeof(g_tc_err), "no tile plan");
    return -1;
  }
  CUtensorMap mxqk, mxv, myqk, myv;
  const int x_rows = v2 ? pl.R4 : pl.TH;                    // the strip kernels load the resident side quarter by quarter
  if (!make_map(&mxqk, xqk, g, g->d_qk, pl.TW, x_rows) || !make_map(&mxv, xv, g, g->d_v, pl.TW, x_rows) ||
      !make_map(&myqk, yqk, g, g->d_qk, pl.KW, pl.KR) || !make_map(&myv, yv, g, g->d_v, pl.KW, pl.KR))
    return -1;
  const KParams p = make_params(g, rope, pl, status);
  const int sms = sm_count();
  dim3 grid(p.n_items < sms ? p.n_items : sms), block(kBwdThreads);   // persistent: one CTA per SM walks the items
  using BwdKernel = void (*)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const CUtensorMap, KParams, const float*,
                             const float*, View4, View4);
  using StripKernel = void (*)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const CUtensorMap, const CUtensorMap,
                               const CUtensorMap, const KParams, const float*, const float*);
  // [dtype][tables staged][n_rdim / 8]: q / k rotated in shared memory, dQ / dK rotated back in the epilogue
  static const BwdKernel fused_table[2][2][5] = {
      {{nullptr, bwd_kernel<false, DKDV, 1, false>, bwd_kernel<false, DKDV, 2, false>, nullptr, bwd_kernel<false, DKDV, 4, false>},
       {nullptr, bwd_kernel<false, DKDV, 1, true>, bwd_kernel<false, DKDV, 2, true>, nullptr, bwd_kernel<false, DKDV, 4, true>}},
      {{nullptr, bwd_kernel<true, DKDV, 1, false>, bwd_kernel<true, DKDV, 2, false>, nullptr, bwd_kernel<true, DKDV, 4, false>},
       {nullptr, bwd_kernel<true, DKDV, 1, true>, bwd_kernel<true, DKDV, 2, true>, nullptr, bwd_kernel<true, DKDV, 4, true>}}};
  // [dtype][heads of at most 64][n_rdim / 8]: no RoPE, or inputs already rotated and only the epilogue rotation
  static const StripKernel prerot_table[2][2][5] = {
      {{bwd2_kernel<false, DKDV, 0, false>, bwd2_kernel<false, DKDV, 1, false>, bwd2_kernel<false, DKDV, 2, false>, nullptr,
        bwd2_kernel<false, DKDV, 4, false>},
       {bwd2_kernel<false, DKDV, 0, true>, bwd2_kernel<false, DKDV, 1, true>, bwd2_kernel<false, DKDV, 2, true>, nullptr, nullptr}},
      {{bwd2_kernel<true, DKDV, 0, false>, bwd2_kernel<true, DKDV, 1, false>, bwd2_kernel<true, DKDV, 2, false>, nullptr,
        bwd2_kernel<true, DKDV, 4, false>},
       {bwd2_kernel<true, DKDV, 0, true>, bwd2_kernel<true, DKDV, 1, true>, bwd2_kernel<true, DKDV, 2, true>, nullptr, nullptr}}};
  const int ni = (rope && rope->idx) ? rope->n_rdim / 8 : 0;
  const int bf = g->dtype == SWA_BF16 ? 1 : 0;
  const BwdKernel kern1 = v2 ? nullptr : fused_table[bf][pl.tab_bytes ? 1 : 0][ni];
  const StripKernel kern2 = v2 ? prerot_table[bf][p.qch == 1 && p.vch == 1 ? 1 : 0][ni] : nullptr;
  const void* kern = v2 ? (const void*)kern2 : (const void*)kern1;
  if (kern == nullptr) {
    snprintf(g_tc_err, sizeof(g_tc_err), "n_rdim %d has no tensor-core kernel", rope ? rope->n_rdim : 0);
    return -1;
  }
  CUtensorMap moqk, mov;                                     // outputs of the strip kernels
  if (v2) {
    if (!make_map(&moqk, out_qk, g, g->d_qk, pl.TW, pl.R4)) return -1;
    mov = moqk;
    if (DKDV && !make_map(&mov, out_v, g, g->d_v, pl.TW, pl.R4)) return -1;
  }
  cudaError_t e = allow_smem((const void*)kern);
  if (e != cudaSuccess) {
    snprintf(g_tc_err, sizeof(g_tc_err), "cudaFuncSetAttribute(%u bytes): %s", pl.smem_bytes, cudaGetErrorString(e));
    return -1;
  }
  if (knobs().verbose)
    fprintf(stderr, "[swa2d] %s plan: tile %dx%d, block %dx%d (N=%d), stages %d, nsb %d, nxb %d, %d quarters per chunk, tables %u, smem %u, %d items on %u CTAs\n",
            DKDV ? "dkdv" : "dq", pl.TH, pl.TW, pl.KR, pl.KW, pl.N, pl.stages, pl.nsb, pl.nxb, pl.nq, pl.tab_bytes, pl.smem_bytes, p.n_items, grid.x);
  if (v2) {
    e = launch_pdl(kern2, grid, block.x, pl.smem_bytes, st, mxqk, mxv, myqk, myv, moqk, mov, p, lse, delta);
    if (e != cudaSuccess) snprintf(g_tc_err, sizeof(g_tc_err), "launch: %s", cudaGetErrorString(e));
    return e == cudaSuccess ? 0 : -1;
  }
  kern1<<<grid, block, pl.smem_bytes, st>>>(mxqk, mxv, myqk, myv, p, lse, delta, make_view(out_qk),
                                            out_v ? make_view(out_v) : View4{nullptr, 0, 0, 0, 0});
  return 0;
}

}  // namespace

int launch_dq(const swa_geom_t* g, const swa_rope_t* rope, const swa_tensor_t* q, const swa_tensor_t* k,
              const swa_tensor_t* v, const swa_tensor_t* d_o, const float* lse, const float* delta,
              const swa_tensor_t* dq, int32_t* status, cudaStream_t st, bool prerotated) {
  return launch_bwd<false>(g, rope, prerotated, q, d_o, k, v, lse, delta, dq, nullptr, status, st);
}

int launch_dkdv(const swa_geom_t* g, const swa_rope_t* rope, const swa_tensor_t* q, const swa_tensor_t* k,
                const swa_tensor_t* v, const swa_tensor_t* d_o, const float* lse, const float* delta,
                const swa_tensor_t* dk, const swa_tensor_t* dv, int32_t* status, cudaStream_t st, bool prerotated) {
  return launch_bwd<true>(g, rope, prerotated, k, v, q, d_o, lse, delta, dk, dv, status, st);
}

}  // namespace tc
}  // namespace swa
