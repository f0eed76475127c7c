// fp32 attention on CUDA cores, tiled: forward, dQ and dK/dV for fp32 tensors with unit last stride, 16-byte aligned
// rows and head dims that are multiples of 4 up to 128 (anything else runs on swa_simt.cuh's one-warp-per-token kernels).
//
// A block of four warps owns 4 grid rows x 8 token columns, a warp 2 x 4 of them; the rows of the halo are staged in shared
// memory band by band (asynchronous copies) and shared by the warps.  A warp takes the streamed tokens of its own window 32
// at a time; lane (a, b), a < 4, b < 8, owns two resident rows, 2a and 2a + 1, throughout:
//   scores       of its two rows with the streamed tokens b, b + 8, ...: six 16-byte loads for 16 packed multiply-adds
//   accumulation of its two rows' head dims 4b .. 4b + 3 (and 32 further on): a 16-byte load per 4 head dims and token for
//                four packed multiply-adds, the 8 x 32 weights passed through shared memory, four tokens a load
// Latency bounds it -- 8 to 12 warps an SM, half of the issue slots and two thirds of the shared-memory wavefronts used --
// and what the bands cost: their barriers, and warps that wait for the one whose window has most of the band
// (tile_band_rows in swa_abi.cu).  In vain are scored the columns of the warp's halo beyond a row's own window,
// (4 + 2 wc) / (2 wc + 1), and one row in 2 wr + 2.  Training steps of 4 slices: 64 x 64, window 21, d = 64 641 -> 499 us, 32 x 32,
// window 31, d = 128 1091 -> 506 us against one streamed token per lane and four resident rows per warp.
#pragma once

#include "swa_simt.cuh"
#include "umma.cuh"

namespace swa {

constexpr int kTileRows = 4, kTileCols = 8, kTileWarps = 4, kTileThreads = kTileWarps * 32;
constexpr int kTileQ = 8;                          // resident rows of a warp: 2 grid rows x 4 columns
constexpr int kTileW = 36;                         // floats from one row of weights to the next

// Tensors of one launch; `kind` 0: forward (x1 = q; y1 = k, y2 = v; o1 = o), 1: dQ (x1 = q, x2 = dO; y1 = k, y2 = v; o1 = dq),
// 2: dK/dV (x1 = k, x2 = v; y1 = q, y2 = dO; o1 = dk, o2 = dv).
struct TileArgs {
  Geom g;
  RopeDev rope;          // inverse rotation of dQ / dK on the way out (idx == nullptr: none)
  View4 x1, x2, y1, y2, o1, o2;
  float* lse_out;        // forward
  const float *lse, *delta;
  View4 o;               // dQ with delta_out: the forward result; delta = rowsum(o * dO) of the block's own rows is made here
  float* delta_out;
  int rb, n_tiles_x, max_keys;   // halo rows per band, tiles per row of tiles, streamed tokens of the largest band
};

// Token columns of the halo of `cols` columns, not clipped to the grid.
inline int64_t tile_halo_cols(int cols, int64_t b, int64_t wc) { return ((cols + b - 2) / b + 1 + 2 * wc) * b; }

// Floats of shared memory of a launch with `keys` staged tokens.  All rows lie 4 floats further apart than they are long:
// rows at distance 1 (streamed) or 2 (resident) start in banks of their own.
__host__ __device__ __forceinline__ size_t tile_smem_floats(int kind, int d1, int d2, int keys) {
  const size_t resident = kTileWarps * kTileQ * (size_t)(kind == 0 ? d1 + 4 : d1 + 4 + d2 + 4);
  const size_t weights = (size_t)kTileWarps * (kTileQ * kTileW * (kind == 2 ? 2 : 1) + 32);
  return resident + weights + (size_t)keys * (d1 + 4 + d2 + 4) + (kind == 2 ? 2 * (size_t)keys : 0);
}

// out[e][i] = x_e . y_i for two resident rows (stride d + 4) and four streamed rows that lie off[i] floats into y.
__device__ __forceinline__ void tile_dot(const float* x, const float* y, const int (&off)[4], int d, float (&out)[2][4]) {
  using namespace ptx;
  uint64_t acc[2][4];
#pragma unroll
  for (int i = 0; i < 4; ++i) acc[0][i] = acc[1][i] = 0ull;
  const float *x1 = x + d + 4, *y0 = y + off[0], *y1 = y + off[1], *y2 = y + off[2], *y3 = y + off[3];
#pragma unroll 4
  for (int c = 0; c < d; c += 4) {
    const ulonglong2 a0 = *reinterpret_cast<const ulonglong2*>(x + c), a1 = *reinterpret_cast<const ulonglong2*>(x1 + c);
    const ulonglong2 b[4] = {*reinterpret_cast<const ulonglong2*>(y0 + c), *reinterpret_cast<const ulonglong2*>(y1 + c),
                             *reinterpret_cast<const ulonglong2*>(y2 + c), *reinterpret_cast<const ulonglong2*>(y3 + c)};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      acc[0][i] = f2_fma(a0.x, b[i].x, acc[0][i]);
      acc[1][i] = f2_fma(a1.x, b[i].x, acc[1][i]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      acc[0][i] = f2_fma(a0.y, b[i].y, acc[0][i]);
      acc[1][i] = f2_fma(a1.y, b[i].y, acc[1][i]);
    }
  }
#pragma unroll
  for (int e = 0; e < 2; ++e)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 v = f2_unpack(acc[e][i]);
      out[e][i] = v.x + v.y;
    }
}

// Accumulators of a lane: [its resident row][32-dim group][pair of head dims].
template <int G>
using TileAcc = uint64_t[2][G][2];

// acc[e] += w[e][k] * y[at[k]] over n staged tokens (rows `stride` floats apart); goff: the lane's head dims in
// each group.
template <int G>
__device__ __forceinline__ void tile_accumulate(TileAcc<G>& acc, const float* w, const int* at, const float* y, int stride,
                                                const int (&goff)[G], int n) {
  using namespace ptx;
#pragma unroll 2
  for (int k = 0; k < n; k += 4) {                               // (tokens beyond the last: weight 0, a valid position)
    const int4 at4 = *reinterpret_cast<const int4*>(at + k);
    const float4 u = *reinterpret_cast<const float4*>(w + k), v = *reinterpret_cast<const float4*>(w + kTileW + k);
    const int pos[4] = {at4.x, at4.y, at4.z, at4.w};
    const float wu[4] = {u.x, u.y, u.z, u.w}, wv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float* row = y + pos[i] * stride;
      const uint64_t w0 = f2_pack(wu[i], wu[i]), w1 = f2_pack(wv[i], wv[i]);
#pragma unroll
      for (int h = 0; h < G; ++h) {
        const ulonglong2 r = *reinterpret_cast<const ulonglong2*>(row + goff[h]);
        acc[0][h][0] = f2_fma(w0, r.x, acc[0][h][0]);
        acc[0][h][1] = f2_fma(w0, r.y, acc[0][h][1]);
        acc[1][h][0] = f2_fma(w1, r.x, acc[1][h][0]);
        acc[1][h][1] = f2_fma(w1, r.y, acc[1][h][1]);
      }
    }
  }
}

template <int G>
__device__ __forceinline__ void tile_scale(TileAcc<G>& acc, int e, float f) {
  const uint64_t ff = ptx::f2_pack(f, f);
#pragma unroll
  for (int h = 0; h < G; ++h) {
    acc[e][h][0] = ptx::f2_mul(acc[e][h][0], ff);
    acc[e][h][1] = ptx::f2_mul(acc[e][h][1], ff);
  }
}
// Row e of the lane's accumulators, times f, to `dst` (the row's first element, 16-byte aligned).
template <int G>
__device__ __forceinline__ void tile_store(const TileAcc<G>& acc, int e, float f, float* dst, int b4, int d) {
#pragma unroll
  for (int h = 0; h < G; ++h) {
    const float2 x = ptx::f2_unpack(acc[e][h][0]), y = ptx::f2_unpack(acc[e][h][1]);
    if (b4 + 32 * h < d) *reinterpret_cast<float4*>(dst + b4 + 32 * h) = make_float4(x.x * f, x.y * f, y.x * f, y.y * f);
  }
}

__device__ __forceinline__ void tile_copy16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void tile_copy_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Whether any of a row's sums is an infinity or a NaN.
template <int G>
__device__ __forceinline__ bool tile_not_finite(const TileAcc<G>& acc, int e) {
  uint64_t z = 0ull;
#pragma unroll
  for (int h = 0; h < G; ++h) z = ptx::f2_fma(acc[e][h][0], 0ull, ptx::f2_fma(acc[e][h][1], 0ull, z));
  const float2 v = ptx::f2_unpack(z);
  return !(v.x + v.y == 0.f);
}

// One row again, over the tokens of its own window only and straight from global memory.  A warp's 32 tokens hold some that a row
// does not see; their weight is 0, which is nothing to a sum until such a token holds an infinity or a NaN (0 * inf).  A row
// whose sums are not finite is therefore done anew, so that what it does not see cannot reach it, and what it does see
// still does.  x1, x2: the resident row; m, l: as in the kernel (forward: l the whole sum).  Results: forward to `dst`; else
// to x1 in shared memory (scaled, not yet rotated back), dV to `dst`.
template <int KIND>
__device__ __noinline__ void tile_row_again(const TileArgs& t, float* x1, const float* x2, float* dst, int rr, int cc, float m, float l) {
  const Geom& g = t.g;
  const int lane = threadIdx.x & 31, bh = blockIdx.y, bi = bh / g.H, hi = bh - bi * g.H, Wtok = g.tw * g.b, cell = cc / g.b;
  const float *y1 = (const float*)t.y1.ptr + bi * t.y1.s0 + hi * t.y1.s1, *y2 = (const float*)t.y2.ptr + bi * t.y2.s0 + hi * t.y2.s1;
  float acc[4] = {}, acc2[4] = {};
  for (int r = max(0, rr - g.wr); r <= min(g.th - 1, rr + g.wr); ++r)
    for (int c = max(0, cell - g.wc) * g.b; c < (min(g.tw - 1, cell + g.wc) + 1) * g.b; ++c) {
      const int64_t n = (int64_t)r * Wtok + c;
      const float *row1 = y1 + n * t.y1.s2, *row2 = y2 + n * t.y2.s2;
      float s = 0.f, dp = 0.f;
      for (int d = lane; d < g.dqk; d += 32) s = fmaf(x1[d], row1[d], s);
      s = warp_sum(s);
      float p, w;
      if constexpr (KIND == 0) {
        s *= g.scale_log2;
        w = p = s == -INFINITY ? 0.f : exp2f(s - m);
      } else {
        for (int d = lane; d < g.dv; d += 32) dp = fmaf(x2[d], row2[d], dp);
        dp = warp_sum(dp);
        const float ls = KIND == 1 ? m : t.lse[(int64_t)bh * g.th * Wtok + n], de = KIND == 1 ? l : t.delta[(int64_t)bh * g.th * Wtok + n];
        p = exp2f(fmaf(s, g.scale_log2, -ls));
        w = p * (dp - de);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int d = lane + 32 * i;
        if (d < (KIND == 0 ? g.dv : g.dqk)) acc[i] = fmaf(w, KIND == 0 ? row2[d] : row1[d], acc[i]);
        if (KIND == 2 && d < g.dv) acc2[i] = fmaf(p, row2[d], acc2[i]);
      }
    }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int d = lane + 32 * i;
    if (KIND == 0 && d < g.dv) dst[d] = acc[i] * (1.f / l);
    if (KIND != 0 && d < g.dqk) x1[d] = acc[i] * g.sm_scale;
    if (KIND == 2 && d < g.dv) dst[d] = acc2[i];
  }
}

// KIND as in TileArgs; G1 / G2: 32-dim groups of the q-k / v tensors (dQ: only G1 is used, forward: only G2).
template <int KIND, int G1, int G2>
__global__ void __launch_bounds__(kTileThreads, 3) simt_tile_kernel(const __grid_constant__ TileArgs t) {
  extern __shared__ __align__(16) float tile_smem[];
  constexpr int WSETS = KIND == 2 ? 2 : 1;
  const Geom& g = t.g;
  const int d1 = g.dqk, d2 = g.dv, s1 = d1 + 4, s2 = d2 + 4, Wtok = g.tw * g.b;
  float* x1 = tile_smem;                                         // resident rows [warp][8][d + 4]
  float* x2 = x1 + kTileWarps * kTileQ * s1;
  float* wbuf = KIND == 0 ? x2 : x2 + kTileWarps * kTileQ * s2;  // weights [warp][1 or 2][8][36]
  int* at_all = reinterpret_cast<int*>(wbuf + kTileWarps * kTileQ * kTileW * WSETS);   // positions of a warp's 32 tokens in the band
  float* y1 = reinterpret_cast<float*>(at_all + kTileWarps * 32);                      // staged tokens
  float* y2 = y1 + t.max_keys * s1;
  float* vec = y2 + t.max_keys * s2;                             // dK/dV: their lse, delta
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, a = lane >> 3, b = lane & 7, b4 = 4 * b;
  const int bh = blockIdx.y, bi = bh / g.H, hi = bh - bi * g.H;
  const int ty = blockIdx.x / t.n_tiles_x, r0 = ty * kTileRows, c0 = (blockIdx.x - ty * t.n_tiles_x) * kTileCols;
  auto slice = [&](const View4& v) { return (float*)v.ptr + bi * v.s0 + hi * v.s1; };

  // the warp's corner; the lane's rows: columns my_c and my_c + 1 of grid row my_r
  const int wr0 = r0 + (warp >> 1) * 2, wc0 = c0 + (warp & 1) * 4, my_r = wr0 + (a >> 1), my_c = wc0 + (a & 1) * 2;
  const bool on = wr0 < g.th && wc0 < Wtok;
  const int n_out = my_r < g.th ? min(2, max(0, Wtok - my_c)) : 0;           // rows of this lane inside the grid
  float* const mx1 = x1 + (warp * kTileQ + 2 * a) * s1;
  float* const mx2 = x2 + (warp * kTileQ + 2 * a) * s2;
  float* const w1 = wbuf + (warp * kTileQ * WSETS + 2 * a) * kTileW;
  float* const w2 = w1 + kTileQ * kTileW;
  int* const at = at_all + warp * 32;
  const int64_t row_base = (int64_t)bh * g.th * Wtok + (int64_t)my_r * Wtok + my_c;

  // halo of the block and of the warp, clipped to the grid
  const int x_lo = max(0, (c0 / g.b - g.wc) * g.b), x_hi = min(Wtok, ((min(c0 + kTileCols, Wtok) - 1) / g.b + g.wc + 1) * g.b);
  const int h_lo = max(0, r0 - g.wr), h_hi = min(g.th - 1, min(r0 + kTileRows, g.th) - 1 + g.wr), nc = x_hi - x_lo;
  const int wx_lo = max(0, (wc0 / g.b - g.wc) * g.b), wx_hi = min(Wtok, ((min(wc0 + 4, Wtok) - 1) / g.b + g.wc + 1) * g.b);
  const int wnc = max(1, wx_hi - wx_lo);
  const uint32_t nc_inv = (0x1000000u + nc - 1) / nc, wnc_inv = (0x1000000u + wnc - 1) / wnc;   // n / nc == (n * nc_inv) >> 24 for n < 4096

  pdl_enter();
  pdl_wait();
  // rows are copied by groups of 8, 16 or 32 lanes, a 16-byte unit each
  auto lanes_log = [](int d) { return d <= 32 ? 3 : d <= 64 ? 4 : 5; };
  auto load_resident = [&](float* dst, const View4& v, int d) {
    const float* src = slice(v);
    const int lg = lanes_log(d), c = (tid & ((1 << lg) - 1)) * 4;
    if (c >= d) return;
    for (int row = tid >> lg; row < kTileWarps * kTileQ; row += kTileThreads >> lg) {      // row: warp * 8 + (grid row, column) in the warp
      const int rr = r0 + (row >> 4) * 2 + ((row >> 2) & 1), cc = c0 + ((row >> 3) & 1) * 4 + (row & 3);
      float* to = dst + row * (d + 4) + c;
      if (rr < g.th && cc < Wtok) tile_copy16(to, src + ((int64_t)rr * Wtok + cc) * v.s2 + c);
      else *reinterpret_cast<float4*>(to) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  load_resident(x1, t.x1, d1);
  if constexpr (KIND != 0) load_resident(x2, t.x2, d2);

  float m[2], l[2];                  // forward: running maximum (the same in all lanes of a row), this lane's part of the sum; dQ: lse, delta
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    m[e] = KIND == 1 ? 0.f : -INFINITY;
    l[e] = 0.f;
    if constexpr (KIND == 1) {
      if (e < n_out) {
        m[e] = t.lse[row_base + e];
        if (!t.delta_out) l[e] = t.delta[row_base + e];
      }
    }
  }
  constexpr int GA = KIND == 0 ? G2 : G1, GB = KIND == 2 ? G2 : 1;
  TileAcc<GA> acc;
  [[maybe_unused]] TileAcc<GB> acc2;
  int goff[GA];
  [[maybe_unused]] int goff2[GB];
#pragma unroll
  for (int h = 0; h < GA; ++h) {                                 // head dims beyond the row: some that exist, sums unused
    acc[0][h][0] = acc[0][h][1] = acc[1][h][0] = acc[1][h][1] = 0ull;
    goff[h] = b4 + 32 * h < (KIND == 0 ? d2 : d1) ? b4 + 32 * h : 0;
  }
#pragma unroll
  for (int h = 0; h < GB; ++h) {
    acc2[0][h][0] = acc2[0][h][1] = acc2[1][h][0] = acc2[1][h][1] = 0ull;
    goff2[h] = b4 + 32 * h < d2 ? b4 + 32 * h : 0;
  }

  for (int b0 = h_lo; b0 <= h_hi; b0 += t.rb) {
    const int b1 = min(b0 + t.rb - 1, h_hi), n_band = (b1 - b0 + 1) * nc;
    __syncthreads();                                             // nobody still reads the previous band
    auto load_band = [&](float* dst, const View4& v, int d, int s) {
      const float* src = slice(v) + ((int64_t)b0 * Wtok + x_lo) * v.s2;
      const int lg = lanes_log(d), c = (tid & ((1 << lg) - 1)) * 4;
      if (c >= d) return;
#pragma unroll 4
      for (int n = tid >> lg; n < n_band; n += kTileThreads >> lg) {
        const int rr = (int)(((uint64_t)(uint32_t)n * nc_inv) >> 24);
        tile_copy16(dst + n * s + c, src + (int64_t)(rr * (Wtok - nc) + n) * v.s2 + c);
      }
    };
    load_band(y1, t.y1, d1, s1);
    load_band(y2, t.y2, d2, s2);
    if constexpr (KIND == 2) {
      for (int i = tid; i < n_band; i += kTileThreads) {
        const int rr = (int)(((uint64_t)(uint32_t)i * nc_inv) >> 24);
        const int64_t src = (int64_t)bh * g.th * Wtok + (int64_t)(b0 + rr) * Wtok + x_lo + i - rr * nc;
        vec[i] = t.lse[src];
        vec[t.max_keys + i] = t.delta[src];
      }
    }
    if constexpr (KIND == 1) {
      if (t.delta_out && b0 == h_lo) {                           // (while the first band is on its way)
        const int64_t row = (int64_t)my_r * Wtok + my_c;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float *po = slice(t.o) + (row + e) * t.o.s2, *pd = slice(t.x2) + (row + e) * t.x2.s2;
          float sum = 0.f;
          for (int c = b4; e < n_out && c < d2; c += 32) {
            const float4 x = *reinterpret_cast<const float4*>(po + c), y = *reinterpret_cast<const float4*>(pd + c);
            sum += x.x * y.x + x.y * y.y + x.z * y.z + x.w * y.w;
          }
#pragma unroll
          for (int o = 4; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
          l[e] = sum;
          if (b == 0 && e < n_out) t.delta_out[row_base + e] = sum;
        }
      }
    }
    tile_copy_wait();
    __syncthreads();
    const int f0 = max(b0, wr0 - g.wr), f1 = min(b1, wr0 + 1 + g.wr);        // this warp's rows of the band
    if (!on || f0 > f1) continue;
    const int n0 = (f0 - b0) * nc + wx_lo - x_lo, n_all = (f1 - f0 + 1) * wnc;
#pragma unroll 1
    for (int k0 = 0; k0 < n_all; k0 += 32) {
      const int cnt = min(32, n_all - k0);
      int n[4], off[4];
      uint32_t see = 0;                                          // bit 4 e + i: row e of the lane and token i see each other
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int k = min(k0 + b + 8 * i, n_all - 1);
        const int kr = (int)(((uint64_t)(uint32_t)k * wnc_inv) >> 24), yx = wx_lo + k - kr * wnc, yc = g.b == 1 ? yx : yx / g.b;
        n[i] = n0 + kr * (nc - wnc) + k;
        off[i] = n[i] * s1;
        const int lo = (yc - g.wc) * g.b - my_c, last = (yc + g.wc + 1) * g.b - 1 - my_c;  // columns the token may interact with
        const bool row = (uint32_t)(f0 + kr - my_r + g.wr) <= (uint32_t)(2 * g.wr) && b + 8 * i < cnt;
        if (row && lo <= 0 && last >= 0) see |= 1u << i;
        if (row && lo <= 1 && last >= 1) see |= 16u << i;
        if (a == 0) at[b + 8 * i] = n[i];
      }
      float s[2][4];
      tile_dot(mx1, y1, off, d1, s);
      if constexpr (KIND == 0) {
        float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            s[e][i] = see >> (4 * e + i) & 1 ? s[e][i] * g.scale_log2 : -INFINITY;
            mx[e] = fmaxf(mx[e], s[e][i]);
          }
        // the maximum is renewed only when a score passes it by more than 2^16: fp32 has the range to spare
        const bool grow = mx[0] > m[0] + 16.f || mx[1] > m[1] + 16.f;        // (no maximum yet: -INFINITY + 16 is that still)
        if (__any_sync(0xffffffffu, grow)) {
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            float v = mx[e];
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
            const float mn = fmaxf(m[e], v), f = m[e] == -INFINITY ? 0.f : exp2f(m[e] - mn);
            m[e] = mn;
            l[e] *= f;
            tile_scale<GA>(acc, e, f);
          }
        }
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            s[e][i] = s[e][i] == -INFINITY ? 0.f : exp2f(s[e][i] - m[e]);
            l[e] += s[e][i];
          }
      } else {
        float dp[2][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) off[i] = n[i] * s2;
        tile_dot(mx2, y2, off, d2, dp);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float ls = KIND == 2 ? vec[n[i]] : 0.f, de = KIND == 2 ? vec[t.max_keys + n[i]] : 0.f;
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const float p = see >> (4 * e + i) & 1 ? exp2f(fmaf(s[e][i], g.scale_log2, -(KIND == 1 ? m[e] : ls))) : 0.f;
            s[e][i] = p * (dp[e][i] - (KIND == 1 ? l[e] : de));
            if constexpr (KIND == 2) w2[e * kTileW + b + 8 * i] = p;
          }
        }
      }
#pragma unroll
      for (int e = 0; e < 2; ++e)
#pragma unroll
        for (int i = 0; i < 4; ++i) w1[e * kTileW + b + 8 * i] = s[e][i];
      __syncwarp();
      if constexpr (KIND == 0) {
        tile_accumulate<GA>(acc, w1, at, y2, s2, goff, cnt);
      } else {
        tile_accumulate<GA>(acc, w1, at, y1, s1, goff, cnt);
        if constexpr (KIND == 2) tile_accumulate<GB>(acc2, w2, at, y2, s2, goff2, cnt);
      }
      __syncwarp();
    }
  }
  if (!on) return;

  // rows of this warp whose sums are not finite (bit e of the lanes' byte): done again (tile_row_again)
  uint32_t again[2];
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    bool bad = tile_not_finite<GA>(acc, e);
    if constexpr (KIND == 2) bad |= tile_not_finite<GB>(acc2, e);
    again[e] = __ballot_sync(0xffffffffu, bad && e < n_out);
    if constexpr (KIND == 0) {
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) l[e] += __shfl_xor_sync(0xffffffffu, l[e], o);
    }
  }
  auto redo = [&](int e) { return (again[e] >> (8 * a) & 255u) != 0; };
  if (again[0] | again[1]) {
#pragma unroll 1
    for (int j = 0; j < kTileQ; ++j) {
      const float mj = __shfl_sync(0xffffffffu, j & 1 ? m[1] : m[0], 4 * (j & 6)), lj = __shfl_sync(0xffffffffu, j & 1 ? l[1] : l[0], 4 * (j & 6));
      if (!((j & 1 ? again[1] : again[0]) >> (4 * (j & 6)) & 255u)) continue;
      const int rr = wr0 + (j >> 2), cc = wc0 + (j & 3), row = warp * kTileQ + j;
      const View4& o = KIND == 0 ? t.o1 : t.o2;
      tile_row_again<KIND>(t, x1 + row * s1, x2 + row * s2, KIND == 1 ? nullptr : slice(o) + ((int64_t)rr * Wtok + cc) * o.s2, rr, cc, mj, lj);
    }
    __syncwarp();
  }

  // out: accumulators scaled, rotated back where asked, rows of this warp
  if constexpr (KIND == 0) {
    float* dst = slice(t.o1) + ((int64_t)my_r * Wtok + my_c) * t.o1.s2;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      if (e >= n_out) continue;
      if (!redo(e)) tile_store<GA>(acc, e, 1.f / l[e], dst + e * t.o1.s2, b4, d2);
      if (b == 0) t.lse_out[row_base + e] = m[e] + log2f(l[e]);
    }
  } else {
    __syncwarp();
#pragma unroll
    for (int e = 0; e < 2; ++e)
      if (!redo(e)) tile_store<GA>(acc, e, g.sm_scale, mx1 + e * s1, b4, d1);   // the resident rows are done with: they take the result
    __syncwarp();
    float* dst = slice(t.o1);
#pragma unroll 1
    for (int j = 0; j < kTileQ; ++j) {
      const int rr = wr0 + (j >> 2), cc = wc0 + (j & 3);
      if (rr >= g.th || cc >= Wtok) continue;
      int irow = -1, icol = -1;
      if (t.rope.idx) decode_idx(t.rope.idx[rr * Wtok + cc], t.rope.max_h, t.rope.max_w, irow, icol);
      for (int d = lane; d < d1; d += 32)
        dst[((int64_t)rr * Wtok + cc) * t.o1.s2 + d] = load_rot<float>(x1 + (warp * kTileQ + j) * s1, 1, d, t.rope, irow, icol, -1.f);
    }
    if constexpr (KIND == 2) {
      float* dst2 = slice(t.o2) + ((int64_t)my_r * Wtok + my_c) * t.o2.s2;
#pragma unroll
      for (int e = 0; e < 2; ++e)
        if (e < n_out && !redo(e)) tile_store<GB>(acc2, e, 1.f, dst2 + e * t.o2.s2, b4, d2);
    }
  }
}

}  // namespace swa
