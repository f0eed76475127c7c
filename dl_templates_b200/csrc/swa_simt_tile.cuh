// fp32 attention on CUDA cores, tiled: forward, dQ and dK/dV for fp32 tensors with unit last stride, 16-byte aligned
// rows and head dims that are multiples of 4 up to 128 (anything else runs on swa_simt.cuh's one-warp-per-token kernels).
//
// A block of eight warps owns 4 grid rows x 8 token columns, a warp 4 columns of a row; the rows of the halo are staged in
// shared memory band by band (asynchronous copies) and shared by the warps.  A warp takes the streamed tokens of its own
// window 32 at a time:
//   scores       lane = streamed token, 4 resident rows read as broadcasts: one 16-byte load of the token's row and
//                four broadcasts per 8 packed multiply-adds
//   accumulation lane = 2 or 4 head dims, the 32 x 4 weights passed through shared memory: one broadcast and one
//                8- or 16-byte load per 4 or 8 packed multiply-adds
// Multiply-adds and shared-memory wavefronts (about as many cycles each) bound it once there are warps enough: three
// blocks share an SM.  Only the columns of the warp's halo are scored in vain, (4 + 2 wc) / (2 wc + 1).
#pragma once

#include "swa_simt.cuh"
#include "umma.cuh"

namespace swa {

constexpr int kTileRows = 4, kTileCols = 8, kTileQ = 4, kTileWarps = 8;
constexpr int kTileTokens = kTileRows * kTileCols;

// Tensors of one launch; `kind` 0: forward (x1 = q; y1 = k, y2 = v; o1 = o), 1: dQ (x1 = q, x2 = dO; y1 = k, y2 = v; o1 = dq),
// 2: dK/dV (x1 = k, x2 = v; y1 = q, y2 = dO; o1 = dk, o2 = dv).
struct TileArgs {
  Geom g;
  RopeDev rope;          // inverse rotation of dQ / dK on the way out (idx == nullptr: none)
  View4 x1, x2, y1, y2, o1, o2;
  float* lse_out;        // forward
  const float *lse, *delta;
  int rb, n_tiles_x, max_keys;   // halo rows per band, tiles per row of tiles, streamed tokens of the largest band
};

__host__ __device__ __forceinline__ int tile_halo_cols(int b, int wc) { return ((kTileCols + b - 2) / b + 1 + 2 * wc) * b; }

// Floats of shared memory of a launch with `keys` staged tokens.
__host__ __device__ __forceinline__ size_t tile_smem_floats(int kind, int d1, int d2, int keys) {
  const size_t resident = kTileTokens * (size_t)(kind == 0 ? d1 : d1 + d2);
  const size_t weights = (size_t)kTileWarps * 32 * (kTileQ * (kind == 2 ? 2 : 1) + 1);
  return resident + weights + (size_t)keys * (d1 + 4 + d2 + 4) + (kind == 2 ? 2 * (size_t)keys : 0);
}

// out[j] = x_j . y for the warp's resident rows x (stride d) and this lane's streamed row y.
__device__ __forceinline__ void tile_dot(const float* x, const float* y, int d, float* out) {
  using namespace ptx;
  uint64_t acc[kTileQ];
#pragma unroll
  for (int j = 0; j < kTileQ; ++j) acc[j] = 0ull;
#pragma unroll 4
  for (int c = 0; c < d; c += 4) {
    const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(y + c);
#pragma unroll
    for (int j = 0; j < kTileQ; ++j) {
      const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(x + j * d + c);
      acc[j] = f2_fma(a.x, b.x, acc[j]);
      acc[j] = f2_fma(a.y, b.y, acc[j]);
    }
  }
#pragma unroll
  for (int j = 0; j < kTileQ; ++j) {
    const float2 v = f2_unpack(acc[j]);
    out[j] = v.x + v.y;
  }
}

// acc[dd][jp] += w[k][2 jp, 2 jp + 1] * y[at[k]][dd] over n staged tokens (at: their positions; rows `stride` floats apart).
template <int P>
__device__ __forceinline__ void tile_accumulate(uint64_t (&acc)[P][2], const float* w, const int* at, const float* y, int stride, int n) {
  using namespace ptx;
  auto one = [&](int k, int pos) {
    const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(w + kTileQ * k);
    const float* row = y + pos * stride;
    float v[P];
    if constexpr (P == 2) {
      const float2 t = *reinterpret_cast<const float2*>(row);
      v[0] = t.x; v[1] = t.y;
    } else {
      const float4 t = *reinterpret_cast<const float4*>(row);
      v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    }
#pragma unroll
    for (int dd = 0; dd < P; ++dd) {
      const uint64_t vv = f2_pack(v[dd], v[dd]);
      acc[dd][0] = f2_fma(a.x, vv, acc[dd][0]);
      acc[dd][1] = f2_fma(a.y, vv, acc[dd][1]);
    }
  };
#pragma unroll 2
  for (int k = 0; k < n; k += 4) {                               // (tokens beyond the last: weight 0, a valid position)
    const int4 pos = *reinterpret_cast<const int4*>(at + k);
    one(k, pos.x);
    one(k + 1, pos.y);
    one(k + 2, pos.z);
    one(k + 3, pos.w);
  }
}

template <int P>
__device__ __forceinline__ void tile_clear(uint64_t (&acc)[P][2]) {
#pragma unroll
  for (int dd = 0; dd < P; ++dd) acc[dd][0] = acc[dd][1] = 0ull;
}
// Element j of a lane's accumulators of head dim dd.
template <int P>
__device__ __forceinline__ float tile_get(const uint64_t (&acc)[P][2], int dd, int j) {
  const float2 v = ptx::f2_unpack(acc[dd][j >> 1]);
  return j & 1 ? v.y : v.x;
}

__device__ __forceinline__ void tile_copy16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void tile_copy_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// KIND as in TileArgs; P1 / P2: head dims of the q-k / v tensors per lane (2: up to 64, 4: up to 128).
template <int KIND, int P1, int P2>
__global__ void __launch_bounds__(kTileWarps * 32, 3) simt_tile_kernel(const __grid_constant__ TileArgs t) {
  using namespace ptx;
  extern __shared__ __align__(16) float tile_smem[];
  constexpr int Q = kTileQ, WSETS = KIND == 2 ? 2 : 1;
  const Geom& g = t.g;
  const int d1 = g.dqk, d2 = g.dv, s1 = d1 + 4, s2 = d2 + 4, Wtok = g.tw * g.b;
  float* x1 = tile_smem;                                         // resident rows [32][d]
  float* x2 = x1 + kTileTokens * d1;
  float* wbuf = KIND == 0 ? x2 : x2 + kTileTokens * d2;          // weights [warp][1 or 2][32][4]
  int* at_all = reinterpret_cast<int*>(wbuf + kTileWarps * 32 * Q * WSETS);   // positions of a warp's 32 tokens in the band
  float* y1 = reinterpret_cast<float*>(at_all + kTileWarps * 32);             // staged tokens
  float* y2 = y1 + t.max_keys * s1;
  float* vec = y2 + t.max_keys * s2;                             // dK/dV: their lse, delta
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int bh = blockIdx.y, bi = bh / g.H, hi = bh - bi * g.H;
  const int ty = blockIdx.x / t.n_tiles_x, r0 = ty * kTileRows, c0 = (blockIdx.x - ty * t.n_tiles_x) * kTileCols;
  auto slice = [&](const View4& v) { return (float*)v.ptr + bi * v.s0 + hi * v.s1; };

  const int my_r = r0 + (warp >> 1), my_c = c0 + (warp & 1) * Q;
  const bool on = my_r < g.th && my_c < Wtok;
  float* const mx1 = x1 + warp * Q * d1;
  float* const mx2 = x2 + warp * Q * d2;
  float* const w1 = wbuf + warp * 32 * Q * WSETS;
  float* const w2 = w1 + 32 * Q;
  int* const at = at_all + warp * 32;
  const int64_t row_base = (int64_t)bh * g.th * Wtok + (int64_t)my_r * Wtok + my_c;

  // halo of the block and of the warp, clipped to the grid
  const int x_lo = max(0, (c0 / g.b - g.wc) * g.b), x_hi = min(Wtok, ((min(c0 + kTileCols, Wtok) - 1) / g.b + g.wc + 1) * g.b);
  const int h_lo = max(0, r0 - g.wr), h_hi = min(g.th - 1, min(r0 + kTileRows, g.th) - 1 + g.wr), nc = x_hi - x_lo;
  const int wx_lo = max(0, (my_c / g.b - g.wc) * g.b), wx_hi = min(Wtok, ((min(my_c + Q, Wtok) - 1) / g.b + g.wc + 1) * g.b);
  const int wnc = max(1, wx_hi - wx_lo);
  const uint32_t nc_inv = (0x1000000u + nc - 1) / nc, wnc_inv = (0x1000000u + wnc - 1) / wnc;   // n / nc == (n * nc_inv) >> 24 for n < 4096

  // rows are copied by groups of 8, 16 or 32 lanes, a 16-byte unit each
  auto lanes_log = [](int d) { return d <= 32 ? 3 : d <= 64 ? 4 : 5; };
  pdl_enter();
  pdl_wait();
  auto load_resident = [&](float* dst, const View4& v, int d) {
    const float* src = slice(v);
    const int lg = lanes_log(d), c = (tid & ((1 << lg) - 1)) * 4;
    if (c >= d) return;
    for (int row = tid >> lg; row < kTileTokens; row += kTileWarps * 32 >> lg) {      // row: warp * 4 + column in the warp
      const int rr = r0 + (row >> 3), cc = c0 + (row & 7);
      if (rr < g.th && cc < Wtok) tile_copy16(dst + row * d + c, src + ((int64_t)rr * Wtok + cc) * v.s2 + c);
      else *reinterpret_cast<float4*>(dst + row * d + c) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  load_resident(x1, t.x1, d1);
  if constexpr (KIND != 0) load_resident(x2, t.x2, d2);

  float m[Q], l[Q];                  // forward: running maximum (the same in all lanes), this lane's part of the sum; dQ: lse, delta
#pragma unroll
  for (int j = 0; j < Q; ++j) {
    m[j] = -INFINITY;
    l[j] = 0.f;
    if constexpr (KIND == 1) {
      m[j] = 0.f;
      if (on && my_c + j < Wtok) {
        m[j] = t.lse[row_base + j];
        l[j] = t.delta[row_base + j];
      }
    }
  }
  constexpr int PA = KIND == 0 ? P2 : P1;
  uint64_t acc[PA][2];
  [[maybe_unused]] uint64_t acc2[P2][2];
  tile_clear(acc);
  if constexpr (KIND == 2) tile_clear(acc2);
  const int ca = lane * PA < (KIND == 0 ? d2 : d1) ? lane * PA : 0;          // this lane's head dims (lanes beyond them: idle copies)
  [[maybe_unused]] const int ca2 = lane * P2 < d2 ? lane * P2 : 0;

  for (int b0 = h_lo; b0 <= h_hi; b0 += t.rb) {
    const int b1 = min(b0 + t.rb - 1, h_hi), n_band = (b1 - b0 + 1) * nc;
    __syncthreads();                                             // nobody still reads the previous band
    auto load_band = [&](float* dst, const View4& v, int d, int s) {
      const float* src = slice(v) + ((int64_t)b0 * Wtok + x_lo) * v.s2;
      const int lg = lanes_log(d), c = (tid & ((1 << lg) - 1)) * 4;
      if (c >= d) return;
#pragma unroll 2
      for (int n = tid >> lg; n < n_band; n += kTileWarps * 32 >> lg) {
        const int rr = (int)(((uint64_t)(uint32_t)n * nc_inv) >> 24);
        tile_copy16(dst + n * s + c, src + (int64_t)(rr * (Wtok - nc) + n) * v.s2 + c);
      }
    };
    load_band(y1, t.y1, d1, s1);
    load_band(y2, t.y2, d2, s2);
    if constexpr (KIND == 2) {
      for (int i = tid; i < n_band; i += kTileWarps * 32) {
        const int rr = (int)(((uint64_t)(uint32_t)i * nc_inv) >> 24);
        const int64_t src = (int64_t)bh * g.th * Wtok + (int64_t)(b0 + rr) * Wtok + x_lo + i - rr * nc;
        vec[i] = t.lse[src];
        vec[t.max_keys + i] = t.delta[src];
      }
    }
    tile_copy_wait();
    __syncthreads();
    const int f0 = max(b0, my_r - g.wr), f1 = min(b1, my_r + g.wr);          // this warp's rows of the band
    if (!on || f0 > f1) continue;
    const int n0 = (f0 - b0) * nc + wx_lo - x_lo, n_all = (f1 - f0 + 1) * wnc;
#pragma unroll 1
    for (int k0 = 0; k0 < n_all; k0 += 32) {
      const int cnt = min(32, n_all - k0), k = min(k0 + lane, n_all - 1);
      const int kr = (int)(((uint64_t)(uint32_t)k * wnc_inv) >> 24), yx = wx_lo + k - kr * wnc, n = n0 + kr * (nc - wnc) + k;
      const int yc = g.b == 1 ? yx : yx / g.b;
      int lo = (yc - g.wc) * g.b - my_c, hi_ = (yc + g.wc + 1) * g.b - 1 - my_c;   // resident columns this token may interact with
      if (lane >= cnt) hi_ = -1;
      at[lane] = n;
      float s[Q];
      tile_dot(mx1, y1 + n * s1, d1, s);
      if constexpr (KIND == 0) {
        bool grow = false;
#pragma unroll
        for (int j = 0; j < Q; ++j) {
          s[j] = j >= lo && j <= hi_ ? s[j] * g.scale_log2 : -INFINITY;
          grow = grow || s[j] > m[j] + 16.f || (m[j] == -INFINITY && s[j] > -INFINITY);
        }
        // the maximum is renewed only when a score passes it by more than 2^16: fp32 has the range to spare
        if (__any_sync(0xffffffffu, grow)) {
          float a[Q];
#pragma unroll
          for (int j = 0; j < Q; ++j) {
            float v = s[j];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
            const float mn = fmaxf(m[j], v);
            a[j] = m[j] == -INFINITY ? 0.f : exp2f(m[j] - mn);
            m[j] = mn;
            l[j] *= a[j];
          }
          const uint64_t fa = f2_pack(a[0], a[1]), fb = f2_pack(a[2], a[3]);
#pragma unroll
          for (int dd = 0; dd < PA; ++dd) {
            acc[dd][0] = f2_mul(acc[dd][0], fa);
            acc[dd][1] = f2_mul(acc[dd][1], fb);
          }
        }
#pragma unroll
        for (int j = 0; j < Q; ++j) {
          s[j] = s[j] == -INFINITY ? 0.f : exp2f(s[j] - m[j]);
          l[j] += s[j];
        }
      } else {
        float dp[Q];
        tile_dot(mx2, y2 + n * s2, d2, dp);
        const float ls = KIND == 2 ? vec[n] : 0.f, de = KIND == 2 ? vec[t.max_keys + n] : 0.f;
#pragma unroll
        for (int j = 0; j < Q; ++j) {
          const bool see = j >= lo && j <= hi_;
          const float p = see ? exp2f(fmaf(s[j], g.scale_log2, -(KIND == 1 ? m[j] : ls))) : 0.f;
          s[j] = p * (dp[j] - (KIND == 1 ? l[j] : de));
          dp[j] = p;
        }
        if constexpr (KIND == 2) *reinterpret_cast<float4*>(w2 + lane * Q) = make_float4(dp[0], dp[1], dp[2], dp[3]);
      }
      *reinterpret_cast<float4*>(w1 + lane * Q) = make_float4(s[0], s[1], s[2], s[3]);
      __syncwarp();
      if constexpr (KIND == 0) {
        tile_accumulate<PA>(acc, w1, at, y2 + ca, s2, cnt);
      } else {
        tile_accumulate<PA>(acc, w1, at, y1 + ca, s1, cnt);
        if constexpr (KIND == 2) tile_accumulate<P2>(acc2, w2, at, y2 + ca2, s2, cnt);
      }
      __syncwarp();
    }
  }
  if (!on) return;

  // out: accumulators scaled, rotated back where asked, rows of this warp
  if constexpr (KIND == 0) {
    float* dst = slice(t.o1) + ((int64_t)my_r * Wtok + my_c) * t.o1.s2;
#pragma unroll
    for (int j = 0; j < Q; ++j) {
      const float lt = warp_sum(l[j]), inv = 1.f / lt;
      if (my_c + j >= Wtok) continue;
#pragma unroll
      for (int dd = 0; dd < PA; ++dd)
        if (lane * PA + dd < d2) dst[j * t.o1.s2 + lane * PA + dd] = tile_get(acc, dd, j) * inv;
      if (lane == 0) t.lse_out[row_base + j] = m[j] + log2f(lt);
    }
  } else {
    float* dst = slice(t.o1) + ((int64_t)my_r * Wtok + my_c) * t.o1.s2;
    __syncwarp();
#pragma unroll
    for (int j = 0; j < Q; ++j)                                  // the resident rows are done with: they take the result
#pragma unroll
      for (int dd = 0; dd < PA; ++dd)
        if (lane * PA + dd < d1) mx1[j * d1 + lane * PA + dd] = tile_get(acc, dd, j) * g.sm_scale;
    __syncwarp();
#pragma unroll 1
    for (int j = 0; j < Q; ++j) {
      if (my_c + j >= Wtok) break;
      int irow = -1, icol = -1;
      if (t.rope.idx) decode_idx(t.rope.idx[my_r * Wtok + my_c + j], t.rope.max_h, t.rope.max_w, irow, icol);
      for (int d = lane; d < d1; d += 32) dst[j * t.o1.s2 + d] = load_rot<float>(mx1 + j * d1, 1, d, t.rope, irow, icol, -1.f);
    }
    if constexpr (KIND == 2) {
      float* dst2 = slice(t.o2) + ((int64_t)my_r * Wtok + my_c) * t.o2.s2;
#pragma unroll
      for (int j = 0; j < Q; ++j) {
        if (my_c + j >= Wtok) continue;
#pragma unroll
        for (int dd = 0; dd < P2; ++dd)
          if (lane * P2 + dd < d2) dst2[j * t.o2.s2 + lane * P2 + dd] = tile_get(acc2, dd, j);
      }
    }
  }
}

}  // namespace swa
