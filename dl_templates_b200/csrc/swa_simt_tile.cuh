// fp32 attention on CUDA cores, tiled: forward, dQ and dK/dV for fp32 tensors with unit last stride, 16-byte aligned
// rows and head dims that are multiples of 4 up to 128 (anything else runs on swa_simt.cuh's one-warp-per-token kernels).
//
// A block of eight warps owns 8 grid rows x 8 token columns, one warp per row; the rows of the halo are staged in shared
// memory band by band and shared by the warps.  A warp takes the streamed tokens of its own window rows 32 at a time:
//   scores       lane = streamed token, 8 resident rows read as broadcasts: one 16-byte load of the token's row and
//                eight broadcasts per 16 packed multiply-adds
//   accumulation lane = 2 or 4 head dims, the 32 x 8 weights passed through shared memory: two broadcasts and one
//                8- or 16-byte load per 8 or 16 packed multiply-adds
// Shared-memory wavefronts (about 1.25 per multiply-add issue slot) bound it; only the columns of the halo are scored in
// vain, (8 + 2 wc) / (2 wc + 1).  One warp per token, with a butterfly per score, needed some 30 instructions for what
// are 4 here.  All products and sums are fp32.
#pragma once

#include "swa_simt.cuh"
#include "umma.cuh"

namespace swa {

constexpr int kTileRows = 8, kTileCols = 8;

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
  const size_t resident = 64 * (size_t)(kind == 0 ? d1 : d1 + d2);
  const size_t weights = (size_t)kTileRows * 32 * 8 * (kind == 2 ? 2 : 1);
  return resident + weights + (size_t)keys * (d1 + 4 + d2 + 4) + (kind == 2 ? 2 * (size_t)keys : 0);
}

// out[j] = x_j . y for the warp's eight resident rows x (stride d) and this lane's streamed row y.
__device__ __forceinline__ void tile_dot8(const float* x, const float* y, int d, float* out) {
  using namespace ptx;
  uint64_t acc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = 0ull;
#pragma unroll 4
  for (int c = 0; c < d; c += 4) {
    const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(y + c);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(x + j * d + c);
      acc[j] = f2_fma(a.x, b.x, acc[j]);
      acc[j] = f2_fma(a.y, b.y, acc[j]);
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float2 v = f2_unpack(acc[j]);
    out[j] = v.x + v.y;
  }
}

// acc[dd][jp] += w[k][2 jp, 2 jp + 1] * y[k][c0 + dd] over n staged tokens (rows `stride` floats apart).
template <int P>
__device__ __forceinline__ void tile_accumulate(uint64_t (&acc)[P][4], const float* w, const float* y, int stride, int n, int c0) {
  using namespace ptx;
#pragma unroll 4
  for (int k = 0; k < n; ++k) {
    const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(w + 8 * k), b = *reinterpret_cast<const ulonglong2*>(w + 8 * k + 4);
    const float* row = y + k * stride + c0;
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
      acc[dd][2] = f2_fma(b.x, vv, acc[dd][2]);
      acc[dd][3] = f2_fma(b.y, vv, acc[dd][3]);
    }
  }
}

template <int P>
__device__ __forceinline__ void tile_clear(uint64_t (&acc)[P][4]) {
#pragma unroll
  for (int dd = 0; dd < P; ++dd)
#pragma unroll
    for (int jp = 0; jp < 4; ++jp) acc[dd][jp] = 0ull;
}

// KIND as in TileArgs; P1 / P2: head dims of the q-k / v tensors per lane (2: up to 64, 4: up to 128).
template <int KIND, int P1, int P2>
__global__ void __launch_bounds__(256) simt_tile_kernel(const __grid_constant__ TileArgs t) {
  using namespace ptx;
  extern __shared__ __align__(16) float tile_smem[];
  const Geom& g = t.g;
  const int d1 = g.dqk, d2 = g.dv, s1 = d1 + 4, s2 = d2 + 4, Wtok = g.tw * g.b;
  float* x1 = tile_smem;                                         // resident rows [64][d]
  float* x2 = x1 + 64 * d1;
  float* wbuf = KIND == 0 ? x2 : x2 + 64 * d2;                   // weights [warp][1 or 2][32][8]
  float* y1 = wbuf + kTileRows * 32 * 8 * (KIND == 2 ? 2 : 1);   // staged tokens
  float* y2 = y1 + t.max_keys * s1;
  float* vec = y2 + t.max_keys * s2;                             // dK/dV: their lse, delta
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int bh = blockIdx.y, bi = bh / g.H, hi = bh - bi * g.H;
  const int ty = blockIdx.x / t.n_tiles_x, r0 = ty * kTileRows, c0 = (blockIdx.x - ty * t.n_tiles_x) * kTileCols;
  auto slice = [&](const View4& v) { return (float*)v.ptr + bi * v.s0 + hi * v.s1; };

  pdl_enter();
  pdl_wait();
  // resident rows (zeros beyond the grid)
  auto load_resident = [&](float* dst, const View4& v, int d) {
    const float* src = slice(v);
    for (int i = tid; i < 16 * d; i += 256) {
      const int row = i / (d >> 2), c = (i - row * (d >> 2)) * 4, rr = r0 + (row >> 3), cc = c0 + (row & 7);
      float4 val = make_float4(0.f, 0.f, 0.f, 0.f);
      if (rr < g.th && cc < Wtok) val = *reinterpret_cast<const float4*>(src + ((int64_t)rr * Wtok + cc) * v.s2 + c);
      *reinterpret_cast<float4*>(dst + row * d + c) = val;
    }
  };
  load_resident(x1, t.x1, d1);
  if constexpr (KIND != 0) load_resident(x2, t.x2, d2);

  const int my_r = r0 + warp;
  const bool on = my_r < g.th;
  float* const mx1 = x1 + warp * 8 * d1;
  float* const mx2 = x2 + warp * 8 * d2;
  float* const w1 = wbuf + warp * 32 * 8 * (KIND == 2 ? 2 : 1);
  float* const w2 = w1 + 32 * 8;
  const int64_t row_base = (int64_t)bh * g.th * Wtok + (int64_t)my_r * Wtok + c0;
  float m[8], l[8];                  // forward: running maximum (the same in all lanes), this lane's part of the sum; dQ: lse, delta
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    m[j] = -INFINITY;
    l[j] = 0.f;
    if constexpr (KIND == 1) {
      m[j] = 0.f;
      if (on && c0 + j < Wtok) {
        m[j] = t.lse[row_base + j];
        l[j] = t.delta[row_base + j];
      }
    }
  }
  constexpr int PA = KIND == 0 ? P2 : P1;
  uint64_t acc[PA][4];
  [[maybe_unused]] uint64_t acc2[P2][4];
  tile_clear(acc);
  if constexpr (KIND == 2) tile_clear(acc2);
  const int ca = lane * PA < (KIND == 0 ? d2 : d1) ? lane * PA : 0;          // this lane's head dims (lanes beyond them: idle copies)
  [[maybe_unused]] const int ca2 = lane * P2 < d2 ? lane * P2 : 0;

  // halo, clipped to the grid
  const int c_last = min(c0 + kTileCols, Wtok) - 1;
  const int x_lo = max(0, (c0 / g.b - g.wc) * g.b), x_hi = min(Wtok, (c_last / g.b + g.wc + 1) * g.b), nc = x_hi - x_lo;
  const int h_lo = max(0, r0 - g.wr), h_hi = min(g.th - 1, min(r0 + kTileRows, g.th) - 1 + g.wr);
  const uint32_t nc_inv = (0x1000000u + nc - 1) / nc;            // n / nc == (n * nc_inv) >> 24 for n < 4096

  for (int b0 = h_lo; b0 <= h_hi; b0 += t.rb) {
    const int b1 = min(b0 + t.rb - 1, h_hi);
    __syncthreads();                                             // nobody still reads the previous band
    auto load_band = [&](float* dst, const View4& v, int d, int s) {
      const float* src = slice(v);
      const int n4 = (b1 - b0 + 1) * nc * (d >> 2);
      for (int i = tid; i < n4; i += 256) {
        const int n = i / (d >> 2), c = (i - n * (d >> 2)) * 4, rr = n / nc;
        *reinterpret_cast<float4*>(dst + n * s + c) =
            *reinterpret_cast<const float4*>(src + ((int64_t)(b0 + rr) * Wtok + x_lo + n - rr * nc) * v.s2 + c);
      }
    };
    load_band(y1, t.y1, d1, s1);
    load_band(y2, t.y2, d2, s2);
    if constexpr (KIND == 2) {
      const int n = (b1 - b0 + 1) * nc;
      for (int i = tid; i < n; i += 256) {
        const int rr = i / nc;
        const int64_t at = (int64_t)bh * g.th * Wtok + (int64_t)(b0 + rr) * Wtok + x_lo + i - rr * nc;
        vec[i] = t.lse[at];
        vec[t.max_keys + i] = t.delta[at];
      }
    }
    __syncthreads();
    const int f0 = max(b0, my_r - g.wr), f1 = min(b1, my_r + g.wr);          // this warp's rows of the band
    if (!on || f0 > f1) continue;
    const int n0 = (f0 - b0) * nc, n_all = (f1 - f0 + 1) * nc;
#pragma unroll 1
    for (int k0 = 0; k0 < n_all; k0 += 32) {
      const int cnt = min(32, n_all - k0), k = min(k0 + lane, n_all - 1);
      const int kr = (int)(((uint64_t)(uint32_t)k * nc_inv) >> 24), yx = x_lo + k - kr * nc, n = n0 + k;
      const int yc = yx / g.b;
      int lo = (yc - g.wc) * g.b - c0, hi_ = (yc + g.wc + 1) * g.b - 1 - c0;  // resident columns this token may interact with
      if (lane >= cnt) hi_ = -1;
      float s[8];
      tile_dot8(mx1, y1 + n * s1, d1, s);
      if constexpr (KIND == 0) {
        bool grow = false;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          s[j] = j >= lo && j <= hi_ ? s[j] * g.scale_log2 : -INFINITY;
          grow = grow || s[j] > m[j] + 16.f || (m[j] == -INFINITY && s[j] > -INFINITY);
        }
        // the maximum is renewed only when a score passes it by more than 2^16: fp32 has the range to spare
        if (__any_sync(0xffffffffu, grow)) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            float v = s[j];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
            const float mn = fmaxf(m[j], v), a = m[j] == -INFINITY ? 0.f : exp2f(m[j] - mn);
            m[j] = mn;
            l[j] *= a;
            w1[lane * 8 + j] = a;                                // rescaling factors, by query pair, for the accumulators
          }
          const ulonglong2 fa = *reinterpret_cast<const ulonglong2*>(w1 + lane * 8), fb = *reinterpret_cast<const ulonglong2*>(w1 + lane * 8 + 4);
#pragma unroll
          for (int dd = 0; dd < PA; ++dd) {
            acc[dd][0] = f2_mul(acc[dd][0], fa.x);
            acc[dd][1] = f2_mul(acc[dd][1], fa.y);
            acc[dd][2] = f2_mul(acc[dd][2], fb.x);
            acc[dd][3] = f2_mul(acc[dd][3], fb.y);
          }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          s[j] = s[j] == -INFINITY ? 0.f : exp2f(s[j] - m[j]);
          l[j] += s[j];
        }
      } else {
        float dp[8];
        tile_dot8(mx2, y2 + n * s2, d2, dp);
        const float ls = KIND == 2 ? vec[n] : 0.f, de = KIND == 2 ? vec[t.max_keys + n] : 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const bool see = j >= lo && j <= hi_;
          const float p = see ? exp2f(fmaf(s[j], g.scale_log2, -(KIND == 1 ? m[j] : ls))) : 0.f;
          s[j] = p * (dp[j] - (KIND == 1 ? l[j] : de));
          dp[j] = p;
        }
        if constexpr (KIND == 2) {
          *reinterpret_cast<float4*>(w2 + lane * 8) = make_float4(dp[0], dp[1], dp[2], dp[3]);
          *reinterpret_cast<float4*>(w2 + lane * 8 + 4) = make_float4(dp[4], dp[5], dp[6], dp[7]);
        }
      }
      *reinterpret_cast<float4*>(w1 + lane * 8) = make_float4(s[0], s[1], s[2], s[3]);
      *reinterpret_cast<float4*>(w1 + lane * 8 + 4) = make_float4(s[4], s[5], s[6], s[7]);
      __syncwarp();
      // the band's tokens of a warp are consecutive: row n0 + k0 + i
      if constexpr (KIND == 0) {
        tile_accumulate<PA>(acc, w1, y2 + (n0 + k0) * s2, s2, cnt, ca);
      } else {
        tile_accumulate<PA>(acc, w1, y1 + (n0 + k0) * s1, s1, cnt, ca);
        if constexpr (KIND == 2) tile_accumulate<P2>(acc2, w2, y2 + (n0 + k0) * s2, s2, cnt, ca2);
      }
      __syncwarp();
    }
  }
  if (!on) return;

  // out: accumulators scaled, rotated back where asked, rows of this warp
  if constexpr (KIND == 0) {
    float* dst = slice(t.o1) + ((int64_t)my_r * Wtok + c0) * t.o1.s2;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float lt = warp_sum(l[j]), inv = 1.f / lt;
      if (c0 + j >= Wtok) continue;
#pragma unroll
      for (int dd = 0; dd < PA; ++dd) {
        const float2 v = f2_unpack(acc[dd][j >> 1]);
        if (lane * PA + dd < d2) dst[j * t.o1.s2 + lane * PA + dd] = (j & 1 ? v.y : v.x) * inv;
      }
      if (lane == 0) t.lse_out[row_base + j] = m[j] + log2f(lt);
    }
  } else {
    float* dst = slice(t.o1) + ((int64_t)my_r * Wtok + c0) * t.o1.s2;
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 8; ++j)                                  // the resident rows are done with: they take the result
#pragma unroll
      for (int dd = 0; dd < PA; ++dd) {
        const float2 v = f2_unpack(acc[dd][j >> 1]);
        if (lane * PA + dd < d1) mx1[j * d1 + lane * PA + dd] = (j & 1 ? v.y : v.x) * g.sm_scale;
      }
    __syncwarp();
#pragma unroll 1
    for (int j = 0; j < 8; ++j) {
      if (c0 + j >= Wtok) break;
      int irow = -1, icol = -1;
      if (t.rope.idx) decode_idx(t.rope.idx[my_r * Wtok + c0 + j], t.rope.max_h, t.rope.max_w, irow, icol);
      for (int d = lane; d < d1; d += 32) dst[j * t.o1.s2 + d] = load_rot<float>(mx1 + j * d1, 1, d, t.rope, irow, icol, -1.f);
    }
    if constexpr (KIND == 2) {
      float* dst2 = slice(t.o2) + ((int64_t)my_r * Wtok + c0) * t.o2.s2;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (c0 + j >= Wtok) continue;
#pragma unroll
        for (int dd = 0; dd < P2; ++dd) {
          const float2 v = f2_unpack(acc2[dd][j >> 1]);
          if (lane * P2 + dd < d2) dst2[j * t.o2.s2 + lane * P2 + dd] = j & 1 ? v.y : v.x;
        }
      }
    }
  }
}

}  // namespace swa
