// Shared device/host helpers for the 2D sliding-window attention kernels.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <mutex>

#include "../../include/swa2d.h"

namespace swa {

constexpr float kLog2e = 1.4426950408889634f;

// ---- element <-> float ---------------------------------------------------------------------
template <typename T> __device__ __forceinline__ float to_f(T v);
template <> __device__ __forceinline__ float to_f<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

template <typename T> __device__ __forceinline__ T from_f(float v);
template <> __device__ __forceinline__ float from_f<float>(float v) { return v; }
template <> __device__ __forceinline__ __half from_f<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// ---- strided [B,H,N,d] view ----------------------------------------------------------------
struct View4 {
  void* ptr;
  int64_t s0, s1, s2, s3;
};

inline View4 make_view(const swa_tensor_t* t) {
  return View4{t->ptr, t->stride[0], t->stride[1], t->stride[2], t->stride[3]};
}

// ---- fused RoPE-2D parameters (idx == nullptr: none) ---------------------------------------
struct RopeDev {
  const int32_t* idx;
  const float* row_cs;
  const float* col_cs;
  int R, max_h, max_w;
};

inline RopeDev make_rope(const swa_rope_t* r) {
  if (r == nullptr || r->idx == nullptr) return RopeDev{nullptr, nullptr, nullptr, 0, 0, 0};
  return RopeDev{r->idx, r->row_cs, r->col_cs, r->n_rdim, r->max_h, r->max_w};
}

// Packed index -> (row, col) as sign-extended 16-bit halves; a negative half
// disables that half's rotation.  Positions are clamped to the table length so a
// bad index can never read outside the table.
__device__ __forceinline__ void decode_idx(int32_t packed, int max_h, int max_w, int& row, int& col) {
  row = packed >> 16;
  col = (int)(int16_t)(packed & 0xFFFF);
  row = row >= max_h ? max_h - 1 : row;
  col = col >= max_w ? max_w - 1 : col;
}

// Geometry handed to every attention kernel.
struct Geom {
  int B, H, b, th, tw, wr, wc, dqk, dv;
  float scale_log2;  // sm_scale * log2(e)
  float sm_scale;
};

// (A window taller than the grid is cut to the grid: the same pairs, and r + wr stays far from overflow.)
inline Geom make_geom(const swa_geom_t* g) {
  Geom r;
  r.B = g->B; r.H = g->H; r.b = g->b_size; r.th = g->t_height; r.tw = g->t_width;
  r.wr = g->row_size < g->t_height ? g->row_size : g->t_height - 1;
  r.wc = g->col_size; r.dqk = g->d_qk; r.dv = g->d_v;
  r.sm_scale = g->sm_scale; r.scale_log2 = g->sm_scale * kLog2e;
  return r;
}

// ---- programmatic dependent launch ---------------------------------------------------------
// The kernels of a step follow each other on one stream, and between two of them lie 2 to 4 us of draining and starting --
// half of a small step's GPU time.  Every kernel lets its successor start at once (launch_dependents), does what needs no
// global memory, and then waits until its predecessor has finished and its writes are visible.  A kernel that allocates tensor
// memory calls pdl_enter only once it has it: a successor resident on the same SM would otherwise hold what it waits for.
//
// Such a kernel is resident while its predecessor still writes what it will read.  So nothing it reads goes through the
// read-only path (__ldg, or `const __restrict__`, which the compiler may turn into it): that path is for data nobody writes while
// the kernel lives, and `__restrict__` would also allow a load to move above pdl_wait, whose memory clobber orders plain loads only.
__device__ __forceinline__ void pdl_enter() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... P, typename... A>
inline cudaError_t launch_pdl(void (*kern)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t st, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
}

// Set an attribute of a kernel once per kernel and device (the call costs a microsecond).
inline cudaError_t set_once(const void* kern, cudaFuncAttribute attr, int value) {
  struct Entry { const void* kern; int dev; };
  static Entry table[512];
  static std::atomic<int> n{0};
  static std::mutex mu;
  int dev = 0;
  if (cudaError_t e = cudaGetDevice(&dev); e != cudaSuccess) return e;
  for (int i = 0, have = n.load(std::memory_order_acquire); i < have; ++i)
    if (table[i].kern == kern && table[i].dev == dev) return cudaSuccess;
  std::lock_guard<std::mutex> lock(mu);
  if (cudaError_t e = cudaFuncSetAttribute(kern, attr, value); e != cudaSuccess) return e;
  const int now = n.load();
  if (now < 512) {
    table[now] = Entry{kern, dev};
    n.store(now + 1, std::memory_order_release);
  }
  return cudaSuccess;
}

// All the dynamic shared memory there is.
inline cudaError_t allow_smem(const void* kern) { return set_once(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024); }

// Streaming kernels (no shared memory, loads in flight wherever L1 has room) ask for all of L1: started early on an SM that the
// attention kernels have split for shared memory, they would keep the 28 KB of L1 that it leaves -- 480 instead of 310 us for
// the 2.1 GB that q and k of 256 slices of 128 x 128 x 64 move.
template <typename... P, typename... A>
inline cudaError_t launch_stream(void (*kern)(P...), dim3 grid, unsigned threads, cudaStream_t st, A&&... args) {
  if (cudaError_t e = set_once((const void*)kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxL1); e != cudaSuccess)
    return e;
  return launch_pdl(kern, grid, threads, 0, st, static_cast<A&&>(args)...);
}

}  // namespace swa
