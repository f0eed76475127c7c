// Native host path of the Python surface: argument checks, output allocation, C-ABI calls and the autograd nodes of
// TiledSwa / TiledSwaRope2D / TiledSwaPackedQKV (src/tiled_swa.py:602-689) in one extension module.
//
// A small call is bound by its host work: the same steps written in Python over ctypes took 120 us per forward and
// 300 us per training step while the GPU was busy for 16 to 110 us of it.  Here a call is METH_FASTCALL argument
// parsing, a handful of allocations from torch's caching allocator and the library's launches; the backward pass runs
// as a C++ autograd node, so the engine never takes the GIL for it.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/TracerMode.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>

#include <array>
#include <atomic>
#include <cstdlib>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/swa2d.h"

namespace {

using at::Tensor;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

// The surface raises AssertionError where the reference asserts; c10 has no such exception.
struct AssertFailed : std::exception {
  const char* msg;
  explicit AssertFailed(const char* m) : msg(m) {}
  const char* what() const noexcept override { return msg; }
};
void require(bool cond, const char* msg) {
  if (!cond) throw AssertFailed(msg);
}

enum Mode : int { kNone = 0, kHandoff, kFused, kPrerotate };
std::atomic<int> g_rope_mode{kHandoff};

struct Win {
  int32_t b, th, tw, wr, wc;
  float sm;
};
struct Rope {
  Tensor idx, row, col;      // idx undefined: no rotation
  bool on() const { return idx.defined(); }
};

// ---- status words -----------------------------------------------------------------------------------------------
// One block of pinned, device-mapped host memory per device: a kernel whose bounded wait gave up writes its first
// words, and every later call looks at them.  Nothing is copied or waited for on the way (a device word mirrored by a
// 16-byte copy and an event cost 3 us of stream time and 10 us of host time per call).
constexpr int kStatusWords = 4096, kMaxDev = 64;
std::mutex g_status_mu;
Tensor g_status[kMaxDev];
std::atomic<int32_t*> g_status_ptr[kMaxDev];

int32_t* status_ptr(int dev) {
  TORCH_CHECK(dev >= 0 && dev < kMaxDev, "device ordinal ", dev, " out of range");
  int32_t* p = g_status_ptr[dev].load(std::memory_order_acquire);
  if (p) return p;
  std::lock_guard<std::mutex> lock(g_status_mu);
  if (!g_status[dev].defined()) {
    c10::cuda::CUDAGuard guard((c10::DeviceIndex)dev);
    g_status[dev] = at::zeros({kStatusWords}, at::TensorOptions().dtype(at::kInt).pinned_memory(true));
  }
  p = g_status[dev].data_ptr<int32_t>();
  g_status_ptr[dev].store(p, std::memory_order_release);
  return p;
}

void raise_if_timed_out(int dev) {
  int32_t* p = g_status_ptr[dev].load(std::memory_order_acquire);
  if (!p || *reinterpret_cast<volatile int32_t*>(p) == 0) return;
  const int32_t v[4] = {p[0], p[1], p[2], p[3]};
  for (int i = 3; i >= 0; --i) p[i] = 0;
  TORCH_CHECK(false, "swa2d kernel reported a bounded-wait timeout on device ", dev, ": status=[", v[0], ", ", v[1], ", ", v[2],
              ", ", v[3], "] (its outputs are incomplete)");
}
void poll_status() {
  for (int d = 0; d < kMaxDev; ++d) {
    if (g_status_ptr[d].load(std::memory_order_relaxed)) raise_if_timed_out(d);
  }
}

void debug_sync() {
  const char* on = std::getenv("SWA_DEBUG_SYNC");      // read on every call: a debugger's switch is set when it is wanted
  if (!on || !*on) return;
  c10::cuda::device_synchronize();
  poll_status();
}

// ---- C-ABI views --------------------------------------------------------------------------------------------------
int32_t dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return SWA_F32;
    case at::kHalf: return SWA_F16;
    case at::kBFloat16: return SWA_BF16;
    default: TORCH_CHECK_TYPE(false, "unsupported dtype ", t, "; supported: float32, float16, bfloat16");
  }
}

swa_tensor_t view4(const Tensor& t) {
  swa_tensor_t r;
  r.ptr = t.data_ptr();
  const auto st = t.strides();
  for (int i = 0; i < 4; ++i) r.stride[i] = st[i];
  return r;
}

// What the planner needs of a rotation; nothing of it is read on the device.
swa_rope_t rope_shape(const Rope& r) {
  require(r.idx.scalar_type() == at::kInt && r.idx.is_contiguous(), "idx must be contiguous int32");
  require(r.row.scalar_type() == at::kFloat && r.col.scalar_type() == at::kFloat, "cos/sin tables must be float32");
  require(r.row.is_contiguous() && r.col.is_contiguous(), "cos/sin tables must be contiguous");
  require(r.row.dim() == 3 && r.col.dim() == 3 && r.row.size(2) == 2 && r.row.size(1) == r.col.size(1),
          "cos/sin tables must be [max, n_rdim, 2] with the same n_rdim");
  return swa_rope_t{r.idx.data_ptr<int32_t>(), r.row.data_ptr<float>(), r.col.data_ptr<float>(), (int32_t)r.row.size(1),
                    (int32_t)r.row.size(0), (int32_t)r.col.size(0)};
}

// ... and for a launch: the kernels read one index per token, and all three tensors as pointers of q's device.
swa_rope_t rope_view(const Rope& r, int64_t n_tokens, const Tensor& q) {
  const swa_rope_t v = rope_shape(r);
  require(r.idx.numel() >= n_tokens, "one index per token expected");
  TORCH_CHECK(r.idx.device() == q.device() && r.row.device() == q.device() && r.col.device() == q.device(),
              "idx and the cos/sin tables must be on the tensors' device: ", r.idx.device(), ", ", r.row.device(), ", ", r.col.device(),
              " beside ", q.device());
  return v;
}

// The tensor-core kernels read the tables by 16 bytes: tables that start elsewhere are copied, like tensors (materialise).
Rope aligned_tables(Rope r) {
  for (Tensor* t : {&r.row, &r.col})
    if (r.on() && t->is_cuda() && reinterpret_cast<uintptr_t>(t->data_ptr()) % 16) *t = t->clone();
  return r;
}

int32_t forced_impl(int32_t impl) {
  const char* e = std::getenv("SWA_FORCE_IMPL");
  if (!e) return impl;
  const std::string s(e);
  return s == "simt" ? SWA_IMPL_SIMT : s == "tc" ? SWA_IMPL_TC : s == "auto" ? SWA_IMPL_AUTO : impl;
}

swa_geom_t geom(const Tensor& q, int64_t d_qk, int64_t d_v, const Win& w, int32_t impl) {
  return swa_geom_t{dtype_code(q.scalar_type()), (int32_t)q.size(0), (int32_t)q.size(1), w.b, w.th, w.tw, w.wr, w.wc,
                    (int32_t)d_qk, (int32_t)d_v, w.sm, impl};
}

void check(int code, const char* what) { TORCH_CHECK(code == 0, what, " failed (", code, "): ", swa_last_error()); }

void check_inputs(const Tensor& q, const Tensor& k, const Tensor& v, const Win& w) {
  poll_status();
  TORCH_CHECK(q.is_cuda() && k.is_cuda() && v.is_cuda(),
              "dl_templates_b200 runs on CUDA tensors only (sm_100a); there is no CPU path");
  TORCH_CHECK(k.device() == q.device() && v.device() == q.device(), "q, k, v must be on one device");
  TORCH_CHECK_VALUE(q.dim() == 4 && v.dim() == 4 && k.sizes() == q.sizes() && v.sizes().slice(0, 3) == q.sizes().slice(0, 3),
                    "expected q,k [B,H,N,d_qk] and v [B,H,N,d_v]");
  TORCH_CHECK_TYPE(q.scalar_type() == k.scalar_type() && q.scalar_type() == v.scalar_type(), "q, k, v must share a dtype");
  require(q.size(2) == (int64_t)w.th * w.tw * w.b, "seqlen should match image size");
}

// Unit last stride, positive strides that are multiples of 8 elements, 16-byte aligned base: what a tensor map of the
// tensor-core kernels can describe.  A 16-bit tensor that is not is copied once rather than sending the call to the SIMT
// kernels; fp32 runs on the SIMT kernels, which take any strides.
Tensor materialise(const Tensor& t) {
  if (t.scalar_type() == at::kFloat) return t;
  const auto st = t.strides();
  const bool ok = st[3] == 1 && st[0] > 0 && st[1] > 0 && st[2] > 0 && ((st[0] | st[1] | st[2]) & 7) == 0 &&
                  reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0;
  return ok ? t : t.contiguous();
}

void check_out(const Tensor& t, at::IntArrayRef shape, const Tensor& like, const char* what) {
  TORCH_CHECK_VALUE(t.sizes() == shape && t.scalar_type() == like.scalar_type() && t.device() == like.device(), what,
                    ": expected shape ", shape, ", dtype ", like.scalar_type(), " on ", like.device());
}

// (d_qk', d_v') if zero-padding the head dims to 64 or 128 moves this problem from the SIMT kernels to the tensor-core
// kernels, else (0, 0).  With RoPE: to the kernels that rotate what they stream.
std::array<int64_t, 2> padded_dims(const Tensor& q, int64_t d_v, const Rope* rope, const Win& w, int32_t impl) {
  const std::array<int64_t, 2> none{0, 0};
  if (impl != SWA_IMPL_AUTO || q.scalar_type() == at::kFloat) return none;
  const int64_t d_qk = q.size(3);
  auto up = [](int64_t d) -> int64_t { return d <= 64 ? 64 : d <= 128 ? 128 : 0; };
  const int64_t p_qk = up(d_qk), p_v = up(d_v);
  if (!p_qk || !p_v || (p_qk == d_qk && p_v == d_v)) return none;
  const char* off = std::getenv("SWA_NO_HEAD_PAD");
  if (off && *off) return none;
  swa_rope_t r;
  const swa_rope_t* rp = nullptr;
  if (rope && rope->on()) { r = rope_shape(*rope); rp = &r; }
  auto all_tc = [&](int64_t a, int64_t b) {
    const swa_geom_t g = geom(q, a, b, w, forced_impl(SWA_IMPL_AUTO));
    if (!rp) return swa_step_select(&g, nullptr) == SWA_IMPL_TC;
    for (int which = 0; which < 3; ++which)
      if (swa_select_impl(&g, rp, which) != SWA_IMPL_TC) return false;
    return true;
  };
  if (all_tc(d_qk, d_v) || !all_tc(p_qk, p_v)) return none;
  return {p_qk, p_v};
}

// Whether the kernels without streamed rotation take the head dims as they are (or fp32, which is never padded).
bool native_dims(const Tensor& q, int64_t d_v, const Rope* rope, const Win& w, int32_t impl) {
  if (impl != SWA_IMPL_AUTO || q.scalar_type() == at::kFloat) return true;
  if (q.dim() != 4) return false;
  swa_rope_t r;
  const swa_rope_t* rp = nullptr;
  if (rope && rope->on()) { r = rope_shape(*rope); rp = &r; }
  const swa_geom_t g = geom(q, q.size(3), d_v, w, forced_impl(SWA_IMPL_AUTO));
  return swa_step_select(&g, rp) == SWA_IMPL_TC;
}

Tensor pad_last(const Tensor& t, int64_t d) {
  return t.size(3) == d ? t : at::constant_pad_nd(t, {0, d - t.size(3)});
}

void* stream_of(const Tensor& t) { return at::cuda::getCurrentCUDAStream(t.get_device()).stream(); }

Tensor new_lse(const Tensor& q) {
  return at::empty({q.size(0), q.size(1), q.size(2)}, q.options().dtype(at::kFloat));
}

// ---- forward / backward over the C ABI ------------------------------------------------------------------------------
struct Fwd {
  Tensor o, lse, q_rot, k_rot;
};
struct Grads {
  Tensor dq, dk, dv;
};

Fwd forward(Tensor q, Tensor k, Tensor v, const Rope& rope_, const Win& w, int32_t impl, Tensor out) {
  check_inputs(q, k, v, w);
  const Rope rope = aligned_tables(rope_);
  q = materialise(q); k = materialise(k); v = materialise(v);
  const auto pad = padded_dims(q, v.size(3), &rope, w, impl);
  if (pad[0]) {
    Fwd f = forward(pad_last(q, pad[0]), pad_last(k, pad[0]), pad_last(v, pad[1]), rope, w, impl, Tensor());
    const Tensor o_v = f.o.narrow(3, 0, v.size(3));
    if (!out.defined()) {
      f.o = o_v.contiguous();
    } else {
      check_out(out, o_v.sizes(), q, "out");
      out.copy_(o_v);
      f.o = out;
    }
    return f;
  }
  const c10::cuda::OptionalCUDAGuard guard(q.device());
  Fwd f;
  const std::array<int64_t, 4> shape{q.size(0), q.size(1), q.size(2), v.size(3)};
  if (out.defined()) check_out(out, shape, q, "out");
  f.o = out.defined() ? out : at::empty(shape, q.options());
  f.lse = new_lse(q);
  const swa_geom_t g = geom(q, q.size(3), v.size(3), w, forced_impl(impl));
  swa_rope_t r;
  if (rope.on()) r = rope_view(rope, q.size(2), q);
  const swa_tensor_t tq = view4(q), tk = view4(k), tv = view4(v), to = view4(f.o);
  if (rope.on())
    check(swa_fwd(&g, &r, &tq, &tk, &tv, &to, f.lse.data_ptr<float>(), status_ptr(q.get_device()), stream_of(q)), "swa_fwd");
  else
    check(swa_step_fwd(&g, nullptr, &tq, &tk, &tv, &to, f.lse.data_ptr<float>(), nullptr, nullptr, status_ptr(q.get_device()),
                       stream_of(q)), "swa_step_fwd");
  debug_sync();
  return f;
}

Fwd forward_rot(Tensor q, Tensor k, Tensor v, const Rope& rope_, const Win& w, int32_t impl, Tensor out) {
  check_inputs(q, k, v, w);
  const Rope rope = aligned_tables(rope_);
  q = materialise(q); k = materialise(k); v = materialise(v);
  const c10::cuda::OptionalCUDAGuard guard(q.device());
  Fwd f;
  const std::array<int64_t, 4> shape{q.size(0), q.size(1), q.size(2), v.size(3)};
  if (out.defined()) check_out(out, shape, q, "out");
  f.o = out.defined() ? out : at::empty(shape, q.options());
  f.lse = new_lse(q);
  f.q_rot = at::empty(q.sizes(), q.options());
  f.k_rot = at::empty(q.sizes(), q.options());
  const swa_geom_t g = geom(q, q.size(3), v.size(3), w, forced_impl(impl));
  const swa_rope_t r = rope_view(rope, q.size(2), q);
  const swa_tensor_t tq = view4(q), tk = view4(k), tv = view4(v), to = view4(f.o), tqr = view4(f.q_rot), tkr = view4(f.k_rot);
  check(swa_step_fwd(&g, &r, &tq, &tk, &tv, &to, f.lse.data_ptr<float>(), &tqr, &tkr, status_ptr(q.get_device()), stream_of(q)),
        "swa_step_fwd");
  debug_sync();
  return f;
}

// What backward reads beside the inputs: the forward's result and its gradient, the softmax statistic.
void check_saved(const Tensor& q, const Tensor& v, const Tensor& o, const Tensor& lse, const Tensor& d_o) {
  for (const Tensor* t : {&o, &d_o}) {
    TORCH_CHECK(t->device() == q.device(), "o and do must be on the device of q");
    TORCH_CHECK_VALUE(t->sizes() == v.sizes(), "expected o, do [B,H,N,d_v]");
    TORCH_CHECK_TYPE(t->scalar_type() == q.scalar_type(), "o and do must have the dtype of q");
  }
  TORCH_CHECK(lse.device() == q.device(), "lse must be on the device of q");
  TORCH_CHECK_TYPE(lse.scalar_type() == at::kFloat, "lse must be float32");
  TORCH_CHECK_VALUE(lse.numel() == q.size(0) * q.size(1) * q.size(2), "expected lse [B,H,N]");
}

// `rotated`: q and k are the rotated copies forward_rot left behind (swa_bwd_*_rot).
Grads backward(Tensor q, Tensor k, Tensor v, Tensor o, Tensor lse, Tensor d_o, const Rope& rope_, bool rotated, const Win& w,
               int32_t impl, Grads out) {
  check_inputs(q, k, v, w);
  check_saved(q, v, o, lse, d_o);
  const Rope rope = aligned_tables(rope_);
  lse = lse.contiguous();
  q = materialise(q); k = materialise(k); v = materialise(v); o = materialise(o); d_o = materialise(d_o);
  const bool given = out.dq.defined();
  if (!rotated) {
    const auto pad = padded_dims(q, v.size(3), &rope, w, impl);
    if (pad[0]) {
      Grads g = backward(pad_last(q, pad[0]), pad_last(k, pad[0]), pad_last(v, pad[1]), pad_last(o, pad[1]), lse,
                         pad_last(d_o, pad[1]), rope, false, w, impl, Grads());
      const Tensor dq = g.dq.narrow(3, 0, q.size(3)), dk = g.dk.narrow(3, 0, k.size(3)), dv = g.dv.narrow(3, 0, v.size(3));
      if (!given) return {dq.contiguous(), dk.contiguous(), dv.contiguous()};
      check_out(out.dq, dq.sizes(), q, "dq");
      check_out(out.dk, dk.sizes(), q, "dk");
      check_out(out.dv, dv.sizes(), q, "dv");
      out.dq.copy_(dq);
      out.dk.copy_(dk);
      out.dv.copy_(dv);
      return out;
    }
  }
  const c10::cuda::OptionalCUDAGuard guard(q.device());
  Grads r;
  if (given) {
    r = out;
    check_out(r.dq, q.sizes(), q, "dq");
    check_out(r.dk, k.sizes(), k, "dk");
    check_out(r.dv, v.sizes(), v, "dv");
  } else {
    r = {at::empty_like(q), at::empty_like(k), at::empty_like(v)};
  }
  const Tensor delta = new_lse(q);
  const swa_geom_t g = geom(q, q.size(3), v.size(3), w, forced_impl(impl));
  swa_rope_t rv;
  if (rope.on()) rv = rope_view(rope, q.size(2), q);
  const swa_rope_t* rp = rope.on() ? &rv : nullptr;
  const swa_tensor_t tq = view4(q), tk = view4(k), tv = view4(v), to = view4(o), tdo = view4(d_o), tdq = view4(r.dq),
                     tdk = view4(r.dk), tdv = view4(r.dv);
  void* st = stream_of(q);
  int32_t* status = status_ptr(q.get_device());
  const float* l = lse.data_ptr<float>();
  float* de = delta.data_ptr<float>();
  if (rope.on() && !rotated) {                       // the kernels that rotate streamed rows
    check(swa_bwd_delta(&g, &to, &tdo, de, st), "swa_bwd_delta");
    check(swa_bwd_dq(&g, rp, &tq, &tk, &tv, &tdo, l, de, &tdq, status, st), "swa_bwd_dq");
    check(swa_bwd_dkdv(&g, rp, &tq, &tk, &tv, &tdo, l, de, &tdk, &tdv, status, st), "swa_bwd_dkdv");
  } else {
    check(swa_step_bwd(&g, rp, &tq, &tk, &tv, &to, &tdo, l, de, &tdq, &tdk, &tdv, status, st), "swa_step_bwd");
  }
  debug_sync();
  return r;
}

// ---- stand-alone RoPE ---------------------------------------------------------------------------------------------
void rope_inplace(const Tensor& x, const Rope& rope, bool inverse) {
  TORCH_CHECK(x.is_cuda(), "dl_templates_b200 runs on CUDA tensors only (sm_100a); there is no CPU path");
  TORCH_CHECK_VALUE(x.dim() == 3, "expected x [batch, N, C]");
  require(rope.row.size(1) == rope.col.size(1), "row and column tables differ in width");
  require(rope.idx.size(0) == x.size(1), "one index per token expected");
  const c10::cuda::OptionalCUDAGuard guard(x.device());
  const swa_rope_t r = rope_view(rope, x.size(1), x);
  const int64_t xs[3] = {x.stride(0), x.stride(1), x.stride(2)};
  check(rope2d_apply(dtype_code(x.scalar_type()), x.data_ptr(), x.size(0), x.size(1), (int32_t)x.size(2), xs, &r, inverse ? 1 : 0,
                     stream_of(x)), "rope2d_apply");
}

Tensor rope_to(const Tensor& x, const Rope& rope, bool inverse) {
  TORCH_CHECK(x.is_cuda(), "dl_templates_b200 runs on CUDA tensors only (sm_100a); there is no CPU path");
  TORCH_CHECK_VALUE(x.dim() == 3, "expected x [batch, N, C]");
  require(rope.row.size(1) == rope.col.size(1) && rope.idx.size(0) == x.size(1), "one index per token and equal table widths expected");
  const Tensor y = at::empty(x.sizes(), x.options());
  const bool rows16 = x.stride(2) == 1 && reinterpret_cast<uintptr_t>(x.data_ptr()) % 16 == 0 && x.stride(0) % 8 == 0 &&
                      x.stride(1) % 8 == 0;
  if ((x.scalar_type() == at::kHalf || x.scalar_type() == at::kBFloat16) && rope.row.size(1) % 8 == 0 && x.size(2) % 8 == 0 && rows16) {
    const c10::cuda::OptionalCUDAGuard guard(x.device());
    const swa_rope_t r = rope_view(rope, x.size(1), x);
    const int64_t xs[3] = {x.stride(0), x.stride(1), x.stride(2)}, ys[3] = {y.stride(0), y.stride(1), y.stride(2)};
    check(rope2d_apply_to(dtype_code(x.scalar_type()), x.data_ptr(), y.data_ptr(), x.size(0), x.size(1), (int32_t)x.size(2), xs, ys,
                          &r, inverse ? 1 : 0, stream_of(x)), "rope2d_apply_to");
    return y;
  }
  y.copy_(x);
  rope_inplace(y, rope, inverse);
  return y;
}

Tensor flat3(const Tensor& t) { return t.reshape({-1, t.size(2), t.size(3)}); }

// ---- autograd -----------------------------------------------------------------------------------------------------
// The mode a call runs in: without RoPE none; head dims that only reach the tensor-core kernels through zero padding
// take the fused path (the padding lives there).
int mode_for(const Tensor& q, int64_t d_v, const Rope& rope, const Win& w) {
  if (!rope.on()) return kNone;
  const int m = g_rope_mode.load(std::memory_order_relaxed);
  if (m == kHandoff && !native_dims(q, d_v, &rope, w, SWA_IMPL_AUTO) && padded_dims(q, d_v, &rope, w, SWA_IMPL_AUTO)[0]) return kFused;
  return m;
}

struct SwaNode : public torch::autograd::Node {
  SavedVariable q, k, v, lse, o, idx, row, col;
  Win win;
  int mode = kNone;
  bool has_rope = false, packed = false;

  variable_list apply(variable_list&& grads) override;
  std::string name() const override { return packed ? "TiledSwaPackedQKVBackward" : "TiledSwaBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    for (SavedVariable* s : {&q, &k, &v, &lse, &o, &idx, &row, &col}) s->reset_data();
  }
};

Tensor head_view(const Tensor& qkv, int i) { return qkv.select(2, i).permute({0, 2, 1, 3}); }

variable_list SwaNode::apply(variable_list&& grads) {
  std::lock_guard<std::mutex> lock(mutex_);
  const at::AutoGradMode no_grad(false);
  const auto self = shared_from_this();
  Rope rope;
  if (has_rope) rope = {idx.unpack(), row.unpack(), col.unpack()};
  const Tensor o_ = o.unpack(self), lse_ = lse.unpack();
  Tensor d_o = grads[0].defined() ? grads[0] : at::zeros_like(o_);
  if (packed) {
    const Tensor qkv = v.unpack();
    const int64_t B = qkv.size(0), N = qkv.size(1), H = qkv.size(3), d = qkv.size(4);
    if (d_o.stride(2) != 1 || d_o.stride(1) % 8 || d_o.stride(0) % 8 || reinterpret_cast<uintptr_t>(d_o.data_ptr()) % 16)
      d_o = d_o.contiguous();
    const Tensor do4 = d_o.view({B, N, H, d}).permute({0, 2, 1, 3}), o4 = o_.view({B, N, H, d}).permute({0, 2, 1, 3});
    const Tensor dqkv = at::empty({B, N, 3, H, d}, qkv.options());
    const Grads outs{head_view(dqkv, 0), head_view(dqkv, 1), head_view(dqkv, 2)};
    if (mode == kHandoff)
      backward(q.unpack(), k.unpack(), head_view(qkv, 2), o4, lse_, do4, rope, true, win, SWA_IMPL_AUTO, outs);
    else
      backward(head_view(qkv, 0), head_view(qkv, 1), head_view(qkv, 2), o4, lse_, do4, rope, false, win, SWA_IMPL_AUTO, outs);
    return {dqkv};
  }
  const Tensor q_ = q.unpack(), k_ = k.unpack(), v_ = v.unpack();
  if (mode == kPrerotate) {
    Grads g = backward(q_, k_, v_, o_, lse_, d_o, Rope(), false, win, SWA_IMPL_AUTO, Grads());
    g.dq = g.dq.contiguous();
    g.dk = g.dk.contiguous();
    rope_inplace(flat3(g.dq), rope, true);
    rope_inplace(flat3(g.dk), rope, true);
    return {g.dq, g.dk, g.dv};
  }
  Grads g = backward(q_, k_, v_, o_, lse_, d_o, rope, mode == kHandoff, win, SWA_IMPL_AUTO, Grads());
  return {g.dq, g.dk, g.dv};
}

bool wants_grad(std::initializer_list<const Tensor*> ts) {
  if (!c10::GradMode::is_enabled()) return false;
  for (const Tensor* t : ts)
    if (t->requires_grad()) return true;
  return false;
}

// Whether the native node records all there is to record.  Forward-mode tangents, functorch's transforms, jit tracing, tensors
// with a Python dispatch of their own and tables that ask for gradients are for the autograd.Function of the same name, which
// refuses or handles them as torch does for every such function (general, below).
bool plain_call(std::initializer_list<const Tensor*> inputs, const Rope& rope) {
  if (c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode) || at::tracer::impl::is_dispatch_enabled())
    return false;
  auto plain = [](const Tensor& t) { return !t._fw_grad(0).defined() && !t.key_set().has(c10::DispatchKey::Python); };
  for (const Tensor* t : inputs)
    if (!plain(*t)) return false;
  if (rope.on())
    for (const Tensor* t : {&rope.row, &rope.col})
      if (!plain(*t) || wants_grad({t})) return false;
  return true;
}

std::shared_ptr<SwaNode> new_node(const Rope& rope, const Win& w, int mode) {
  std::shared_ptr<SwaNode> n(new SwaNode(), torch::autograd::deleteNode);
  n->win = w;
  n->mode = mode;
  n->has_rope = rope.on();
  if (rope.on()) {
    n->idx = SavedVariable(rope.idx, false);
    n->row = SavedVariable(rope.row, false);
    n->col = SavedVariable(rope.col, false);
  }
  return n;
}

Tensor apply_swa(const Tensor& q, const Tensor& k, const Tensor& v, const Rope& rope, const Win& w) {
  if (rope.on()) {
    require(q.dim() == 4 && rope.idx.size(0) == q.size(2), "one index per token expected");
    require(rope.row.size(1) == rope.col.size(1), "row and column tables differ in width");
  }
  const bool grad = wants_grad({&q, &k, &v});
  const at::AutoGradMode no_grad(false);
  check_inputs(q, k, v, w);
  const int mode = mode_for(q, v.size(3), rope, w);
  Tensor qs = q, ks = k;                       // what backward reads
  Fwd f;
  if (mode == kHandoff) {
    f = forward_rot(q, k, v, rope, w, SWA_IMPL_AUTO, Tensor());
    qs = f.q_rot;
    ks = f.k_rot;
  } else if (mode == kPrerotate) {
    qs = rope_to(flat3(q), rope, false).view(q.sizes());
    ks = rope_to(flat3(k), rope, false).view(k.sizes());
    f = forward(qs, ks, v, Rope(), w, SWA_IMPL_AUTO, Tensor());
  } else {
    f = forward(q, k, v, rope, w, SWA_IMPL_AUTO, Tensor());
  }
  if (grad) {
    auto n = new_node(rope, w, mode);
    n->set_next_edges(torch::autograd::collect_next_edges(q, k, v));
    n->q = SavedVariable(qs, false);
    n->k = SavedVariable(ks, false);
    n->v = SavedVariable(v, false);
    n->lse = SavedVariable(f.lse, false);
    torch::autograd::set_history(f.o, n);
    n->o = SavedVariable(f.o, true);
  }
  return f.o;
}

Tensor apply_packed(const Tensor& qkv, const Rope& rope, const Win& w) {
  TORCH_CHECK_VALUE(qkv.dim() == 5 && qkv.size(2) == 3, "expected qkv [B, N, 3, H, d]");
  const bool grad = wants_grad({&qkv});
  const at::AutoGradMode no_grad(false);
  const int64_t B = qkv.size(0), N = qkv.size(1), H = qkv.size(3), d = qkv.size(4);
  const Tensor q = head_view(qkv, 0), k = head_view(qkv, 1), v = head_view(qkv, 2);
  const int mode = mode_for(q, d, rope, w);
  Tensor o = at::empty({B, N, H * d}, qkv.options());
  const Tensor o4 = o.view({B, N, H, d}).permute({0, 2, 1, 3});
  Fwd f = mode == kHandoff ? forward_rot(q, k, v, rope, w, SWA_IMPL_AUTO, o4) : forward(q, k, v, rope, w, SWA_IMPL_AUTO, o4);
  if (grad) {
    auto n = new_node(rope, w, mode);
    n->packed = true;
    n->set_next_edges(torch::autograd::collect_next_edges(qkv));
    n->v = SavedVariable(qkv, false);
    if (mode == kHandoff) {
      n->q = SavedVariable(f.q_rot, false);
      n->k = SavedVariable(f.k_rot, false);
    }
    n->lse = SavedVariable(f.lse, false);
    torch::autograd::set_history(o, n);
    n->o = SavedVariable(o, true);
  }
  return o;
}

// ---- Python ---------------------------------------------------------------------------------------------------------
// Positional arguments of a METH_FASTCALL function, taken one by one.
struct Args {
  PyObject* const* a;
  Py_ssize_t n, at = 0;
  PyObject* next() {
    if (at >= n) {
      PyErr_Format(PyExc_TypeError, "expected more than %zd positional arguments", n);
      throw python_error();
    }
    return a[at++];
  }
  Tensor tensor() {
    PyObject* o = next();
    if (!THPVariable_Check(o)) {
      PyErr_Format(PyExc_TypeError, "argument %zd must be a tensor, not %s", at, Py_TYPE(o)->tp_name);
      throw python_error();
    }
    return THPVariable_Unpack(o);
  }
  Tensor maybe_tensor() {
    if (at < n && a[at] == Py_None) { ++at; return Tensor(); }
    return tensor();
  }
  int32_t i32() {
    const long v = PyLong_AsLong(next());
    if (v == -1 && PyErr_Occurred()) throw python_error();
    if (v > INT32_MAX || v < INT32_MIN) {
      PyErr_SetString(PyExc_OverflowError, "integer argument out of range");
      throw python_error();
    }
    return (int32_t)v;
  }
  float f32() {
    const double v = PyFloat_AsDouble(next());
    if (v == -1.0 && PyErr_Occurred()) throw python_error();
    return (float)v;
  }
  Rope rope() {
    Rope r;
    PyObject* i = next();
    PyObject *rr = next(), *cc = next();
    if (i == Py_None) return r;
    for (PyObject* o : {i, rr, cc})
      if (!THPVariable_Check(o)) {
        PyErr_SetString(PyExc_TypeError, "idx and the cos/sin tables must be tensors");
        throw python_error();
      }
    r.idx = THPVariable_Unpack(i);
    r.row = THPVariable_Unpack(rr);
    r.col = THPVariable_Unpack(cc);
    return r;
  }
  Win win() {
    Win w;
    w.b = i32(); w.th = i32(); w.tw = i32(); w.wr = i32(); w.wc = i32();
    w.sm = f32();
    return w;
  }
  void done() {
    if (at != n) {
      PyErr_Format(PyExc_TypeError, "expected %zd positional arguments, got %zd", at, n);
      throw python_error();
    }
  }
};

// Runs `body`; an AssertFailed becomes AssertionError, everything else what torch makes of it.
template <typename F>
PyObject* guarded(F&& body) {
  HANDLE_TH_ERRORS
  try {
    return body();
  } catch (AssertFailed& e) {
    PyErr_SetString(PyExc_AssertionError, e.msg);
    return nullptr;
  }
  END_HANDLE_TH_ERRORS
}

struct NoGil {
  PyThreadState* s = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(s); }
};
// Allocations and launches run without the interpreter's lock: a launch waits for room when the stream's queue is full, and
// other Python threads -- one of which the GPU may be waiting for -- have to run meanwhile.  The tensors a call works on are held by
// copies of its own (Args::tensor), whatever another thread does to its arguments.
template <typename F>
auto without_gil(F&& f) {
  const NoGil nogil;
  return f();
}

PyObject* pack(std::initializer_list<Tensor> ts) {
  PyObject* t = PyTuple_New((Py_ssize_t)ts.size());
  if (!t) throw python_error();
  Py_ssize_t i = 0;
  for (const Tensor& x : ts) PyTuple_SET_ITEM(t, i++, THPVariable_Wrap(x));
  return t;
}

// The `apply` of torch.autograd.Function for TiledSwa, TiledSwaRope2D and TiledSwaPackedQKV: what is no plain_call goes there.
// (Asked from here: a Python method around the native entry that looks at its answer costs every call 0.4 us.)
PyObject* g_general[3] = {};
PyObject* general(int i, PyObject* const* args, Py_ssize_t n) {
  TORCH_CHECK(g_general[i], "set_general has not been called");
  return PyObject_Vectorcall(g_general[i], args, (size_t)n, nullptr);
}
// set_general(three callables)
PyObject* py_set_general(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args a{args, n};
    for (PyObject*& g : g_general) {
      PyObject* o = a.next();
      Py_INCREF(o);
      Py_XSETREF(g, o);
    }
    a.done();
    Py_RETURN_NONE;
  });
}

// apply(q, k, v, b_size, t_height, t_width, row_size, col_size, sm_scale)
PyObject* py_tiled_swa(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args a{args, n};
    const Tensor q = a.tensor(), k = a.tensor(), v = a.tensor();
    const Win w = a.win();
    a.done();
    if (!plain_call({&q, &k, &v}, Rope())) return general(0, args, n);
    return THPVariable_Wrap(without_gil([&] { return apply_swa(q, k, v, Rope(), w); }));
  });
}
// apply(q, k, v, idx, row_cs, col_cs, b_size, t_height, t_width, row_size, col_size, sm_scale)
PyObject* py_tiled_swa_rope2d(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args a{args, n};
    const Tensor q = a.tensor(), k = a.tensor(), v = a.tensor();
    const Rope r = a.rope();
    const Win w = a.win();
    a.done();
    if (!plain_call({&q, &k, &v}, r)) return general(1, args, n);
    return THPVariable_Wrap(without_gil([&] { return apply_swa(q, k, v, r, w); }));
  });
}
// apply(qkv, idx, row_cs, col_cs, b_size, t_height, t_width, row_size, col_size, sm_scale)
PyObject* py_tiled_swa_packed(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args a{args, n};
    const Tensor qkv = a.tensor();
    const Rope r = a.rope();
    const Win w = a.win();
    a.done();
    if (!plain_call({&qkv}, r)) return general(2, args, n);
    return THPVariable_Wrap(without_gil([&] { return apply_packed(qkv, r, w); }));
  });
}
// forward(q, k, v, idx, row_cs, col_cs, window..., sm_scale, impl, out) -> (o, lse)
PyObject* py_forward(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args a{args, n};
    const Tensor q = a.tensor(), k = a.tensor(), v = a.tensor();
    const Rope r = a.rope();
    const Win w = a.win();
    const int32_t impl = a.i32();
    const Tensor out = a.maybe_tensor();
    a.done();
    const at::AutoGradMode no_grad(false);
    const Fwd f = without_gil([&] { return forward(q, k, v, r, w, impl, out); });
    return pack({f.o, f.lse});
  });
}
// forward_rot(same arguments) -> (o, lse, q_rot, k_rot)
PyObject* py_forward_rot(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args a{args, n};
    const Tensor q = a.tensor(), k = a.tensor(), v = a.tensor();
    const Rope r = a.rope();
    const Win w = a.win();
    const int32_t impl = a.i32();
    const Tensor out = a.maybe_tensor();
    a.done();
    const at::AutoGradMode no_grad(false);
    const Fwd f = without_gil([&] { return forward_rot(q, k, v, r, w, impl, out); });
    return pack({f.o, f.lse, f.q_rot, f.k_rot});
  });
}
// backward(q, k, v, o, lse, do, idx, row_cs, col_cs, window..., sm_scale, impl, rotated, dq, dk, dv) -> (dq, dk, dv)
PyObject* py_backward(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args a{args, n};
    const Tensor q = a.tensor(), k = a.tensor(), v = a.tensor(), o = a.tensor(), lse = a.tensor(), d_o = a.tensor();
    const Rope r = a.rope();
    const Win w = a.win();
    const int32_t impl = a.i32(), rotated = a.i32();
    const Grads out{a.maybe_tensor(), a.maybe_tensor(), a.maybe_tensor()};
    a.done();
    const at::AutoGradMode no_grad(false);
    const Grads g = without_gil([&] { return backward(q, k, v, o, lse, d_o, r, rotated != 0, w, impl, out); });
    return pack({g.dq, g.dk, g.dv});
  });
}
// check_backward(q, k, v, o, lse, do, idx, row_cs, col_cs, window..., sm_scale): raises what backward would raise, launches nothing
PyObject* py_check_backward(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args a{args, n};
    const Tensor q = a.tensor(), k = a.tensor(), v = a.tensor(), o = a.tensor(), lse = a.tensor(), d_o = a.tensor();
    const Rope r = a.rope();
    const Win w = a.win();
    a.done();
    check_inputs(q, k, v, w);
    check_saved(q, v, o, lse, d_o);
    if (r.on()) rope_view(r, q.size(2), q);
    Py_RETURN_NONE;
  });
}
// rope2d_(x [batch,N,C], idx, row_cs, col_cs, inverse) -> x, rotated in place
PyObject* py_rope2d_inplace(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args a{args, n};
    const Tensor x = a.tensor();
    const Rope r = a.rope();
    const bool inverse = a.i32() != 0;
    a.done();
    without_gil([&] { rope_inplace(x, r, inverse); });
    Py_INCREF(args[0]);
    return args[0];
  });
}
// rope2d_to(x [batch,N,C], idx, row_cs, col_cs, inverse) -> rotated copy
PyObject* py_rope2d_to(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args a{args, n};
    const Tensor x = a.tensor();
    const Rope r = a.rope();
    const bool inverse = a.i32() != 0;
    a.done();
    const at::AutoGradMode no_grad(false);
    return THPVariable_Wrap(without_gil([&] { return rope_to(x, r, inverse); }));
  });
}
// rope2d_heads_(x [B,H,N,C], idx, row_cs, col_cs) -> view of x (of a copy when x cannot be flattened), rotated in place.
// None when autograd has to record the operation: the caller then takes its autograd function.
PyObject* py_rope2d_heads_inplace(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args a{args, n};
    const Tensor x = a.tensor();
    const Rope r = a.rope();
    a.done();
    if (x.dim() != 4 || wants_grad({&x}) || !plain_call({&x}, r)) Py_RETURN_NONE;
    return THPVariable_Wrap(without_gil([&] {
      const Tensor flat = flat3(x);
      rope_inplace(flat, r, false);
      flat.unsafeGetTensorImpl()->bump_version();
      return flat.view(x.sizes());
    }));
  });
}
// padded_dims(q, d_v, idx, row_cs, col_cs, window..., sm_scale, impl) -> (d_qk', d_v') or None
PyObject* py_padded_dims(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args a{args, n};
    const Tensor q = a.tensor();
    const int32_t d_v = a.i32();
    const Rope r = a.rope();
    const Win w = a.win();
    const int32_t impl = a.i32();
    a.done();
    const auto p = padded_dims(q, d_v, &r, w, impl);
    if (!p[0]) Py_RETURN_NONE;
    return Py_BuildValue("(LL)", (long long)p[0], (long long)p[1]);
  });
}
// rope_mode(q, d_v, idx, row_cs, col_cs, window..., sm_scale) -> code of the mode a call runs in
PyObject* py_rope_mode(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args a{args, n};
    const Tensor q = a.tensor();
    const int32_t d_v = a.i32();
    const Rope r = a.rope();
    const Win w = a.win();
    a.done();
    return PyLong_FromLong(mode_for(q, d_v, r, w));
  });
}
PyObject* py_set_rope_mode(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args a{args, n};
    const int32_t m = a.i32();
    a.done();
    return PyLong_FromLong(g_rope_mode.exchange(m));
  });
}
// status_words(device index) -> the int32 tensor (pinned host memory) the kernels of that device report to
PyObject* py_status_words(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args a{args, n};
    const int32_t dev = a.i32();
    a.done();
    status_ptr(dev);
    return THPVariable_Wrap(g_status[dev]);
  });
}
// check_status(): wait for every device that has been used and raise if a kernel reported a timed-out wait
PyObject* py_check_status(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args{args, n}.done();
    for (int d = 0; d < kMaxDev; ++d) {
      if (!g_status_ptr[d].load(std::memory_order_relaxed)) continue;
      {
        NoGil nogil;
        c10::cuda::CUDAGuard guard((c10::DeviceIndex)d);
        c10::cuda::device_synchronize();
      }
      raise_if_timed_out(d);
    }
    Py_RETURN_NONE;
  });
}
PyObject* py_poll_status(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args{args, n}.done();
    poll_status();
    Py_RETURN_NONE;
  });
}

#define SWA_DEF(name, fn) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(fn)), METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {SWA_DEF("tiled_swa", py_tiled_swa),
                           SWA_DEF("tiled_swa_rope2d", py_tiled_swa_rope2d),
                           SWA_DEF("tiled_swa_packed", py_tiled_swa_packed),
                           SWA_DEF("set_general", py_set_general),
                           SWA_DEF("forward", py_forward),
                           SWA_DEF("forward_rot", py_forward_rot),
                           SWA_DEF("backward", py_backward),
                           SWA_DEF("check_backward", py_check_backward),
                           SWA_DEF("rope2d_", py_rope2d_inplace),
                           SWA_DEF("rope2d_to", py_rope2d_to),
                           SWA_DEF("rope2d_heads_", py_rope2d_heads_inplace),
                           SWA_DEF("padded_dims", py_padded_dims),
                           SWA_DEF("rope_mode", py_rope_mode),
                           SWA_DEF("set_rope_mode", py_set_rope_mode),
                           SWA_DEF("status_words", py_status_words),
                           SWA_DEF("check_status", py_check_status),
                           SWA_DEF("poll_status", py_poll_status),
                           {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_swa2d_torch", nullptr, -1, g_methods};

}  // namespace

PyMODINIT_FUNC PyInit__swa2d_torch() { return PyModule_Create(&g_module); }
