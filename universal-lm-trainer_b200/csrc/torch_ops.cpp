// The host side of the ops as native autograd functions: argument checks, output allocation, the C-ABI call
// (include/ulm_b200.h) and the backward's node, without the interpreter.
//
// What bounds a small call is this path and not the kernels: at 4 x 201 tokens the six kernels of RoPE + attention
// forward and backward take 35 us on the device, while the same ops written as Python autograd functions over
// ctypes kept the host busy for 310 us (argument structs, shape and stride queries, an interpreter lock per
// backward node).  The Python modules keep their functions and their documentation and forward to this file; the
// semantics of every op are documented there.
//
// Nothing here computes: every kernel is the library's, plus the library GEMMs of the linear layers.
#include <ATen/ATen.h>
#include <ATen/ThreadLocalPythonObjects.h>
#include <ATen/autocast_mode.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/AutogradState.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/csrc/utils/pybind.h>

#include <algorithm>
#include <atomic>
#include <functional>
#include <memory>
#include <mutex>
#include <string>
#include <unordered_map>
#include <utility>
#include <vector>

#include "../../include/ulm_b200.h"

namespace {

using at::Tensor;
using torch::autograd::variable_list;
using OptTensor = std::optional<Tensor>;

void check(int rc, const char* what) {
  if (rc == ULM_OK) return;
  const char* msg = ulm_last_error();
  TORCH_CHECK_VALUE(rc != ULM_ERR_ARG, what, ": ", msg);
  TORCH_CHECK(false, what, ": ", msg, " (code ", rc, ")");
}

void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

bool is_16bit(at::ScalarType t) { return t == at::kHalf || t == at::kBFloat16; }
int code_of(at::ScalarType t) { return t == at::kHalf ? ULM_F16 : t == at::kBFloat16 ? ULM_BF16 : ULM_F32; }
bool known(at::ScalarType t) { return is_16bit(t) || t == at::kFloat; }

// Device tensors straight from the caching allocator: no dispatcher round trip.
Tensor empty_strided(at::IntArrayRef sizes, at::IntArrayRef strides, at::ScalarType dtype, const Tensor& like) {
  return at::detail::empty_strided_cuda(sizes, strides, dtype, like.device());
}
Tensor empty_cuda(at::IntArrayRef sizes, at::ScalarType dtype, const Tensor& like) {
  return at::detail::empty_cuda(sizes, dtype, like.device(), std::nullopt);
}
// (B,H,S,64) stored as (B,S,H,64)
Tensor empty_bshd(int64_t B, int64_t H, int64_t S, const Tensor& like) {
  return empty_strided({B, H, S, 64}, {S * H * 64, 64, H * 64, 1}, like.scalar_type(), like);
}

// True when the call will not be differentiated: the op then runs without a graph node.
template <typename... Ts>
bool no_graph(const Ts&... ts) {
  return !at::GradMode::is_enabled() || !(ts.requires_grad() || ...);
}

// What surrounds every op's own work: no recording below it and no autocast of the tensors it has already cast.
struct OpScope {
  at::NoGradGuard no_grad;
  at::AutoDispatchBelowADInplaceOrView below;
  c10::impl::ExcludeDispatchKeyGuard no_autocast{c10::DispatchKeySet(c10::DispatchKey::AutocastCUDA)};
};

// Base of the ops' backward nodes: the tensors they keep, unpacked through autograd's own saved variables (version
// checks, saved-tensor hooks, release after the backward).  All are unpacked BEFORE the op's scope opens: a hook may run
// a checkpointed forward again, which has to record its graph and to autocast as it did the first time.
struct OpNode : torch::autograd::Node {
  std::vector<torch::autograd::SavedVariable> saved;
  void keep(const Tensor& t, bool is_output = false) { saved.emplace_back(t, is_output); }
  // the zero gradient of input i; undefined where none is asked for
  Tensor zero_grad(size_t i) {
    if (!task_should_compute_output(i)) return Tensor();
    const torch::autograd::Edge& e = next_edge(i);
    return e.function->input_metadata(e.input_nr).zeros_like();
  }
  // the gradients of the inputs, from those of the outputs (at least one is defined) and the tensors kept
  virtual variable_list backward(variable_list& g, const variable_list& kept) = 0;
  // the same for a backward that is itself recorded (create_graph); the library's kernels have no derivative of their own
  virtual variable_list backward_recorded(variable_list& g, const variable_list& kept) {
    OpScope scope;
    return backward(g, kept);
  }
  variable_list apply(variable_list&& g) final {
    if (std::none_of(g.begin(), g.end(), [](const Tensor& t) { return t.defined(); })) {
      // an input that no gradient reaches has a zero one, not none: an optimiser treats the two differently
      variable_list zeros;
      for (size_t i = 0; i < num_outputs(); ++i) zeros.push_back(zero_grad(i));
      return zeros;
    }
    variable_list kept;
    {
      std::lock_guard<std::mutex> lock(mutex_);
      kept.reserve(saved.size());
      for (const auto& s : saved) kept.push_back(s.unpack(getptr()));
    }
    if (at::GradMode::is_enabled()) return backward_recorded(g, kept);
    OpScope scope;
    return backward(g, kept);
  }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    for (auto& s : saved) s.reset_data();
  }
};
// The node's edges to the inputs that may receive a gradient, in the order `apply` returns them.
template <typename N, typename... Ts>
std::shared_ptr<N> make_node(const Ts&... inputs) {
  std::shared_ptr<N> n(new N(), torch::autograd::deleteNode);
  n->set_next_edges(torch::autograd::collect_next_edges(inputs...));
  return n;
}

// ---------------------------------------------------------------------------
// status word: one int32 per device that the kernels OR their timeout bits into
// ---------------------------------------------------------------------------
constexpr int kMaxDevices = 64;
std::mutex g_status_mu;
std::atomic<uint32_t*> g_status_ptr[kMaxDevices];
Tensor* g_status[kMaxDevices];                   // never destroyed: no exit-order hazards

Tensor status_tensor(int64_t index) {
  TORCH_CHECK(index >= 0 && index < kMaxDevices, "device index ", index, " beyond ", kMaxDevices - 1);
  std::lock_guard<std::mutex> lock(g_status_mu);
  if (!g_status[index]) {
    g_status[index] = new Tensor(at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, (c10::DeviceIndex)index)));
    g_status_ptr[index].store(static_cast<uint32_t*>(g_status[index]->data_ptr()), std::memory_order_release);
  }
  return *g_status[index];
}
uint32_t* status_ptr(const Tensor& t) {
  const int i = t.device().index();
  uint32_t* p = g_status_ptr[i].load(std::memory_order_acquire);
  return p ? p : (status_tensor(i), g_status_ptr[i].load(std::memory_order_acquire));
}

// ---------------------------------------------------------------------------
// attention and RoPE
// ---------------------------------------------------------------------------
// (B,H,S,64) 16-bit, innermost contiguous, 32-byte aligned base and strides
bool fa_ready(const Tensor& t) {
  if (!t.is_cuda() || !is_16bit(t.scalar_type()) || t.dim() != 4) return false;
  const auto n = t.sizes(), s = t.strides();
  if (n[3] != 64 || s[3] != 1 || (reinterpret_cast<uintptr_t>(t.data_ptr()) & 31)) return false;
  for (int i = 0; i < 3; ++i)
    if (s[i] % 16 || (s[i] <= 0 && n[i] != 1)) return false;
  return n[2] == 1 || s[2] >= 64;
}
bool can_use(const Tensor& q, const Tensor& k, const Tensor& v) {
  return fa_ready(q) && fa_ready(k) && fa_ready(v) && q.sizes() == k.sizes() && k.sizes() == v.sizes() &&
         q.scalar_type() == k.scalar_type() && k.scalar_type() == v.scalar_type();
}
bool table_ok(const Tensor& t, int64_t rows, const Tensor& like) {
  return t.scalar_type() == at::kFloat && t.device() == like.device() && t.dim() == 2 && t.size(0) == rows && t.size(1) == 64 &&
         t.stride(1) == 1 && t.stride(0) % 4 == 0 && !(reinterpret_cast<uintptr_t>(t.data_ptr()) & 15);
}
bool rope_can_use(const Tensor& q, const Tensor& k, const Tensor& cos, const Tensor& sin) {
  return fa_ready(q) && fa_ready(k) && q.sizes() == k.sizes() && q.scalar_type() == k.scalar_type() &&
         table_ok(cos, q.size(2), q) && table_ok(sin, q.size(2), q);
}

// Dense output in the input's memory order: fused-qkv views come back as (B,S,H,64)-ordered tensors
Tensor rope_out_like(at::IntArrayRef n, at::IntArrayRef s, const Tensor& like) {
  int64_t extent = 1, numel = 1;
  for (int i = 0; i < 4; ++i) { extent += (n[i] - 1) * s[i]; numel *= n[i]; }
  if (extent == numel) return empty_strided(n, s, like.scalar_type(), like);
  if (s[1] == n[3] && s[2] >= n[1] * n[3]) return empty_bshd(n[0], n[1], n[2], like);
  return empty_cuda(n, like.scalar_type(), like);
}

// q (and qo) may be undefined: only k is rotated then
void rope_launch(const Tensor& q, const Tensor& k, const Tensor& qo, const Tensor& ko, const Tensor& cos, const Tensor& sin, bool backward) {
  ulm_rope_args a{};
  a.k = k.data_ptr(); a.ko = ko.data_ptr();
  a.k_sb = k.stride(0); a.k_sh = k.stride(1); a.k_ss = k.stride(2);
  a.ko_sb = ko.stride(0); a.ko_sh = ko.stride(1); a.ko_ss = ko.stride(2);
  if (q.defined()) {
    a.q = q.data_ptr(); a.qo = qo.data_ptr();
    a.q_sb = q.stride(0); a.q_sh = q.stride(1); a.q_ss = q.stride(2);
    a.qo_sb = qo.stride(0); a.qo_sh = qo.stride(1); a.qo_ss = qo.stride(2);
  }
  a.cos_tab = cos.data_ptr<float>(); a.sin_tab = sin.data_ptr<float>();
  a.cos_stride = cos.stride(0); a.sin_stride = sin.stride(0);
  a.B = (int32_t)k.size(0); a.H = (int32_t)k.size(1); a.S = (int32_t)k.size(2);
  a.dtype = code_of(k.scalar_type()); a.backward = backward;
  a.stream = stream_of(k);
  check(ulm_rope(&a), "rope");
}

struct AttnArgs {
  double dropout_p; bool causal; double scale; int64_t seed;
};

// Whether the attention forward rotates Q and K itself: sequences of one query tile, and no more of them than run at a
// time (two CTAs on each of 148 SMs).  Then the saved launch is what counts: 12 heads x 67 tokens x 1 sequence 7.2 us
// against 8.2, x 24 (288 CTAs) 9.9 against 10.8.  With more, every further wave pays for the rotation at the start of its
// CTAs: x 64 24.7 against 21.2, 16 heads x 256 sequences x 16 / 67 / 128 tokens 78 / 112 / 125 against 59 / 95 / 121 us.
bool rope_in_tile(int64_t B, int64_t H, int64_t S) { return S <= 128 && B * H <= 2 * 148; }

// -> (o, lse); with tables q comes unrotated and, where q_rot is defined, its rotated copy is written there; with k_rot
// (S <= 128) k comes unrotated too
void attn_forward(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, const Tensor& lse, const AttnArgs& p,
                  const Tensor& cos = Tensor(), const Tensor& sin = Tensor(), const Tensor& q_rot = Tensor(), const Tensor& k_rot = Tensor()) {
  ulm_attn_fwd_args a{};
  a.q = q.data_ptr(); a.k = k.data_ptr(); a.v = v.data_ptr(); a.o = o.data_ptr(); a.lse = lse.data_ptr<float>();
  a.q_sb = q.stride(0); a.q_sh = q.stride(1); a.q_ss = q.stride(2);
  a.k_sb = k.stride(0); a.k_sh = k.stride(1); a.k_ss = k.stride(2);
  a.v_sb = v.stride(0); a.v_sh = v.stride(1); a.v_ss = v.stride(2);
  a.o_sb = o.stride(0); a.o_sh = o.stride(1); a.o_ss = o.stride(2);
  a.B = (int32_t)q.size(0); a.H = (int32_t)q.size(1); a.S = (int32_t)q.size(2);
  a.dtype = code_of(q.scalar_type()); a.causal = p.causal;
  a.softmax_scale = (float)p.scale; a.dropout_p = (float)p.dropout_p; a.seed = (uint32_t)p.seed;
  a.status_dev = status_ptr(q); a.stream = stream_of(q);
  if (cos.defined()) {
    a.cos_tab = cos.data_ptr<float>(); a.sin_tab = sin.data_ptr<float>();
    a.cos_stride = cos.stride(0); a.sin_stride = sin.stride(0);
    if (q_rot.defined()) {
      a.q_rot = q_rot.data_ptr();
      a.qr_sb = q_rot.stride(0); a.qr_sh = q_rot.stride(1); a.qr_ss = q_rot.stride(2);
    }
  }
  check(k_rot.defined() ? ulm_attn_fwd_rope_qk(&a, k_rot.data_ptr(), k_rot.stride(0), k_rot.stride(1), k_rot.stride(2)) : ulm_attn_fwd(&a),
        "flash_attn_v100 forward");
}

void attn_backward(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o_in, const Tensor& lse, const Tensor& do_in,
                   const Tensor& dq, const Tensor& dk, const Tensor& dv, const AttnArgs& p, const Tensor& cos = Tensor(), const Tensor& sin = Tensor(),
                   int64_t mode = 7, const Tensor& delta_in = Tensor()) {
  const Tensor go = fa_ready(do_in) ? do_in : do_in.contiguous(), o = fa_ready(o_in) ? o_in : o_in.contiguous();
  const Tensor delta = delta_in.defined() ? delta_in : empty_cuda({q.size(0), q.size(1), q.size(2)}, at::kFloat, q);
  ulm_attn_bwd_args a{};
  a.q = q.data_ptr(); a.k = k.data_ptr(); a.v = v.data_ptr(); a.o = o.data_ptr(); a.d_o = go.data_ptr();
  a.lse = lse.data_ptr<float>(); a.delta = delta.data_ptr<float>();
  a.dq = dq.data_ptr(); a.dk = dk.data_ptr(); a.dv = dv.data_ptr();
  a.q_sb = q.stride(0); a.q_sh = q.stride(1); a.q_ss = q.stride(2);
  a.k_sb = k.stride(0); a.k_sh = k.stride(1); a.k_ss = k.stride(2);
  a.v_sb = v.stride(0); a.v_sh = v.stride(1); a.v_ss = v.stride(2);
  a.o_sb = o.stride(0); a.o_sh = o.stride(1); a.o_ss = o.stride(2);
  a.do_sb = go.stride(0); a.do_sh = go.stride(1); a.do_ss = go.stride(2);
  a.dq_sb = dq.stride(0); a.dq_sh = dq.stride(1); a.dq_ss = dq.stride(2);
  a.dk_sb = dk.stride(0); a.dk_sh = dk.stride(1); a.dk_ss = dk.stride(2);
  a.dv_sb = dv.stride(0); a.dv_sh = dv.stride(1); a.dv_ss = dv.stride(2);
  a.B = (int32_t)q.size(0); a.H = (int32_t)q.size(1); a.S = (int32_t)q.size(2);
  a.dtype = code_of(q.scalar_type()); a.causal = p.causal; a.mode = (int32_t)mode;
  a.softmax_scale = (float)p.scale; a.dropout_p = (float)p.dropout_p; a.seed = (uint32_t)p.seed;
  a.status_dev = status_ptr(q); a.stream = stream_of(q);
  if (cos.defined()) {
    a.cos_tab = cos.data_ptr<float>(); a.sin_tab = sin.data_ptr<float>();
    a.cos_stride = cos.stride(0); a.sin_stride = sin.stride(0);
  }
  check(ulm_attn_bwd(&a), "flash_attn_v100 backward");
}

Tensor empty_lse(const Tensor& q) { return empty_cuda({q.size(0), q.size(1), q.size(2)}, at::kFloat, q); }

// dq, dk, dv of one allocation, each (B,H,S,64) stored as (B,S,H,64)
std::array<Tensor, 3> empty_grads(const Tensor& q) {
  const int64_t B = q.size(0), H = q.size(1), S = q.size(2), n = B * H * S * 64;
  const Tensor buf = empty_cuda({3 * n}, q.scalar_type(), q);
  std::array<Tensor, 3> out;
  for (int i = 0; i < 3; ++i) out[i] = buf.as_strided({B, H, S, 64}, {S * H * 64, 64, H * 64, 1}, i * n);
  return out;
}

struct RopeBwd : OpNode {
  std::vector<int64_t> n, qs, ks;                          // shape and input strides
  variable_list backward(variable_list& g, const variable_list& kept) override {
    const bool has_q = g[0].defined(), has_k = g[1].defined();
    auto ready = [](const Tensor& t) {
      return t.stride(3) == 1 && !(reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) && t.stride(0) % 8 == 0 && t.stride(1) % 8 == 0 && t.stride(2) % 8 == 0;
    };
    const Tensor cos = kept[0], sin = kept[1];
    Tensor in[2], out[2];
    for (int i = 0; i < 2; ++i)
      if (g[i].defined()) {
        in[i] = ready(g[i]) ? g[i] : g[i].contiguous();
        out[i] = rope_out_like(n, i ? ks : qs, in[i]);
      }
    // a branch whose output went unused has a zero gradient: only the other one is rotated
    if (has_k) rope_launch(in[0], in[1], out[0], out[1], cos, sin, true);
    else rope_launch(Tensor(), in[0], Tensor(), out[0], cos, sin, true);
    for (int i = 0; i < 2; ++i)
      if (!out[i].defined()) out[i] = zero_grad(i);
    return {out[0], out[1]};
  }
};

std::tuple<Tensor, Tensor> rope(const Tensor& q, const Tensor& k, const Tensor& cos, const Tensor& sin) {
  TORCH_CHECK_VALUE(q.is_cuda() && k.is_cuda() && is_16bit(q.scalar_type()) && q.dim() == 4 && k.dim() == 4 && q.sizes() == k.sizes() && q.scalar_type() == k.scalar_type(),
                    "rope needs CUDA fp16/bf16 (B,H,S,64) tensors of one shape");
  Tensor qo, ko;
  {
    OpScope scope;
    c10::cuda::CUDAGuard dev(q.device());
    qo = rope_out_like(q.sizes(), q.strides(), q);
    ko = rope_out_like(k.sizes(), k.strides(), k);
    rope_launch(q, k, qo, ko, cos, sin, false);
  }
  if (!no_graph(q, k)) {
    auto node = make_node<RopeBwd>(q, k);
    node->n = q.sizes().vec(); node->qs = q.strides().vec(); node->ks = k.strides().vec();
    node->keep(cos); node->keep(sin);
    torch::autograd::set_history(qo, node);
    torch::autograd::set_history(ko, node);
  }
  return {qo, ko};
}

struct FlashBwd : OpNode {
  AttnArgs p{};
  variable_list backward(variable_list& g, const variable_list& kept) override {
    const Tensor q = kept[0];
    auto d = empty_grads(q);
    attn_backward(q, kept[1], kept[2], kept[3], kept[4], g[0], d[0], d[1], d[2], p);
    return {d[0], d[1], d[2]};
  }
};

Tensor flash_attn(const Tensor& q_in, const Tensor& k_in, const Tensor& v_in, double dropout_p, bool causal, double scale, int64_t seed) {
  TORCH_CHECK_VALUE(q_in.is_cuda() && is_16bit(q_in.scalar_type()) && q_in.dim() == 4 && q_in.size(3) == 64,
                    "flash_attn_v100 needs CUDA fp16/bf16 inputs with head_dim 64");
  const Tensor q = fa_ready(q_in) ? q_in : q_in.contiguous(), k = fa_ready(k_in) ? k_in : k_in.contiguous(), v = fa_ready(v_in) ? v_in : v_in.contiguous();
  const AttnArgs p{dropout_p, causal, scale, seed};
  Tensor o, lse;
  {
    OpScope scope;
    c10::cuda::CUDAGuard dev(q.device());
    o = empty_bshd(q.size(0), q.size(1), q.size(2), q);
    lse = empty_lse(q);
    attn_forward(q, k, v, o, lse, p);
  }
  if (!no_graph(q, k, v)) {
    auto node = make_node<FlashBwd>(q, k, v);
    node->p = p;
    torch::autograd::set_history(o, node);
    node->keep(q); node->keep(k); node->keep(v); node->keep(o, true); node->keep(lse);
  }
  return o;
}

// Where the RoPE work runs: 0 stand-alone kernels, 1 Q rotated inside the forward, 2 also the adjoint behind the
// backward kernels.  All give the same bits.
enum Fuse : int64_t { kFuseNone = 0, kFuseFwd = 1, kFuseAll = 2 };

// o and lse are written; returns the rotated (q, k)
std::pair<Tensor, Tensor> rope_attn_forward(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& cos, const Tensor& sin,
                                            const Tensor& o, const Tensor& lse, const AttnArgs& p, int64_t fuse) {
  const Tensor ko = rope_out_like(k.sizes(), k.strides(), k);
  Tensor qo;
  if (rope_in_tile(q.size(0), q.size(1), q.size(2))) {
    qo = rope_out_like(q.sizes(), q.strides(), q);
    attn_forward(q, k, v, o, lse, p, cos, sin, qo, ko);
  } else if (fuse == kFuseNone) {
    qo = rope_out_like(q.sizes(), q.strides(), q);
    rope_launch(q, k, qo, ko, cos, sin, false);
    attn_forward(qo, ko, v, o, lse, p);
  } else {
    qo = empty_bshd(q.size(0), q.size(1), q.size(2), q);
    rope_launch(Tensor(), k, Tensor(), ko, cos, sin, false);
    attn_forward(q, ko, v, o, lse, p, cos, sin, qo);
  }
  return {qo, ko};
}

// gradients of the UNROTATED q, k and of v.  The stand-alone adjoint runs in place: a thread reads both halves of
// what it rotates before it writes them, and the 16-bit gradients need no second buffer.
void rope_attn_backward(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, const Tensor& lse, const Tensor& go,
                        const Tensor& cos, const Tensor& sin, const Tensor& dq, const Tensor& dk, const Tensor& dv, const AttnArgs& p, int64_t fuse) {
  if (!cos.defined()) { attn_backward(q, k, v, o, lse, go, dq, dk, dv, p); return; }
  if (fuse == kFuseAll) { attn_backward(q, k, v, o, lse, go, dq, dk, dv, p, cos, sin); return; }
  attn_backward(q, k, v, o, lse, go, dq, dk, dv, p);
  rope_launch(dq, dk, dq, dk, cos, sin, true);
}

struct RopeFlashBwd : OpNode {
  AttnArgs p{};
  int64_t fuse = 0;
  variable_list backward(variable_list& g, const variable_list& kept) override {
    const Tensor q = kept[0];
    auto d = empty_grads(q);
    rope_attn_backward(q, kept[1], kept[2], kept[3], kept[4], g[0], kept[5], kept[6], d[0], d[1], d[2], p, fuse);
    return {d[0], d[1], d[2]};
  }
};

Tensor rope_flash_attn(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& cos, const Tensor& sin, double dropout_p, bool causal,
                       double scale, int64_t seed, int64_t fuse) {
  TORCH_CHECK_VALUE(rope_can_use(q, k, cos, sin) && can_use(q, k, v), "rope_flash_attn needs 16-bit (B,H,S,64) CUDA views and fp32 (S,64) tables");
  const AttnArgs p{dropout_p, causal, scale, seed};
  Tensor o, lse, qr, kr;
  {
    OpScope scope;
    c10::cuda::CUDAGuard dev(q.device());
    o = empty_bshd(q.size(0), q.size(1), q.size(2), q);
    lse = empty_lse(q);
    std::tie(qr, kr) = rope_attn_forward(q, k, v, cos, sin, o, lse, p, fuse);
  }
  if (!no_graph(q, k, v)) {
    auto node = make_node<RopeFlashBwd>(q, k, v);
    node->p = p; node->fuse = fuse;
    torch::autograd::set_history(o, node);
    node->keep(qr); node->keep(kr); node->keep(v); node->keep(o, true); node->keep(lse); node->keep(cos); node->keep(sin);
  }
  return o;
}

// Third `i` (0 q, 1 k, 2 v) of the first B*S rows of a contiguous [.., 3*H*64] tensor as a (B,H,S,64) view
Tensor qkv_part(const Tensor& qkv, int i, int64_t B, int64_t S, int64_t H) {
  const int64_t w = 3 * H * 64;
  return qkv.as_strided({B, H, S, 64}, {S * w, 64, w, 1}, qkv.storage_offset() + i * H * 64);
}
// the first B*S rows of a contiguous [.., H*64] tensor as a (B,H,S,64) view
Tensor heads_of(const Tensor& x, int64_t B, int64_t S, int64_t H) {
  return x.as_strided({B, H, S, 64}, {S * H * 64, 64, H * 64, 1}, x.storage_offset());
}

struct QkvBwd : OpNode {
  AttnArgs p{};
  int64_t fuse = 0, B = 0, S = 0, H = 0, rows = -1;        // rows >= 0: the flattened form with padding rows
  variable_list backward(variable_list& g, const variable_list& kept) override {
    const Tensor qkv = kept[0], cos = kept[5], sin = kept[6];
    const Tensor q = cos.defined() ? kept[1] : qkv_part(qkv, 0, B, S, H), k = cos.defined() ? kept[2] : qkv_part(qkv, 1, B, S, H);
    const Tensor go = heads_of(g[0].contiguous(), B, S, H);
    const Tensor d = empty_cuda(qkv.sizes(), qkv.scalar_type(), qkv);
    if (rows > B * S) d.narrow(0, B * S, rows - B * S).zero_();
    rope_attn_backward(q, k, qkv_part(qkv, 2, B, S, H), heads_of(kept[3], B, S, H), kept[4], go, cos, sin,
                       qkv_part(d, 0, B, S, H), qkv_part(d, 1, B, S, H), qkv_part(d, 2, B, S, H), p, fuse);
    return {d};
  }
};

Tensor qkv_attn(const Tensor& qkv, int64_t H, const OptTensor& cos_o, const OptTensor& sin_o, double dropout_p, bool causal, double scale,
                int64_t seed, int64_t fuse, int64_t flat_b, int64_t flat_s) {
  const bool flat = flat_b >= 0;
  TORCH_CHECK_VALUE(!flat || (qkv.dim() == 2 && qkv.size(0) >= flat_b * flat_s), "flat_shape=(n, L) needs a 2-D qkv with at least n*L rows");
  TORCH_CHECK_VALUE(qkv.is_cuda() && is_16bit(qkv.scalar_type()) && (flat || qkv.dim() == 3) && qkv.is_contiguous() && qkv.size(-1) == 3 * H * 64 &&
                        !(reinterpret_cast<uintptr_t>(qkv.data_ptr()) & 31),
                    "qkv_rope_flash_attn needs a contiguous CUDA fp16/bf16 [n, L, 3*n_heads*64] tensor");
  const int64_t B = flat ? flat_b : qkv.size(0), S = flat ? flat_s : qkv.size(1), rows = flat ? qkv.size(0) : -1;
  const Tensor cos = cos_o.value_or(Tensor()), sin = sin_o.value_or(Tensor());
  TORCH_CHECK_VALUE(cos.defined() == sin.defined(), "cos2d and sin2d must be given together");
  TORCH_CHECK_VALUE(!cos.defined() || (table_ok(cos, S, qkv) && table_ok(sin, S, qkv)),
                    "RoPE tables must be fp32 (L,64) views on the same device, 16-byte aligned rows");
  if (B * S == 0) {
    auto n = qkv.sizes().vec();
    n.back() = H * 64;
    return at::zeros(n, qkv.options()) + 0 * qkv.sum();
  }
  const AttnArgs p{dropout_p, causal, scale, seed};
  Tensor out, lse, qr, kr;
  {
    OpScope scope;
    c10::cuda::CUDAGuard dev(qkv.device());
    out = flat ? empty_cuda({rows, H * 64}, qkv.scalar_type(), qkv) : empty_cuda({B, S, H * 64}, qkv.scalar_type(), qkv);
    if (rows > B * S) out.narrow(0, B * S, rows - B * S).zero_();
    const Tensor o = heads_of(out, B, S, H), v = qkv_part(qkv, 2, B, S, H);
    const Tensor q = qkv_part(qkv, 0, B, S, H), k = qkv_part(qkv, 1, B, S, H);
    lse = empty_lse(q);
    if (cos.defined()) std::tie(qr, kr) = rope_attn_forward(q, k, v, cos, sin, o, lse, p, fuse);
    else attn_forward(q, k, v, o, lse, p);
  }
  if (!no_graph(qkv)) {
    auto node = make_node<QkvBwd>(qkv);
    node->p = p; node->fuse = fuse; node->B = B; node->S = S; node->H = H; node->rows = rows;
    torch::autograd::set_history(out, node);
    node->keep(qkv); node->keep(qr); node->keep(kr); node->keep(out, true); node->keep(lse); node->keep(cos); node->keep(sin);
  }
  return out;
}

// Forward alone, nothing kept.  Where Q and K are not rotated in their tile (rope_in_tile) the launch that rotates K takes Q
// along while the rotated copy stays in L2, against Q rotated inside the kernel, at the start of every CTA: 2-15 % for
// short sequences (12 heads x 67 x 128: 37.4 us against 40.7, x 300 x 64: 74.3 / 77.4), 0-4 % for long ones (16 x 4096 x 1:
// 63.7 / 66.4, x 4: 234 / 240; 12 x 4096 x 6: 277 / 273, within the spread).  From about 20 M elements the two are equal
// for short sequences (12 x 128 x 2048: 733 both) and the copy's traffic costs more for long ones (12 x 4096 x 8: 356 / 336).
constexpr int64_t kRopeAloneElems = 20 << 20;
std::tuple<Tensor, Tensor, Tensor> causal_attention(const Tensor& qkv_in, int64_t H, const OptTensor& cos_o, const OptTensor& sin_o, double scale) {
  TORCH_CHECK_VALUE(cos_o.has_value() == sin_o.has_value(), "cos and sin must be given together");
  OpScope scope;
  const Tensor qkv = qkv_in.detach();
  TORCH_CHECK_VALUE(qkv.is_cuda() && is_16bit(qkv.scalar_type()) && qkv.dim() == 3 && qkv.size(2) == 3 * H * 64 && (qkv.is_contiguous() || qkv.stride(2) == 1),
                    "causal_attention needs a CUDA fp16/bf16 [n, L, 3*n_heads*64] tensor with contiguous rows");
  c10::cuda::CUDAGuard dev(qkv.device());
  const int64_t B = qkv.size(0), S = qkv.size(1);
  // rows that lie further apart (a slice of a wider tensor) are read in place
  auto part = [&](int i) {
    return qkv.is_contiguous() ? qkv_part(qkv, i, B, S, H)
                               : qkv.as_strided({B, H, S, 64}, {qkv.stride(0), 64, qkv.stride(1), 1}, qkv.storage_offset() + i * H * 64);
  };
  const Tensor q = part(0), v = part(2), out = empty_cuda({B, S, H * 64}, qkv.scalar_type(), qkv);
  Tensor k = part(1), cos, sin;
  const Tensor lse = empty_lse(q);
  const AttnArgs p{0.0, true, scale, 0};
  if (cos_o) {
    // the model's [1, L, >=64] or [L, >=64] tables
    auto table = [&](const Tensor& t) {
      if (t.dim() == 2 && t.size(0) == S && t.size(1) == 64) return t;
      const Tensor t2 = t.reshape({-1, t.size(-1)});
      return t2.size(0) >= S && t2.size(1) >= 64 ? t2.as_strided({S, 64}, t2.strides(), t2.storage_offset()) : t2;
    };
    cos = table(*cos_o); sin = table(*sin_o);
    TORCH_CHECK_VALUE(rope_can_use(q, k, cos, sin), "causal_attention needs fp32 RoPE tables of at least 64 columns on the same device");
    const Tensor ko = rope_out_like(k.sizes(), k.strides(), k);
    if (rope_in_tile(B, H, S)) {
      attn_forward(q, k, v, heads_of(out, B, S, H), lse, p, cos, sin, Tensor(), ko);
      return {out, ko, v};
    }
    if (B * S * H * 64 <= kRopeAloneElems) {
      const Tensor qo = rope_out_like(q.sizes(), q.strides(), q);
      rope_launch(q, k, qo, ko, cos, sin, false);
      attn_forward(qo, ko, v, heads_of(out, B, S, H), lse, p);
      return {out, ko, v};
    }
    rope_launch(Tensor(), k, Tensor(), ko, cos, sin, false);
    k = ko;
  }
  attn_forward(q, k, v, heads_of(out, B, S, H), lse, p, cos, sin);
  return {out, k, v};
}

// ---------------------------------------------------------------------------
// single launches, as the reference's extension exposes them (tests and timings of one kernel)
// ---------------------------------------------------------------------------
std::tuple<Tensor, Tensor, OptTensor> single_forward(const Tensor& q, const Tensor& k, const Tensor& v, double dropout_p, bool causal, double scale, int64_t seed,
                                                     const OptTensor& cos, const OptTensor& sin, bool want_q_rot, const OptTensor& o_out) {
  OpScope scope;
  c10::cuda::CUDAGuard dev(q.device());
  const Tensor o = o_out ? *o_out : empty_bshd(q.size(0), q.size(1), q.size(2), q), lse = empty_lse(q);
  Tensor q_rot;
  if (cos && want_q_rot) q_rot = empty_bshd(q.size(0), q.size(1), q.size(2), q);
  attn_forward(q, k, v, o, lse, {dropout_p, causal, scale, seed}, cos.value_or(Tensor()), sin.value_or(Tensor()), q_rot);
  return {o, lse, q_rot.defined() ? OptTensor(q_rot) : std::nullopt};
}

std::array<Tensor, 3> single_backward(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, const Tensor& lse, const Tensor& go, double dropout_p,
                                      bool causal, double scale, int64_t seed, int64_t mode, const OptTensor& delta, const OptTensor& cos, const OptTensor& sin,
                                      const std::optional<std::array<Tensor, 3>>& out) {
  OpScope scope;
  c10::cuda::CUDAGuard dev(q.device());
  const std::array<Tensor, 3> d = out ? *out : empty_grads(q);
  attn_backward(q, k, v, o, lse, go, d[0], d[1], d[2], {dropout_p, causal, scale, seed}, cos.value_or(Tensor()), sin.value_or(Tensor()), mode,
                delta.value_or(Tensor()));
  return d;
}

std::tuple<OptTensor, Tensor> single_rope(const OptTensor& q, const Tensor& k, const Tensor& cos, const Tensor& sin, bool backward) {
  OpScope scope;
  c10::cuda::CUDAGuard dev(k.device());
  const Tensor ko = rope_out_like(k.sizes(), k.strides(), k), qo = q ? rope_out_like(q->sizes(), q->strides(), *q) : Tensor();
  rope_launch(q.value_or(Tensor()), k, qo, ko, cos, sin, backward);
  return {q ? OptTensor(qo) : std::nullopt, ko};
}

// o, lse, rotated q and k of unrotated q and k, and the gradients of those
std::array<Tensor, 4> single_rope_forward(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& cos, const Tensor& sin, double dropout_p, bool causal,
                                          double scale, int64_t seed, int64_t fuse) {
  OpScope scope;
  c10::cuda::CUDAGuard dev(q.device());
  const Tensor o = empty_bshd(q.size(0), q.size(1), q.size(2), q), lse = empty_lse(q);
  auto [qr, kr] = rope_attn_forward(q, k, v, cos, sin, o, lse, {dropout_p, causal, scale, seed}, fuse);
  return {o, lse, qr, kr};
}
std::array<Tensor, 3> single_rope_backward(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, const Tensor& lse, const Tensor& go, const Tensor& cos,
                                           const Tensor& sin, double dropout_p, bool causal, double scale, int64_t seed, int64_t fuse) {
  OpScope scope;
  c10::cuda::CUDAGuard dev(q.device());
  auto d = empty_grads(q);
  rope_attn_backward(q, k, v, o, lse, go, cos, sin, d[0], d[1], d[2], {dropout_p, causal, scale, seed}, fuse);
  return d;
}

// ---------------------------------------------------------------------------
// RMSNorm, SwiGLU
// ---------------------------------------------------------------------------
// [.., d] as [rows, d] with contiguous 16-byte aligned rows
Tensor rows_of(const Tensor& x) {
  const Tensor x2 = x.dim() == 2 ? x : x.reshape({-1, x.size(-1)});
  const bool ok = x2.stride(1) == 1 && !(reinterpret_cast<uintptr_t>(x2.data_ptr()) & 15) && (x2.stride(0) * x2.element_size()) % 16 == 0;
  return ok ? x2 : x2.contiguous();
}
int y_kind(at::ScalarType y, at::ScalarType x) { return y == x ? ULM_Y_SAME : y == at::kHalf ? ULM_Y_F16 : ULM_Y_BF16; }

// dx (and d_branch) and dw of one norm; ga: the gradient reaching the normalised tensor from elsewhere
Tensor norm_backward(const Tensor& x, const Tensor& w, const Tensor& rstd, const Tensor& dy, double eps, int kind, const Tensor& dx,
                     const Tensor& ga, const Tensor& d_branch) {
  const int64_t rows = x.size(0), d = x.size(1);
  const Tensor dw = empty_cuda({d}, at::kFloat, x);
  const Tensor partial = empty_cuda({ulm_rmsnorm_bwd_partial_rows(rows), d}, at::kFloat, x);
  ulm_rmsnorm_bwd_args a{};
  a.x = x.data_ptr(); a.w = w.data_ptr(); a.dy = dy.data_ptr(); a.rstd = rstd.data_ptr<float>();
  a.dx = dx.data_ptr(); a.dw = dw.data_ptr<float>(); a.partial = partial.data_ptr<float>();
  a.x_stride = x.stride(0); a.dy_stride = dy.stride(0); a.dx_stride = dx.stride(0);
  a.rows = rows; a.d = (int32_t)d; a.x_dtype = code_of(x.scalar_type()); a.w_dtype = code_of(w.scalar_type());
  a.eps = (float)eps; a.stream = stream_of(x); a.dy_kind = kind;
  if (ga.defined()) { a.g_add = ga.data_ptr(); a.gadd_stride = ga.stride(0); }
  if (d_branch.defined()) { a.d_branch = d_branch.data_ptr(); a.dbranch_stride = d_branch.stride(0); }
  check(ulm_rmsnorm_bwd(&a), d_branch.defined() ? "add_rms_norm backward" : "rms_norm backward");
  return dw;
}

struct NormBwd : OpNode {
  double eps = 0;
  std::vector<int64_t> shape;
  at::ScalarType wdtype, ydtype;
  variable_list backward(variable_list& g, const variable_list& kept) override {
    const Tensor x = kept[0], w = kept[1], rstd = kept[2];
    const Tensor dy = rows_of(g[0].to(ydtype)), dx = empty_cuda({x.size(0), x.size(1)}, x.scalar_type(), x);
    const Tensor dw = norm_backward(x, w, rstd, dy, eps, y_kind(ydtype, x.scalar_type()), dx, Tensor(), Tensor());
    return {dx.view(shape), dw.to(wdtype)};
  }
};

Tensor rms_norm(const Tensor& x, const Tensor& weight, double eps, std::optional<at::ScalarType> out_dtype) {
  TORCH_CHECK_VALUE(x.is_cuda() && known(x.scalar_type()), "rms_norm needs a CUDA fp16/bf16/fp32 tensor");
  at::ScalarType yt = x.scalar_type();
  if (out_dtype) yt = *out_dtype;
  else if (yt == at::kFloat && at::autocast::is_autocast_enabled(at::kCUDA)) yt = at::autocast::get_autocast_dtype(at::kCUDA);
  TORCH_CHECK_VALUE(yt == x.scalar_type() || (x.scalar_type() == at::kFloat && is_16bit(yt)),
                    "rms_norm: a different output dtype needs an fp32 input and a 16-bit output");
  Tensor y, x2, w, rstd;
  {
    OpScope scope;
    c10::cuda::CUDAGuard dev(x.device());
    x2 = rows_of(x);
    const int64_t rows = x2.size(0), d = x2.size(1);
    y = empty_cuda(x.sizes(), yt, x);
    rstd = empty_cuda({rows}, at::kFloat, x);
    w = weight.scalar_type() == x.scalar_type() || weight.scalar_type() == at::kFloat ? weight : weight.to(at::kFloat);
    w = w.contiguous();
    ulm_rmsnorm_fwd_args a{};
    a.x = x2.data_ptr(); a.w = w.data_ptr(); a.y = y.data_ptr(); a.rstd = rstd.data_ptr<float>();
    a.x_stride = x2.stride(0); a.y_stride = d; a.rows = rows; a.d = (int32_t)d;
    a.x_dtype = code_of(x.scalar_type()); a.w_dtype = code_of(w.scalar_type()); a.eps = (float)eps; a.stream = stream_of(x);
    a.y_kind = y_kind(yt, x.scalar_type());
    check(ulm_rmsnorm_fwd(&a), "rms_norm forward");
  }
  if (!no_graph(x, weight)) {
    auto node = make_node<NormBwd>(x, weight);
    node->eps = eps; node->shape = x.sizes().vec(); node->wdtype = weight.scalar_type(); node->ydtype = yt;
    node->keep(x2); node->keep(w); node->keep(rstd);
    torch::autograd::set_history(y, node);
  }
  return y;
}

struct AddNormBwd : OpNode {
  double eps = 0;
  std::vector<int64_t> shape;
  at::ScalarType wdtype, bdtype;
  variable_list backward(variable_list& g, const variable_list& kept) override {
    if (!g[1].defined()) return {g[0], g[0].to(bdtype), zero_grad(2)};      // the normalised output went unused
    const Tensor x = kept[0], w = kept[1], rstd = kept[2];
    const int64_t rows = x.size(0), d = x.size(1);
    const Tensor dy = rows_of(g[1].to(bdtype)), ga = g[0].defined() ? rows_of(g[0].to(at::kFloat)) : Tensor();
    const Tensor dx = empty_cuda({rows, d}, at::kFloat, x), db = empty_cuda({rows, d}, bdtype, x);
    const Tensor dw = norm_backward(x.view({rows, d}), w, rstd, dy, eps, y_kind(bdtype, at::kFloat), dx, ga, db);
    return {dx.view(shape), db.view(shape), dw.to(wdtype)};
  }
};

std::tuple<Tensor, Tensor> add_rms_norm(const Tensor& x, const Tensor& branch, const Tensor& weight, double eps) {
  TORCH_CHECK_VALUE(x.is_cuda() && x.scalar_type() == at::kFloat && is_16bit(branch.scalar_type()) && branch.sizes() == x.sizes(),
                    "add_rms_norm needs an fp32 CUDA x and a 16-bit branch of the same shape");
  TORCH_CHECK_VALUE(x.size(-1) <= 1024 && x.size(-1) % 4 == 0, "add_rms_norm takes rows of at most 1024 elements, a multiple of 4");
  Tensor x_new, y, w, rstd;
  {
    OpScope scope;
    c10::cuda::CUDAGuard dev(x.device());
    const Tensor x2 = rows_of(x), b2 = rows_of(branch);
    const int64_t rows = x2.size(0), d = x2.size(1);
    x_new = empty_cuda(x.sizes(), at::kFloat, x);
    y = empty_cuda(x.sizes(), branch.scalar_type(), x);
    rstd = empty_cuda({rows}, at::kFloat, x);
    w = weight.to(at::kFloat).contiguous();
    ulm_rmsnorm_fwd_args a{};
    a.x = x2.data_ptr(); a.w = w.data_ptr(); a.y = y.data_ptr(); a.rstd = rstd.data_ptr<float>();
    a.x_stride = x2.stride(0); a.y_stride = d; a.rows = rows; a.d = (int32_t)d;
    a.x_dtype = ULM_F32; a.w_dtype = ULM_F32; a.eps = (float)eps; a.stream = stream_of(x); a.y_kind = y_kind(branch.scalar_type(), at::kFloat);
    a.branch = b2.data_ptr(); a.x_out = x_new.data_ptr(); a.branch_stride = b2.stride(0); a.xout_stride = d;
    check(ulm_rmsnorm_fwd(&a), "add_rms_norm forward");
  }
  if (!no_graph(x, branch, weight)) {
    auto node = make_node<AddNormBwd>(x, branch, weight);
    node->eps = eps; node->shape = x.sizes().vec(); node->wdtype = weight.scalar_type(); node->bdtype = branch.scalar_type();
    torch::autograd::set_history(x_new, node);
    torch::autograd::set_history(y, node);
    node->keep(x_new, true); node->keep(w); node->keep(rstd);
  }
  return {x_new, y};
}

struct SwigluBwd : OpNode {
  variable_list backward(variable_list& g, const variable_list& kept) override {
    const Tensor a = kept[0], b = kept[1], dy = g[0].to(a.scalar_type()).contiguous();
    const Tensor da = empty_cuda(a.sizes(), a.scalar_type(), a), db = empty_cuda(a.sizes(), a.scalar_type(), a);
    ulm_swiglu_args p{a.data_ptr(), b.data_ptr(), nullptr, dy.data_ptr(), da.data_ptr(), db.data_ptr(), a.numel(), code_of(a.scalar_type()), 0, stream_of(a)};
    check(ulm_swiglu_bwd(&p), "swiglu backward");
    return {da, db};
  }
};

Tensor swiglu(const Tensor& a_in, const Tensor& b_in) {
  TORCH_CHECK_VALUE(a_in.is_cuda() && known(a_in.scalar_type()) && b_in.scalar_type() == a_in.scalar_type() && b_in.sizes() == a_in.sizes(),
                    "swiglu needs two CUDA tensors of one shape and one of fp16/bf16/fp32");
  Tensor a, b, y;
  {
    OpScope scope;
    c10::cuda::CUDAGuard dev(a_in.device());
    a = a_in.contiguous(); b = b_in.contiguous();
    y = empty_cuda(a.sizes(), a.scalar_type(), a);
    ulm_swiglu_args p{a.data_ptr(), b.data_ptr(), y.data_ptr(), nullptr, nullptr, nullptr, a.numel(), code_of(a.scalar_type()), 0, stream_of(a)};
    check(ulm_swiglu_fwd(&p), "swiglu forward");
  }
  if (!no_graph(a_in, b_in)) {
    auto node = make_node<SwigluBwd>(a_in, b_in);
    node->keep(a); node->keep(b);
    torch::autograd::set_history(y, node);
  }
  return y;
}

// ---------------------------------------------------------------------------
// linear layers
// ---------------------------------------------------------------------------
// What `wgrad_in_place` and `weight_cast_scope` switch on belongs to the thread that entered them and to the backward
// passes it starts there: it travels in the thread-local state that autograd hands to its workers.  Another thread, with
// another model, sees neither.
//
// A cast scope keeps the 16-bit copy of a leaf weight and reuses it, on the stream that made it.  Keyed by the parameter's
// implementation object, which an entry keeps alive.  A closed scope, which a worker may still hold, gives nothing.
struct CastScope {
  struct Entry { Tensor param, copy; int64_t stream; };
  std::mutex mu;
  bool open = true;
  std::unordered_map<const c10::TensorImpl*, Entry> made;
};
struct OpContext : c10::SafePyObject {
  bool wgrad_in_place = false;
  std::shared_ptr<CastScope> casts;
  OpContext() : SafePyObject(nullptr, nullptr) {}
};
using ContextPtr = std::shared_ptr<c10::SafePyObject>;
const std::string kContextKey = "ulm_ops";
ContextPtr context() {
  using TLS = at::impl::ThreadLocalPythonObjects;
  return TLS::contains(kContextKey) ? TLS::get(kContextKey) : nullptr;
}
const OpContext& context_of(const ContextPtr& c) {
  static const OpContext none;
  return c ? static_cast<const OpContext&>(*c) : none;
}
bool wgrad_in_place() { return context_of(context()).wgrad_in_place; }
int64_t stream_id(const Tensor& t) { return t.is_cuda() ? (int64_t)c10::cuda::getCurrentCUDAStream(t.device().index()).id() : 0; }

// The state a context manager found and puts back on leaving; `casts` is the scope it opened, if it did.
struct ContextToken { ContextPtr before; std::shared_ptr<CastScope> casts; };
ContextToken enter_context(const std::function<void(OpContext&)>& change) {
  ContextToken t{context(), nullptr};
  auto next = std::make_shared<OpContext>();
  next->wgrad_in_place = context_of(t.before).wgrad_in_place;
  next->casts = context_of(t.before).casts;
  change(*next);
  if (next->casts != context_of(t.before).casts) t.casts = next->casts;
  at::impl::ThreadLocalPythonObjects::set(kContextKey, next);
  return t;
}
void leave_context(ContextToken& t) {
  if (t.casts) {
    decltype(t.casts->made) gone;                        // the tensors are released outside the lock
    std::lock_guard<std::mutex> lock(t.casts->mu);
    t.casts->open = false;
    gone.swap(t.casts->made);
  }
  at::impl::ThreadLocalPythonObjects::set(kContextKey, t.before ? t.before : std::make_shared<OpContext>());
}

// 16-bit copies of a fixed set of fp32 weights in one buffer, in the given order: one fused cast fills them all where a
// scope would otherwise make each on first use (a launch and about 12 us of host time per weight), and weights that
// follow one another in the list do so in memory, so that two projections of one input can run as one GEMM.  A training
// program keeps the object and refreshes it once per step.
struct WeightCopies {
  std::vector<Tensor> params, views;
  WeightCopies(std::vector<Tensor> ps, at::ScalarType dtype) : params(std::move(ps)) {
    if (params.empty()) return;
    OpScope scope;
    int64_t n = 0;
    for (const Tensor& p : params) n += (p.numel() + 7) / 8 * 8;              // 16-byte aligned starts
    const Tensor flat = at::empty({n}, params[0].options().dtype(dtype).requires_grad(false));
    int64_t off = 0;
    for (const Tensor& p : params) {
      views.push_back(flat.narrow(0, off, p.numel()).view(p.sizes()));
      off += (p.numel() + 7) / 8 * 8;
    }
  }
  void refresh() {
    if (params.empty()) return;
    OpScope scope;
    // the buffer outlives a step and may be filled and read on another stream than the one it was allocated on: what is
    // queued there has to end before the allocator hands the memory out again
    if (views[0].is_cuda())
      c10::cuda::CUDACachingAllocator::recordStream(views[0].storage().data_ptr(), c10::cuda::getCurrentCUDAStream(views[0].device().index()));
    at::_foreach_copy_(views, params);
  }
};

// `copies` (already refreshed, on the current stream) seeds the scope
ContextToken enter_casts(const std::shared_ptr<WeightCopies>& copies) {
  auto scope = std::make_shared<CastScope>();
  if (copies)
    for (size_t i = 0; i < copies->params.size(); ++i)
      scope->made[copies->params[i].unsafeGetTensorImpl()] = {copies->params[i], copies->views[i], stream_id(copies->views[i])};
  return enter_context([&](OpContext& c) { c.casts = scope; });
}
Tensor cast_cached(const Tensor& weight, at::ScalarType dtype) {
  if (weight.scalar_type() == dtype) return weight;
  const ContextPtr held = context();
  const std::shared_ptr<CastScope>& scope = context_of(held).casts;
  if (!scope || !weight.is_leaf()) return weight.detach().to(dtype);
  const c10::TensorImpl* key = weight.unsafeGetTensorImpl();
  const int64_t stream = stream_id(weight);
  {
    std::lock_guard<std::mutex> lock(scope->mu);
    auto it = scope->made.find(key);
    if (it != scope->made.end() && it->second.copy.scalar_type() == dtype && it->second.copy.device() == weight.device() && it->second.stream == stream)
      return it->second.copy;
  }
  const Tensor c = weight.detach().to(dtype);
  std::lock_guard<std::mutex> lock(scope->mu);
  if (scope->open) scope->made.insert_or_assign(key, CastScope::Entry{weight, c, stream});
  return c;
}

// dW = dy^T x for autograd, or an undefined tensor after adding it into weight.grad in place
Tensor weight_grad(const Tensor& weight, const Tensor& dy, const Tensor& x) {
  const bool half_gemm = dy.is_cuda() && is_16bit(dy.scalar_type());
  if (half_gemm && wgrad_in_place()) {
    Tensor g = weight.grad();
    if (g.defined() && g.scalar_type() == at::kFloat && g.is_contiguous()) {
      at::addmm_out(g, g, dy.t(), x, at::kFloat);
      return Tensor();
    }
  }
  // fp32 parameters get the fp32 sums directly: no 16-bit rounding and no cast pass
  if (half_gemm && weight.scalar_type() == at::kFloat) return at::mm(dy.t(), x, at::kFloat);
  return at::mm(dy.t(), x).to(weight.scalar_type());
}

struct LinearBwd : OpNode {
  at::ScalarType cd, x_dtype;
  variable_list backward(variable_list& g, const variable_list& kept) override {
    const Tensor x = kept[0], weight = kept[1];
    const Tensor dy = g[0].reshape({-1, g[0].size(-1)}).to(cd);
    Tensor dx, dw;
    if (task_should_compute_output(0)) dx = at::mm(dy, cast_cached(weight, cd)).view(x.sizes()).to(x_dtype);
    if (task_should_compute_output(1)) dw = weight_grad(weight, dy, x.reshape({-1, x.size(-1)}));
    return {dx, dw};
  }
  // two library GEMMs, which autograd can differentiate
  variable_list backward_recorded(variable_list& g, const variable_list& kept) override {
    c10::impl::ExcludeDispatchKeyGuard no_autocast{c10::DispatchKeySet(c10::DispatchKey::AutocastCUDA)};
    const Tensor x = kept[0], weight = kept[1];
    const Tensor dy = g[0].reshape({-1, g[0].size(-1)}).to(cd);
    Tensor dx, dw;
    if (task_should_compute_output(0)) dx = at::mm(dy, cast_cached(weight, cd)).view(x.sizes()).to(x_dtype);
    if (task_should_compute_output(1)) dw = at::mm(dy.t(), x.reshape({-1, x.size(-1)})).to(weight.scalar_type());
    return {dx, dw};
  }
};

Tensor linear(const Tensor& x, const Tensor& weight) {
  at::ScalarType cd = x.scalar_type();
  if (x.is_cuda() && at::autocast::is_autocast_enabled(at::kCUDA)) cd = at::autocast::get_autocast_dtype(at::kCUDA);
  Tensor xc, y;
  {
    OpScope scope;
    c10::OptionalDeviceGuard dev(x.device());
    xc = x.to(cd);
    const Tensor wt = cast_cached(weight, cd).t();
    if (xc.dim() == 2) {
      y = at::mm(xc, wt);
    } else {
      auto n = xc.sizes().vec();
      n.back() = weight.size(0);
      y = at::mm(xc.reshape({-1, xc.size(-1)}), wt).view(n);
    }
  }
  if (!no_graph(x, weight)) {
    auto node = make_node<LinearBwd>(x, weight);
    node->cd = cd; node->x_dtype = x.scalar_type();
    node->keep(xc); node->keep(weight);
    torch::autograd::set_history(y, node);
  }
  return y;
}

// ---------------------------------------------------------------------------
// gated projections: silu(x w1^T) * (x w3^T)
// ---------------------------------------------------------------------------
// Two equal-shaped contiguous matrices that follow one another in one storage, as one matrix; undefined otherwise
Tensor stacked(const Tensor& a, const Tensor& b) {
  if (!a.is_contiguous() || !b.is_contiguous() || a.scalar_type() != b.scalar_type() || !a.storage().is_alias_of(b.storage()) ||
      b.storage_offset() != a.storage_offset() + a.numel())
    return Tensor();
  return a.as_strided({a.size(0) + b.size(0), a.size(1)}, {a.size(1), 1}, a.storage_offset());
}

void swiglu_rows(const Tensor& ab, const Tensor& y, const Tensor& dy, const Tensor& dab, bool backward) {
  const int64_t d = ab.size(1) / 2, half = d * ab.element_size();
  auto at_half = [&](const Tensor& t, int h) -> void* { return t.defined() ? static_cast<char*>(t.data_ptr()) + h * half : nullptr; };
  ulm_swiglu_args p{at_half(ab, 0), at_half(ab, 1), at_half(y, 0), at_half(dy, 0), at_half(dab, 0), at_half(dab, 1), ab.size(0) * d,
                    code_of(ab.scalar_type()), 0, stream_of(ab)};
  check(ulm_swiglu_rows(&p, backward, d, 2 * d), backward ? "swiglu backward" : "swiglu forward");
}

struct GatedBwd : OpNode {
  at::ScalarType cd, x_dtype;
  variable_list backward(variable_list& g, const variable_list& kept) override {
    const Tensor x = kept[0], w1 = kept[1], w3 = kept[2], ab = kept[3];
    const Tensor dy = g[0].reshape({-1, g[0].size(-1)}).to(cd).contiguous(), x2 = x.reshape({-1, x.size(-1)});
    const Tensor dab = empty_cuda(ab.sizes(), cd, ab);
    swiglu_rows(ab, Tensor(), dy, dab, true);
    const int64_t ff = w1.size(0);
    const Tensor da = dab.narrow(1, 0, ff), db = dab.narrow(1, ff, ff);
    Tensor dx, dw1, dw3;
    if (task_should_compute_output(0)) {
      const Tensor c1 = cast_cached(w1, cd), c3 = cast_cached(w3, cd), both = stacked(c1, c3);
      dx = both.defined() ? at::mm(dab, both) : at::mm(da, c1).addmm_(db, c3);      // one GEMM sums the two branches in fp32
      dx = dx.view(x.sizes()).to(x_dtype);
    }
    const bool need1 = task_should_compute_output(1), need3 = task_should_compute_output(2);
    if (need1 && need3) {
      const Tensor g1 = w1.grad(), g3 = w3.grad();
      if (is_16bit(cd) && wgrad_in_place() && g1.defined() && g3.defined() && g1.scalar_type() == at::kFloat) {
        Tensor both = stacked(g1, g3);
        if (both.defined()) {
          at::addmm_out(both, both, dab.t(), x2, at::kFloat);
          return {dx, Tensor(), Tensor()};
        }
      } else if (is_16bit(cd) && w1.scalar_type() == at::kFloat && w3.scalar_type() == at::kFloat) {
        const Tensor dw = at::mm(dab.t(), x2, at::kFloat);
        return {dx, dw.narrow(0, 0, ff), dw.narrow(0, ff, ff)};
      }
    }
    if (need1) dw1 = weight_grad(w1, da, x2);
    if (need3) dw3 = weight_grad(w3, db, x2);
    return {dx, dw1, dw3};
  }
};

// Both projections write the two halves of one [rows, 2 ff] matrix: as one GEMM where the weights' 16-bit copies lie one
// behind the other (WeightCopies).  Against two linears and a gate that is one GEMM less forward, two less backward,
// and no pass that adds the two branches' gradients of x.
Tensor gated_linear(const Tensor& x, const Tensor& w1, const Tensor& w3) {
  at::ScalarType cd = x.scalar_type();
  if (x.is_cuda() && at::autocast::is_autocast_enabled(at::kCUDA)) cd = at::autocast::get_autocast_dtype(at::kCUDA);
  const int64_t ff = w1.size(0);
  if (!x.is_cuda() || !known(cd) || w3.sizes() != w1.sizes() || ff % (16 / (int64_t)c10::elementSize(cd))) return ::swiglu(::linear(x, w1), ::linear(x, w3));
  Tensor xc, ab, y;
  {
    OpScope scope;
    c10::cuda::CUDAGuard dev(x.device());
    xc = x.to(cd);
    const Tensor x2 = xc.reshape({-1, xc.size(-1)}), c1 = cast_cached(w1, cd), c3 = cast_cached(w3, cd), both = stacked(c1, c3);
    if (both.defined()) {
      ab = at::mm(x2, both.t());
    } else {
      ab = empty_cuda({x2.size(0), 2 * ff}, cd, x2);
      Tensor a = ab.narrow(1, 0, ff), b = ab.narrow(1, ff, ff);
      at::mm_out(a, x2, c1.t());
      at::mm_out(b, x2, c3.t());
    }
    auto n = xc.sizes().vec();
    n.back() = ff;
    y = empty_cuda(n, cd, x2);
    swiglu_rows(ab, y, Tensor(), Tensor(), false);
  }
  if (!no_graph(x, w1, w3)) {
    auto node = make_node<GatedBwd>(x, w1, w3);
    node->cd = cd; node->x_dtype = x.scalar_type();
    node->keep(xc); node->keep(w1); node->keep(w3); node->keep(ab);
    torch::autograd::set_history(y, node);
  }
  return y;
}

// ---------------------------------------------------------------------------
// lm head + cross-entropy, the form that keeps the 16-bit logits between forward and backward
// ---------------------------------------------------------------------------
// operands, scratch and stream of one lm-head launch; `part` holds the fp32 scratch
ulm_lmhead_lse_args lmhead_args(const Tensor& h, const Tensor& w, int64_t ignore_index, Tensor& part) {
  TORCH_CHECK_VALUE(is_16bit(h.scalar_type()) && w.scalar_type() == h.scalar_type(), "lm_head_lse takes fp16 or bf16 operands of one dtype");
  TORCH_CHECK_VALUE(h.dim() == 2 && w.dim() == 2 && h.size(1) == w.size(1) && h.stride(1) == 1 && w.stride(1) == 1,
                    "lm_head_lse takes hidden [rows, d] and weight [V, d] with contiguous rows");
  const int64_t rows = h.size(0), d = h.size(1), V = w.size(0);
  const int64_t n_part = std::max<int64_t>(rows, 1) * ulm_lmhead_parts(rows, (int32_t)V);
  part = empty_cuda({3, n_part}, at::kFloat, h);
  ulm_lmhead_lse_args a{};
  a.h = h.data_ptr(); a.w = w.data_ptr();
  a.part_m = part.data_ptr<float>(); a.part_s = a.part_m + n_part;
  a.h_stride = h.stride(0); a.w_stride = w.stride(0);
  a.rows = rows; a.V = (int32_t)V; a.d = (int32_t)d; a.dtype = code_of(h.scalar_type());
  a.ignore_index = ignore_index; a.status_dev = status_ptr(h); a.stream = stream_of(h);
  return a;
}

// -> lse, loss rows (undefined without targets or logits), logits (undefined unless kept)
std::tuple<Tensor, Tensor, Tensor> lm_head_lse(const Tensor& h, const Tensor& w, const OptTensor& target, int64_t ignore_index, bool keep_logits) {
  OpScope scope;
  c10::cuda::CUDAGuard dev(h.device());
  Tensor part, logits, loss;
  ulm_lmhead_lse_args a = lmhead_args(h, w, ignore_index, part);
  const Tensor lse = empty_cuda({a.rows}, at::kFloat, h);
  a.lse = lse.data_ptr<float>();
  if (keep_logits) { logits = empty_cuda({a.rows, a.V}, h.scalar_type(), h); a.logits = logits.data_ptr(); a.z_stride = a.V; }
  if (keep_logits && target) { loss = empty_cuda({a.rows}, at::kFloat, h); a.loss = loss.data_ptr<float>(); a.target = target->data_ptr<int64_t>(); }
  check(ulm_lmhead_lse(&a), "lm-head GEMM + LSE");
  return {lse, loss, logits};
}

// -> loss rows, whether the target has the row's largest logit (uint8)
std::tuple<Tensor, Tensor> lm_head_score(const Tensor& h, const Tensor& w, const Tensor& target, int64_t ignore_index) {
  OpScope scope;
  c10::cuda::CUDAGuard dev(h.device());
  TORCH_CHECK_VALUE(target.scalar_type() == at::kLong && target.is_contiguous() && target.numel() == h.size(0), "lm_head_score takes one int64 target per row");
  Tensor part;
  ulm_lmhead_lse_args a = lmhead_args(h, w, ignore_index, part);
  const Tensor loss = empty_cuda({a.rows}, at::kFloat, h), hit = empty_cuda({a.rows}, at::kByte, h);
  a.loss = loss.data_ptr<float>(); a.target = target.data_ptr<int64_t>();
  check(ulm_lmhead_score(&a, hit.data_ptr<uint8_t>(), reinterpret_cast<int32_t*>(a.part_s + part.size(1))), "lm-head GEMM + score");
  return {loss, hit};
}

// The kernel's form of ulm_ops.token_targets; empty where the tensors are not what it reads (device, type, shape)
std::optional<std::tuple<Tensor, Tensor>> token_targets(const Tensor& ids, const Tensor& labels, int64_t padded, int64_t ignore_index) {
  if (!ids.is_cuda() || labels.device() != ids.device() || ids.scalar_type() != at::kLong || labels.scalar_type() != at::kLong || ids.dim() != 2 ||
      labels.sizes() != ids.sizes() || !ids.is_contiguous() || !labels.is_contiguous())
    return std::nullopt;
  const int64_t n = ids.size(0), L = ids.size(1);
  TORCH_CHECK_VALUE(padded >= n * L, "token_targets: ", padded, " rows do not hold ", n, " x ", L, " tokens");
  OpScope scope;
  c10::cuda::CUDAGuard dev(ids.device());
  const Tensor out = empty_cuda({2, padded}, at::kLong, ids), flat = out.select(0, 0), target = out.select(0, 1);
  check(ulm_token_targets(ids.data_ptr<int64_t>(), labels.data_ptr<int64_t>(), n, L, padded, ignore_index, flat.data_ptr<int64_t>(),
                          target.data_ptr<int64_t>(), stream_of(ids)), "token_targets");
  return std::make_tuple(flat, target);
}

Tensor grad_clip(const Tensor& flat, const Tensor& sumsq, double max_norm) {
  auto ok = [&](const Tensor& t) { return t.is_cuda() && t.device() == flat.device() && t.scalar_type() == at::kFloat && t.is_contiguous(); };
  TORCH_CHECK_VALUE(ok(flat) && ok(sumsq) && sumsq.numel() >= 1, "grad_clip_ takes contiguous fp32 gradients and their squared norm on one CUDA device");
  OpScope scope;
  c10::cuda::CUDAGuard dev(flat.device());
  const Tensor norm = empty_cuda({}, at::kFloat, flat);
  check(ulm_grad_clip(flat.data_ptr<float>(), flat.numel(), sumsq.data_ptr<float>(), (float)max_norm, norm.data_ptr<float>(), stream_of(flat)), "grad_clip");
  return norm;
}

// One int64 target per row of `hidden`, where the cross-entropy kernels can read it
void check_target(const Tensor& hidden, const Tensor& target) {
  TORCH_CHECK_VALUE(target.scalar_type() == at::kLong && target.device() == hidden.device() && target.numel() >= hidden.size(0),
                    "chunked_cross_entropy takes one int64 target per row, on the device of hidden");
}

struct KeptCeBwd : OpNode {
  int64_t ignore_index = 0;
  at::ScalarType cd;
  std::atomic<bool> consumed{false};
  variable_list backward(variable_list& g, const variable_list& kept) override {
    const Tensor hidden = kept[0], weight = kept[1], target = kept[2], lse = kept[3], logits = kept[4], inv = kept[5], wc = kept[6], hc = kept[7];
    TORCH_CHECK(!consumed.exchange(true),
                "chunked_cross_entropy: the kept logits were turned into their gradient in place by the first backward; a second "
                "backward through the same graph is not supported");
    const Tensor gs = g[0].to(at::kFloat).mul(inv);                            // d loss / d row loss
    ulm_ce_bwd_args a{};
    a.logits = logits.data_ptr(); a.target = target.data_ptr<int64_t>(); a.lse = lse.data_ptr<float>();
    a.gscale_dev = gs.data_ptr<float>(); a.gscale = 1.f;
    a.row_stride = logits.stride(0); a.rows = logits.size(0); a.V = (int32_t)logits.size(1); a.dtype = code_of(cd);
    a.ignore_index = ignore_index; a.stream = stream_of(logits);
    check(ulm_ce_bwd(&a), "cross-entropy backward");                             // in place over the kept logits
    Tensor dh, dw;
    if (task_should_compute_output(0)) dh = at::mm(logits, wc).to(hidden.scalar_type());
    if (task_should_compute_output(1)) dw = weight_grad(weight, logits, hc);
    return {dh, dw};
  }
};

Tensor kept_cross_entropy(const Tensor& hidden, const Tensor& weight, const Tensor& target, int64_t ignore_index, at::ScalarType cd,
                          const OptTensor& denom_dev, double denom, bool fused) {
  check_target(hidden, target);
  Tensor loss, lse, rows_loss, logits, inv, wc, hc;
  {
    OpScope scope;
    c10::cuda::CUDAGuard dev(hidden.device());
    wc = cast_cached(weight, cd);
    hc = hidden.to(cd);
    if (fused && is_16bit(cd) && hc.size(1) % 64 == 0 && wc.size(0) % 64 == 0 && hc.is_contiguous() && wc.is_contiguous()) {
      std::tie(lse, rows_loss, logits) = lm_head_lse(hc, wc, target, ignore_index, true);
    } else {
      logits = at::mm(hc, wc.t());
      lse = empty_cuda({logits.size(0)}, at::kFloat, hc);
      rows_loss = empty_cuda({logits.size(0)}, at::kFloat, hc);
      ulm_ce_fwd_args a{logits.data_ptr(), target.data_ptr<int64_t>(), lse.data_ptr<float>(), rows_loss.data_ptr<float>(),
                        logits.stride(0), logits.size(0), (int32_t)logits.size(1), code_of(cd), ignore_index, stream_of(hc)};
      check(ulm_ce_fwd(&a), "cross-entropy forward");
    }
    loss = empty_cuda({}, at::kFloat, hc);                  // sum of the row losses / denominator
    inv = empty_cuda({}, at::kFloat, hc);                   // 1 / denominator
    Tensor dd;
    if (denom_dev) dd = denom_dev->to(hidden.device(), at::kFloat);
    check(ulm_loss_mean(rows_loss.data_ptr<float>(), target.data_ptr<int64_t>(), rows_loss.size(0), ignore_index,
                        dd.defined() ? dd.data_ptr<float>() : nullptr, (float)denom, loss.data_ptr<float>(), inv.data_ptr<float>(), stream_of(hc)),
          "loss mean");
  }
  if (!no_graph(hidden, weight)) {
    auto node = make_node<KeptCeBwd>(hidden, weight);
    node->ignore_index = ignore_index; node->cd = cd;
    node->keep(hidden); node->keep(weight); node->keep(target); node->keep(lse); node->keep(logits); node->keep(inv); node->keep(wc); node->keep(hc);
    torch::autograd::set_history(loss, node);
  }
  return loss;
}

// ---------------------------------------------------------------------------
// bindings
// ---------------------------------------------------------------------------
template <typename T> bool has_tangent(const T&) { return false; }
bool has_tangent(const Tensor& t) { return t.defined() && t._fw_grad(/*level=*/0).defined(); }

// A differentiable op.  A tracer, a functorch level or a forward-mode tangent would not notice a node made in C++: there
// the call goes through a Python autograd function (ulm_recorded.py), which each of them knows how to record or refuse.
template <typename R, typename... A>
void def_op(pybind11::module_& m, const char* name, R (*f)(A...)) {
  m.def(name, [name, f](A... a) -> pybind11::object {
    if (torch::jit::tracer::isTracing() || c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode) ||
        (c10::AutogradState::get_tls_state().get_fw_grad_mode() && (has_tangent(a) || ...)))
      return pybind11::module_::import("ulm_recorded").attr("Recorded").attr("apply")(name, a...);
    auto run = [&]() -> R {
      pybind11::gil_scoped_release nogil;
      return f(a...);
    };
    return pybind11::cast(run());
  });
}

}  // namespace

PYBIND11_MODULE(_ulm_torch, m) {
  namespace py = pybind11;
  using no_gil = py::call_guard<py::gil_scoped_release>;
  m.def("status_tensor", &status_tensor, no_gil());
  m.def("fa_ready", &fa_ready);
  m.def("can_use", &can_use);
  m.def("rope_can_use", &rope_can_use);
  def_op(m, "rope", &::rope);
  def_op(m, "flash_attn", &::flash_attn);
  def_op(m, "rope_flash_attn", &::rope_flash_attn);
  def_op(m, "qkv_attn", &::qkv_attn);
  m.def("attn_forward", &single_forward, no_gil());
  m.def("attn_backward", &single_backward, no_gil());
  m.def("rope_launch", &single_rope, no_gil());
  m.def("rope_attn_forward", &single_rope_forward, no_gil());
  m.def("rope_attn_backward", &single_rope_backward, no_gil());
  m.def("causal_attention", &causal_attention, no_gil());
  def_op(m, "rms_norm", &::rms_norm);
  def_op(m, "add_rms_norm", &::add_rms_norm);
  def_op(m, "swiglu", &::swiglu);
  py::class_<ContextToken>(m, "ContextToken").def("leave", &leave_context);
  m.def("enter_wgrad_in_place", [](bool on) { return enter_context([on](OpContext& c) { c.wgrad_in_place = on; }); });
  py::class_<WeightCopies, std::shared_ptr<WeightCopies>>(m, "WeightCopies")
      .def(py::init<std::vector<Tensor>, at::ScalarType>())
      .def_readonly("views", &WeightCopies::views)
      .def("refresh", &WeightCopies::refresh, no_gil());
  m.def("enter_casts", &enter_casts);
  m.def("cast_cached", &cast_cached, no_gil());
  m.def("weight_grad", [](const Tensor& w, const Tensor& dy, const Tensor& x) -> OptTensor {
    OpScope scope;
    Tensor g = weight_grad(w, dy, x);
    return g.defined() ? OptTensor(g) : std::nullopt;
  }, no_gil());
  def_op(m, "linear", &::linear);
  def_op(m, "gated_linear", &::gated_linear);
  m.def("lm_head_lse", &lm_head_lse, no_gil());
  m.def("lm_head_score", &lm_head_score, no_gil());
  m.def("token_targets", &token_targets, no_gil());
  m.def("grad_clip", &grad_clip, no_gil());
  m.def("check_target", &check_target);
  def_op(m, "kept_cross_entropy", &::kept_cross_entropy);
}
