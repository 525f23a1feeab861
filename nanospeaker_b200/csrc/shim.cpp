// The pybind shim over the C ABI: the block (and the FFN sublayer around it) called on torch tensors,
// with the backward as a native autograd node. A step through Python (ctypes marshalling, one
// torch.empty per kept tensor, a Python autograd function) cost the host 330 us on top of the 90 us
// that the library's launches take; this side of the call is about 30 us, so that a step of a few
// thousand tokens is bound by the GPU again.
//
// Only memory, streams and autograd are torch's: every kernel is launched through the C ABI, whose
// addresses the Python binding hands over (bind()), so that it and this file use one library.
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/CUDAGraph.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/autograd/variable.h>
#include <torch/extension.h>

#include <algorithm>
#include <array>
#include <atomic>
#include <memory>
#include <mutex>
#include <optional>
#include <vector>

#include "../../include/moe_b200.h"

namespace {

using at::Tensor;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;
using OptTensor = std::optional<Tensor>;

// ------------------------------------------------------------------------------ the C ABI
struct Abi {
  decltype(&moe_b200_error_string) error_string;
  decltype(&moe_b200_block_kept_bytes) kept_bytes;
  decltype(&moe_b200_block_forward_scratch_bytes) forward_scratch_bytes;
  decltype(&moe_b200_block_backward_scratch_bytes) backward_scratch_bytes;
  decltype(&moe_b200_block_forward) forward;
  decltype(&moe_b200_block_backward) backward;
  decltype(&moe_b200_muon_scratch_bytes) muon_scratch_bytes;
  decltype(&moe_b200_muon_step) muon_step;
  decltype(&moe_b200_rmsnorm) rmsnorm;
  decltype(&moe_b200_rmsnorm_bwd) rmsnorm_bwd;
} abi{};

py::object* status_word_of = nullptr;   // device index -> address of its status word
std::atomic<int64_t> n_launched{0};

template <typename F>
void take(const py::dict& d, const char* name, F& f) {
  f = reinterpret_cast<F>(d[name].cast<uintptr_t>());
}
void bind(const py::dict& d, const py::object& status) {
  take(d, "moe_b200_error_string", abi.error_string);
  take(d, "moe_b200_block_kept_bytes", abi.kept_bytes);
  take(d, "moe_b200_block_forward_scratch_bytes", abi.forward_scratch_bytes);
  take(d, "moe_b200_block_backward_scratch_bytes", abi.backward_scratch_bytes);
  take(d, "moe_b200_block_forward", abi.forward);
  take(d, "moe_b200_block_backward", abi.backward);
  take(d, "moe_b200_muon_scratch_bytes", abi.muon_scratch_bytes);
  take(d, "moe_b200_muon_step", abi.muon_step);
  take(d, "moe_b200_rmsnorm", abi.rmsnorm);
  take(d, "moe_b200_rmsnorm_bwd", abi.rmsnorm_bwd);
  status_word_of = new py::object(status);   // lives as long as the process
}

void check(int rc, const char* what) {
  TORCH_CHECK(rc == MOE_B200_OK, what, " failed: ", abi.error_string(rc), " (code ", rc, ")");
}

constexpr int MAX_DEVICES = 64;
int32_t* status_word(int device) {
  static std::atomic<int32_t*> words[MAX_DEVICES] = {};
  TORCH_CHECK(device >= 0 && device < MAX_DEVICES, "device index ", device);
  int32_t* w = words[device].load(std::memory_order_acquire);
  if (w == nullptr) {
    py::gil_scoped_acquire gil;
    w = reinterpret_cast<int32_t*>((*status_word_of)(device).cast<uintptr_t>());
    words[device].store(w, std::memory_order_release);
  }
  return w;
}

// Two more streams per device for the independent branches of the backward; the library forks them
// from the caller's stream and joins them back with events, so callers (and graph capture) only
// ever see the current stream.
struct SideStreams {
  c10::cuda::CUDAStream a, b;
};
const SideStreams& side_streams(int device) {
  static std::mutex m;
  static std::optional<SideStreams> s[MAX_DEVICES];
  std::lock_guard<std::mutex> lock(m);
  if (!s[device])
    s[device] = SideStreams{c10::cuda::getStreamFromPool(false, device),
                            c10::cuda::getStreamFromPool(false, device)};
  return *s[device];
}

// ----------------------------------------------------------------------------- the block
struct Options {
  int64_t top_k, activation, capacity;
  bool normalize, full_softmax, store, mm_logits, one_stream;
  double aux_coef;
};
// The tensors of one call, undefined where absent; all bf16, contiguous, on one device.
struct Operands {
  Tensor x, router_w, logits, w_in, w_out, w_sh_in, w_sh_out, b_in, b_out, b_sh_in, b_sh_out;
  Tensor logit_bias, noise, residual;
};
inline const void* ptr(const Tensor& t) { return t.defined() ? t.const_data_ptr() : nullptr; }

moe_b200_block_desc describe(const Operands& p, const Options& o) {
  moe_b200_block_desc d{};
  d.n_tokens = p.x.size(0);
  d.d_model = int32_t(p.x.size(1));
  d.d_hidden = int32_t(p.w_in.size(2) / 2);
  d.n_experts = int32_t(p.w_in.size(0));
  d.n_shared = p.w_sh_in.defined() ? int32_t(p.w_sh_in.size(0)) : 0;
  d.top_k = int32_t(o.top_k);
  d.normalize = o.normalize;
  d.full_softmax = o.full_softmax;
  d.activation = int32_t(o.activation);
  d.store_combine = o.store;
  d.capacity = int32_t(o.capacity);
  d.aux_coef = float(o.aux_coef);
  d.x = ptr(p.x);
  d.router_w = ptr(p.router_w);
  d.logits_in = ptr(p.logits);
  d.logit_bias = static_cast<const float*>(ptr(p.logit_bias));
  d.noise = static_cast<const float*>(ptr(p.noise));
  d.w_in = ptr(p.w_in);
  d.w_out = ptr(p.w_out);
  d.w_sh_in = ptr(p.w_sh_in);
  d.w_sh_out = ptr(p.w_sh_out);
  d.b_in = ptr(p.b_in);
  d.b_out = ptr(p.b_out);
  d.b_sh_in = ptr(p.b_sh_in);
  d.b_sh_out = ptr(p.b_sh_out);
  d.residual = ptr(p.residual);
  d.status = status_word(p.x.get_device());
  return d;
}

void check_operands(const Operands& p, const Options& o) {
  const Tensor& x = p.x;
  TORCH_CHECK(x.dim() == 2 && p.w_in.dim() == 3 && p.w_out.dim() == 3 && p.router_w.dim() == 2,
              "x [T, D], router_w [D, E], w_in [E, D, 2H], w_out [E, H, D] expected");
  const int64_t t = x.size(0), d = x.size(1), e = p.w_in.size(0), h = p.w_in.size(2) / 2;
  auto shaped = [&](const Tensor& v, at::IntArrayRef want, at::ScalarType dtype, const char* name) {
    if (!v.defined()) return;
    TORCH_CHECK(v.sizes() == want && v.scalar_type() == dtype && v.get_device() == x.get_device() &&
                    v.is_contiguous(),
                name, ": expected a contiguous ", dtype, " tensor of shape ", want, " beside x");
  };
  const auto bf = at::kBFloat16;
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == bf,
              "moe_b200 kernels need CUDA bf16 tensors, got ", x.device(), " ", x.scalar_type(),
              "; there is no CPU or other-dtype implementation behind these ops");
  shaped(x, {t, d}, bf, "x");
  shaped(p.router_w, {d, e}, bf, "router_w");
  shaped(p.w_in, {e, d, 2 * h}, bf, "w_in");
  shaped(p.w_out, {e, h, d}, bf, "w_out");
  TORCH_CHECK(p.w_sh_in.defined() == p.w_sh_out.defined(), "w_sh_in and w_sh_out go together");
  if (p.w_sh_in.defined()) {
    const int64_t s = p.w_sh_in.size(0);
    shaped(p.w_sh_in, {s, d, 2 * h}, bf, "w_sh_in");
    shaped(p.w_sh_out, {s, h, d}, bf, "w_sh_out");
    shaped(p.b_sh_in, {s, 2 * h}, bf, "b_sh_in");
    shaped(p.b_sh_out, {s, d}, bf, "b_sh_out");
  }
  shaped(p.b_in, {e, 2 * h}, bf, "b_in");
  shaped(p.b_out, {e, d}, bf, "b_out");
  shaped(p.logit_bias, {e}, at::kFloat, "logit_bias");
  shaped(p.noise, {t, e}, at::kFloat, "noise");
  shaped(p.residual, {t, d}, bf, "residual");
  TORCH_CHECK(o.top_k >= 1 && o.top_k <= e, "top_k ", o.top_k, " of ", e, " experts");
}

Tensor bytes_like(const Tensor& x, size_t n) {
  return at::empty({int64_t(n)}, x.options().dtype(at::kByte));
}

struct Results {
  Tensor out, aux, counts, dropped, kept;
};

// The forward's launches (no autograd here). p.logits is filled in when the caller wants torch's
// own matmul to form them.
Results launch_forward(Operands& p, const Options& o, bool train) {
  const c10::cuda::CUDAGuard on(p.x.device());
  if (o.mm_logits) p.logits = at::mm(p.x, p.router_w);
  const moe_b200_block_desc d = describe(p, o);
  Results r;
  r.out = at::empty_like(p.x);
  r.aux = at::empty({}, o.full_softmax ? p.x.options().dtype(at::kFloat) : p.x.options());
  r.counts = at::empty({d.n_experts}, p.x.options().dtype(at::kInt));
  if (o.capacity > 0) r.dropped = at::empty({}, p.x.options().dtype(at::kLong));
  const size_t kept = abi.kept_bytes(&d, train), scratch = abi.forward_scratch_bytes(&d);
  r.kept = bytes_like(p.x, kept);
  const Tensor tmp = bytes_like(p.x, scratch);
  int32_t n = 0;
  check(abi.forward(&d, train, r.out.mutable_data_ptr(), r.aux.mutable_data_ptr(),
                    !o.full_softmax, r.counts.mutable_data_ptr<int32_t>(),
                    r.dropped.defined() ? r.dropped.mutable_data_ptr<int64_t>() : nullptr,
                    r.kept.mutable_data_ptr(), kept, tmp.mutable_data_ptr(), scratch, &n,
                    c10::cuda::getCurrentCUDAStream().stream()),
        "moe_b200_block_forward");
  n_launched += n;
  return r;
}

struct Grads {
  Tensor dx, d_router, dw_in, dw_out, dw_sh_in, dw_sh_out, db_in, db_out, db_sh_in, db_sh_out;
};

Grads empty_grads(const Operands& p) {
  Grads g;
  g.dx = at::empty_like(p.x);
  g.d_router = at::empty_like(p.router_w);
  g.dw_in = at::empty_like(p.w_in);
  g.dw_out = at::empty_like(p.w_out);
  if (p.w_sh_in.defined()) {
    g.dw_sh_in = at::empty_like(p.w_sh_in);
    g.dw_sh_out = at::empty_like(p.w_sh_out);
  }
  return g;
}

// Fills g (empty_grads); the biases' gradients come with it.
void launch_backward(const Operands& p, const Options& o, const Tensor& kept,
                     const Tensor& grad_out, const Tensor& grad_aux, Grads& g) {
  const c10::cuda::CUDAGuard on(p.x.device());
  const moe_b200_block_desc d = describe(p, o);
  const int64_t e = d.n_experts, s = d.n_shared;
  Tensor db_in, db_out;   // one row per group of both weight stacks
  if (p.b_in.defined() || p.b_sh_in.defined())
    db_in = at::empty({e + s, p.w_in.size(2)}, p.x.options());
  if (p.b_out.defined() || p.b_sh_out.defined())
    db_out = at::empty({e + s, d.d_model}, p.x.options());
  const size_t scratch = abi.backward_scratch_bytes(&d);
  const Tensor tmp = bytes_like(p.x, scratch);
  // (memory of this stream is used on the side streams too: the library joins them back before it
  // returns, so whatever reuses the memory later is ordered after them)
  void *sa = nullptr, *sb = nullptr;
  if (!o.one_stream) {
    const SideStreams& side = side_streams(p.x.get_device());
    sa = side.a.stream();
    sb = side.b.stream();
  }
  auto mut = [](const Tensor& t) { return t.defined() ? t.mutable_data_ptr() : nullptr; };
  int32_t n = 0;
  check(abi.backward(&d, grad_out.const_data_ptr(),
                     static_cast<const float*>(ptr(grad_aux)), kept.const_data_ptr(),
                     size_t(kept.numel()), mut(g.dx), mut(g.d_router), mut(g.dw_in), mut(g.dw_out),
                     mut(g.dw_sh_in), mut(g.dw_sh_out), mut(db_in), mut(db_out),
                     tmp.mutable_data_ptr(), scratch, sa, sb, &n,
                     c10::cuda::getCurrentCUDAStream().stream()),
        "moe_b200_block_backward");
  n_launched += n;
  if (p.b_in.defined()) g.db_in = db_in.narrow(0, 0, e);
  if (p.b_sh_in.defined()) g.db_sh_in = db_in.narrow(0, e, s);
  if (p.b_out.defined()) g.db_out = db_out.narrow(0, 0, e);
  if (p.b_sh_out.defined()) g.db_sh_out = db_out.narrow(0, e, s);
}
Grads launch_backward(const Operands& p, const Options& o, const Tensor& kept,
                      const Tensor& grad_out, const Tensor& grad_aux) {
  const c10::cuda::CUDAGuard on(p.x.device());
  Grads g = empty_grads(p);
  launch_backward(p, o, kept, grad_out, grad_aux, g);
  return g;
}

// ------------------------------------------------------------------------------- autograd
// Operands held for the backward.
struct SavedOperands {
  SavedVariable x, router_w, logits, w_in, w_out, w_sh_in, w_sh_out, b_in, b_out, b_sh_in, b_sh_out,
      logit_bias, noise, kept;
  void save(const Operands& p, const Tensor& kept_buffer) {
    auto hold = [](const Tensor& t) { return SavedVariable(t, false); };
    x = hold(p.x);
    router_w = hold(p.router_w);
    logits = hold(p.logits);
    w_in = hold(p.w_in);
    w_out = hold(p.w_out);
    w_sh_in = hold(p.w_sh_in);
    w_sh_out = hold(p.w_sh_out);
    b_in = hold(p.b_in);
    b_out = hold(p.b_out);
    b_sh_in = hold(p.b_sh_in);
    b_sh_out = hold(p.b_sh_out);
    logit_bias = hold(p.logit_bias);
    noise = hold(p.noise);
    kept = hold(kept_buffer);
  }
  Operands unpack() const {
    Operands p;
    p.x = x.unpack();
    p.router_w = router_w.unpack();
    p.logits = logits.unpack();
    p.w_in = w_in.unpack();
    p.w_out = w_out.unpack();
    p.w_sh_in = w_sh_in.unpack();
    p.w_sh_out = w_sh_out.unpack();
    p.b_in = b_in.unpack();
    p.b_out = b_out.unpack();
    p.b_sh_in = b_sh_in.unpack();
    p.b_sh_out = b_sh_out.unpack();
    p.logit_bias = logit_bias.unpack();
    p.noise = noise.unpack();
    return p;
  }
  void release() {
    for (SavedVariable* v : {&x, &router_w, &logits, &w_in, &w_out, &w_sh_in, &w_sh_out, &b_in,
                             &b_out, &b_sh_in, &b_sh_out, &logit_bias, &noise, &kept})
      v->reset_data();
  }
};

Tensor as_grad(const Tensor& g, const Tensor& like) {
  if (!g.defined()) return at::zeros_like(like);
  return g.to(like.scalar_type()).contiguous();
}
Tensor as_grad_aux(const Tensor& g) {
  return g.defined() ? g.to(at::kFloat).reshape({1}) : Tensor();
}

// What a backward returns. It is made without grad mode, so that under create_graph the gradients would
// pass for constants; differentiating them again is an error.
variable_list once(variable_list grads) {
  if (!at::GradMode::is_enabled()) return grads;
  for (Tensor& g : grads)
    if (g.defined()) g = g.detach().set_requires_grad(true);
  auto error = std::make_shared<torch::autograd::DelayedError>(
      "the MoE block's backward cannot be differentiated again", int64_t(grads.size()));
  return (*error)(std::move(grads));
}

// Edges, in order: x, router_w, w_in, w_out, w_sh_in, w_sh_out, b_in, b_out, b_sh_in, b_sh_out,
// residual.
struct MoEBlockBackward : public torch::autograd::Node {
  SavedOperands saved;
  Options opt;
  bool has_residual = false;
  std::string name() const override { return "MoEBlockBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    saved.release();
  }
  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    if (!grads[0].defined() && !grads[1].defined()) return variable_list(11);
    return once(gradients(grads));
  }

 private:
  variable_list gradients(const variable_list& grads) {
    const Operands p = saved.unpack();
    const Tensor kept = saved.kept.unpack();
    at::NoGradGuard no_grad;
    const Tensor go = as_grad(grads[0], p.x);
    Grads g = launch_backward(p, opt, kept, go, as_grad_aux(grads[1]));
    return {g.dx, g.d_router, g.dw_in, g.dw_out, g.dw_sh_in, g.dw_sh_out, g.db_in, g.db_out,
            g.db_sh_in, g.db_sh_out, has_residual ? go : Tensor()};
  }
};

// Edges: x, gamma, router_w, w_in, w_out, w_sh_in, w_sh_out. out = x + block(rmsnorm(x) * gamma).
struct MoESublayerBackward : public torch::autograd::Node {
  SavedOperands saved;      // of the block: its x is the normalised input
  SavedVariable x, gamma, rstd;
  Options opt;
  std::string name() const override { return "MoESublayerBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    saved.release();
    for (SavedVariable* v : {&x, &gamma, &rstd}) v->reset_data();
  }
  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    if (!grads[0].defined() && !grads[1].defined()) return variable_list(7);
    return once(gradients(grads));
  }

 private:
  variable_list gradients(const variable_list& grads) {
    const Operands p = saved.unpack();
    const Tensor kept = saved.kept.unpack();
    const Tensor xx = x.unpack(), gm = gamma.unpack(), rs = rstd.unpack();
    at::NoGradGuard no_grad;
    const Tensor go = as_grad(grads[0], xx);
    Grads g = launch_backward(p, opt, kept, go, as_grad_aux(grads[1]));
    const c10::cuda::CUDAGuard on(xx.device());
    const Tensor dx = at::empty_like(xx);
    const Tensor dgamma = at::zeros({xx.size(1)}, xx.options().dtype(at::kFloat));
    check(abi.rmsnorm_bwd(g.dx.const_data_ptr(), xx.const_data_ptr(), rs.const_data_ptr<float>(),
                          gm.const_data_ptr(), go.const_data_ptr(), xx.size(0),
                          int32_t(xx.size(1)), dx.mutable_data_ptr(),
                          dgamma.mutable_data_ptr<float>(),
                          c10::cuda::getCurrentCUDAStream().stream()),
          "moe_b200_rmsnorm_bwd");
    ++n_launched;
    return {dx, dgamma.to(gm.scalar_type()), g.d_router, g.dw_in, g.dw_out, g.dw_sh_in,
            g.dw_sh_out};
  }
};

template <typename... T>
bool any_grad(const T&... t) {
  return at::GradMode::is_enabled() && ((t.defined() && t.requires_grad()) || ...);
}
// The nodes here have no forward-mode derivative; an operand's would be dropped without a word.
template <typename... T>
void refuse_forward_mode(const T&... t) {
  TORCH_CHECK_NOT_IMPLEMENTED(!((t.defined() && t._fw_grad(0).defined()) || ...),
                              "the MoE block does not support forward mode AD");
}
template <typename N>
std::shared_ptr<N> new_node() {
  return std::shared_ptr<N>(new N(), torch::autograd::deleteNode);
}

// A parameter as the kernels take it: x's dtype (what autocast would do; the gradient flows back
// through the cast), contiguous.
Tensor operand(const OptTensor& t, const Tensor& x) {
  if (!t || !t->defined()) return {};
  return (t->scalar_type() == x.scalar_type() ? *t : t->to(x.scalar_type())).contiguous();
}
Tensor fp32(const OptTensor& t) {
  if (!t || !t->defined()) return {};
  return (t->scalar_type() == at::kFloat ? *t : t->to(at::kFloat)).contiguous();
}

Operands operands(const Tensor& x, const Tensor& router_w, const OptTensor& logit_bias,
                  const OptTensor& noise, const Tensor& w_in, const Tensor& w_out,
                  const OptTensor& w_sh_in, const OptTensor& w_sh_out) {
  Operands p;
  p.x = x.contiguous();
  p.router_w = operand(router_w, x);
  p.logit_bias = fp32(logit_bias);
  p.noise = fp32(noise);
  p.w_in = operand(w_in, x);
  p.w_out = operand(w_out, x);
  p.w_sh_in = operand(w_sh_in, x);
  p.w_sh_out = operand(w_sh_out, x);
  return p;
}

// (out, aux, counts, dropped): the whole block on x [T, D].
std::tuple<Tensor, Tensor, Tensor, OptTensor> block(
    const Tensor& x, const Tensor& router_w, const OptTensor& logit_bias, const OptTensor& noise,
    const Tensor& w_in, const Tensor& w_out, const OptTensor& w_sh_in, const OptTensor& w_sh_out,
    const OptTensor& b_in, const OptTensor& b_out, const OptTensor& b_sh_in,
    const OptTensor& b_sh_out, const OptTensor& residual, int64_t top_k, bool normalize,
    bool full_softmax, double aux_coef, int64_t activation, int64_t capacity, bool store,
    bool mm_logits, bool one_stream) {
  Operands p = operands(x, router_w, logit_bias, noise, w_in, w_out, w_sh_in, w_sh_out);
  p.b_in = operand(b_in, x);
  p.b_out = operand(b_out, x);
  p.b_sh_in = operand(b_sh_in, x);
  p.b_sh_out = operand(b_sh_out, x);
  p.residual = operand(residual, x);
  const Options o{top_k, activation, capacity, normalize, full_softmax, store, mm_logits,
                  one_stream, aux_coef};
  check_operands(p, o);
  std::shared_ptr<MoEBlockBackward> node;
  if (any_grad(p.x, p.router_w, p.w_in, p.w_out, p.w_sh_in, p.w_sh_out, p.b_in, p.b_out, p.b_sh_in,
               p.b_sh_out, p.residual)) {
    refuse_forward_mode(p.x, p.router_w, p.w_in, p.w_out, p.w_sh_in, p.w_sh_out, p.b_in, p.b_out,
                        p.b_sh_in, p.b_sh_out, p.residual);
    node = new_node<MoEBlockBackward>();
    node->set_next_edges(torch::autograd::collect_next_edges(
        p.x, p.router_w, p.w_in, p.w_out, p.w_sh_in, p.w_sh_out, p.b_in, p.b_out, p.b_sh_in,
        p.b_sh_out, p.residual));
  }
  Results r;
  {
    at::NoGradGuard no_grad;
    r = launch_forward(p, o, node != nullptr);
  }
  if (node) {
    node->saved.save(p, r.kept);
    node->opt = o;
    node->has_residual = p.residual.defined();
    torch::autograd::set_history(r.out, node);
    if (o.full_softmax)
      torch::autograd::set_history(r.aux, node);
    else
      node->add_input_metadata(torch::autograd::Node::undefined_input());
  }
  return {r.out, r.aux, r.counts, r.dropped.defined() ? OptTensor(r.dropped) : OptTensor()};
}

// (out, aux, counts): x + block(rmsnorm(x) * gamma) on x [T, D].
std::tuple<Tensor, Tensor, Tensor> sublayer(
    const Tensor& x_in, const Tensor& gamma_in, double eps, const Tensor& router_w,
    const OptTensor& logit_bias, const Tensor& w_in, const Tensor& w_out, const OptTensor& w_sh_in,
    const OptTensor& w_sh_out, int64_t top_k, bool normalize, bool full_softmax, double aux_coef,
    int64_t activation, bool store, bool one_stream) {
  const Tensor x = x_in.contiguous(), gamma = operand(gamma_in, x);
  Operands p = operands(x, router_w, logit_bias, OptTensor(), w_in, w_out, w_sh_in, w_sh_out);
  const Options o{top_k, activation, 0, normalize, full_softmax, store, false, one_stream,
                  aux_coef};
  check_operands(p, o);
  TORCH_CHECK(gamma.dim() == 1 && gamma.size(0) == x.size(1), "gamma: expected [", x.size(1), "]");
  refuse_forward_mode(x, gamma, p.router_w, p.w_in, p.w_out, p.w_sh_in, p.w_sh_out);
  std::shared_ptr<MoESublayerBackward> node;
  if (any_grad(x, gamma, p.router_w, p.w_in, p.w_out, p.w_sh_in, p.w_sh_out)) {
    node = new_node<MoESublayerBackward>();
    node->set_next_edges(torch::autograd::collect_next_edges(x, gamma, p.router_w, p.w_in, p.w_out,
                                                             p.w_sh_in, p.w_sh_out));
  }
  Results r;
  Tensor rstd;
  {
    at::NoGradGuard no_grad;
    const c10::cuda::CUDAGuard on(x.device());
    p.x = at::empty_like(x);
    rstd = at::empty({x.size(0)}, x.options().dtype(at::kFloat));
    check(abi.rmsnorm(x.const_data_ptr(), gamma.const_data_ptr(), x.size(0), int32_t(x.size(1)),
                      float(eps), p.x.mutable_data_ptr(), rstd.mutable_data_ptr<float>(),
                      c10::cuda::getCurrentCUDAStream().stream()),
          "moe_b200_rmsnorm");
    ++n_launched;
    p.residual = x;
    r = launch_forward(p, o, node != nullptr);
    p.residual = Tensor();   // the backward adds its gradient itself
  }
  if (node) {
    node->saved.save(p, r.kept);
    node->x = SavedVariable(x, false);
    node->gamma = SavedVariable(gamma, false);
    node->rstd = SavedVariable(rstd, false);
    node->opt = o;
    torch::autograd::set_history(r.out, node);
    if (o.full_softmax)
      torch::autograd::set_history(r.aux, node);
    else
      node->add_input_metadata(torch::autograd::Node::undefined_input());
  }
  return {r.out, r.aux, r.counts};
}

// --------------------------------------------------------------------- replay from graphs
// The block's training step for one input shape, forward and backward each captured in a CUDA graph
// and replayed behind an autograd node. Inputs and incoming gradients are copied into the graphs'
// own buffers. The forward's results are those buffers (overwritten by the next call); a gradient is
// whoever's it has become: autograd takes it as p.grad without a copy, and a second micro-step adds to
// it. So the backward replays into buffers that nobody else holds: a trainer that clears its gradients
// always meets the first set, one that accumulates has the first set as p.grad and the second on the
// way, and where those two are both held the last set's results leave as copies.
class GraphedBlock : public std::enable_shared_from_this<GraphedBlock> {
 public:
  GraphedBlock(const Tensor& x, const Tensor& router_w, const OptTensor& logit_bias,
               const Tensor& w_in, const Tensor& w_out, const OptTensor& w_sh_in,
               const OptTensor& w_sh_out, int64_t top_k, bool normalize, bool full_softmax,
               double aux_coef, int64_t activation, bool store, int64_t warmup_iters)
      : opt_{top_k, activation, 0, normalize, full_softmax, store, false, false, aux_coef} {
    at::NoGradGuard no_grad;
    const c10::cuda::CUDAGuard on(x.device());
    auto plain = [](const Tensor& t) { return t.defined() ? t.detach() : t; };
    p_ = operands(x.clone(), router_w, logit_bias, OptTensor(), w_in, w_out, w_sh_in, w_sh_out);
    for (Tensor* t : {&p_.x, &p_.router_w, &p_.w_in, &p_.w_out, &p_.w_sh_in, &p_.w_sh_out,
                      &p_.logit_bias})
      *t = plain(*t);
    check_operands(p_, opt_);
    grad_out_ = at::zeros_like(p_.x);
    grad_aux_ = at::zeros({1}, p_.x.options().dtype(at::kFloat));
    // at least once outside the capture: lazy initialisations, the status word, the side streams
    const auto main = c10::cuda::getCurrentCUDAStream();
    const auto side = c10::cuda::getStreamFromPool(false, p_.x.get_device());
    C10_CUDA_CHECK(cudaStreamSynchronize(main.stream()));
    {
      const c10::cuda::CUDAStreamGuard work(side);
      for (int64_t i = 0; i < std::max<int64_t>(1, warmup_iters); ++i) {
        Results r = launch_forward(p_, opt_, true);
        launch_backward(p_, opt_, r.kept, grad_out_, grad_aux_);
      }
      C10_CUDA_CHECK(cudaStreamSynchronize(side.stream()));
      const int64_t l0 = n_launched;
      fwd_.capture_begin();
      r_ = launch_forward(p_, opt_, true);
      fwd_.capture_end();
      n_fwd_ = n_launched - l0;
      capture_backward(cudaStreamCaptureModeGlobal);
    }
  }

  std::tuple<Tensor, Tensor, Tensor> run(const Tensor& x_in, const Tensor& router_w,
                                         const Tensor& w_in, const Tensor& w_out,
                                         const OptTensor& w_sh_in, const OptTensor& w_sh_out);
  Grads backward(const Tensor& grad_out, const Tensor& grad_aux) {
    const c10::cuda::CUDAGuard on(p_.x.device());
    if (grad_out.defined())
      grad_out_.copy_(grad_out, true);
    else
      grad_out_.zero_();
    if (grad_aux.defined())
      grad_aux_.copy_(grad_aux.reshape({1}), true);
    else if (opt_.full_softmax)
      grad_aux_.zero_();
    size_t i = 0;
    while (i < bwd_.size() && held(bwd_[i]->grads)) ++i;
    if (i == bwd_.size()) {
      const c10::cuda::CUDAStreamGuard work(
          c10::cuda::getStreamFromPool(false, p_.x.get_device()));
      capture_backward(cudaStreamCaptureModeThreadLocal);   // (other threads may be at work by now)
    }
    bwd_[i]->graph.replay();
    n_launched += n_bwd_;
    Grads g = bwd_[i]->grads;
    for (Tensor* t : all(g))
      if (t->defined()) *t = i < SETS_GIVEN_OUT ? t->detach() : t->clone();
    return g;
  }

 private:
  // A capture of the backward and the gradients it leaves.
  struct BackwardGraph {
    at::cuda::CUDAGraph graph;
    Grads grads;
  };
  static constexpr size_t SETS_GIVEN_OUT = 2;

  static std::array<Tensor*, 6> all(Grads& g) {
    return {&g.dx, &g.d_router, &g.dw_in, &g.dw_out, &g.dw_sh_in, &g.dw_sh_out};
  }
  // Whether anybody else refers to these buffers.
  static bool held(Grads& g) {
    for (const Tensor* t : all(g))
      if (t->defined() && t->storage().use_count() > 1) return true;
    return false;
  }
  // On the current stream. The gradients are allocated ahead of the capture: its pool is scratch that
  // the other graphs use as well, one after the other.
  void capture_backward(cudaStreamCaptureMode mode) {
    auto b = std::make_unique<BackwardGraph>();
    b->grads = empty_grads(p_);
    const int64_t l0 = n_launched;
    b->graph.capture_begin(fwd_.pool(), mode);
    launch_backward(p_, opt_, r_.kept, grad_out_, grad_aux_, b->grads);
    b->graph.capture_end();
    n_bwd_ = n_launched - l0;
    n_launched -= n_bwd_;   // (a capture launches nothing)
    bwd_.push_back(std::move(b));
  }

  Options opt_;
  Operands p_;
  Results r_;
  Tensor grad_out_, grad_aux_;
  at::cuda::CUDAGraph fwd_;
  std::vector<std::unique_ptr<BackwardGraph>> bwd_;
  int64_t n_fwd_ = 0, n_bwd_ = 0;
};

// Edges: x, router_w, w_in, w_out, w_sh_in, w_sh_out.
struct MoEGraphedBackward : public torch::autograd::Node {
  std::shared_ptr<GraphedBlock> graphs;
  std::string name() const override { return "MoEGraphedBackward"; }
  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    if (!grads[0].defined() && !grads[1].defined()) return variable_list(6);
    Grads g;
    {
      at::NoGradGuard no_grad;
      g = graphs->backward(grads[0], grads[1]);
    }
    return once({g.dx, g.d_router, g.dw_in, g.dw_out, g.dw_sh_in, g.dw_sh_out});
  }
};

std::tuple<Tensor, Tensor, Tensor> GraphedBlock::run(const Tensor& x_in, const Tensor& router_w,
                                                     const Tensor& w_in, const Tensor& w_out,
                                                     const OptTensor& w_sh_in,
                                                     const OptTensor& w_sh_out) {
  TORCH_CHECK(x_in.sizes() == p_.x.sizes() && x_in.scalar_type() == p_.x.scalar_type() &&
                  x_in.device() == p_.x.device(),
              "the graphs were captured for another input shape");
  const Tensor si = w_sh_in.value_or(Tensor()), so = w_sh_out.value_or(Tensor());
  refuse_forward_mode(x_in, router_w, w_in, w_out, si, so);
  std::shared_ptr<MoEGraphedBackward> node;
  if (any_grad(x_in, router_w, w_in, w_out, si, so)) {
    node = new_node<MoEGraphedBackward>();
    node->set_next_edges(
        torch::autograd::collect_next_edges(x_in, router_w, w_in, w_out, si, so));
    node->graphs = shared_from_this();
  }
  Tensor out, aux, counts;
  {
    at::NoGradGuard no_grad;
    const c10::cuda::CUDAGuard on(p_.x.device());
    p_.x.copy_(x_in, true);
    fwd_.replay();
    n_launched += n_fwd_;
    out = r_.out.detach();
    aux = r_.aux.detach();
    counts = r_.counts.clone();   // (kept by callers for their logs)
  }
  if (node) {
    torch::autograd::set_history(out, node);
    if (opt_.full_softmax)
      torch::autograd::set_history(aux, node);
    else
      node->add_input_metadata(torch::autograd::Node::undefined_input());
  }
  return {out, aux, counts};
}

// ----------------------------------------------------------------------------------- Muon
// One optimizer step over CUDA matrices or stacks of them, all of one device and of shapes
// moe_b200_muon_supported takes. Returns fp32 [2]: |dW|^2 and |W|^2 over all of them.
Tensor muon_step(const std::vector<Tensor>& params, const std::vector<Tensor>& grads,
                 const std::vector<Tensor>& bufs, double lr, double momentum, double weight_decay,
                 int64_t steps, double a, double b, double c, double eps) {
  TORCH_CHECK(!params.empty() && params.size() == grads.size() && params.size() == bufs.size(),
              "one gradient and one momentum buffer per parameter");
  at::NoGradGuard no_grad;
  const Tensor& first = params[0];
  const c10::cuda::CUDAGuard on(first.device());
  std::vector<moe_b200_muon_param> ps(params.size());
  for (size_t i = 0; i < params.size(); ++i) {
    const Tensor &p = params[i], &g = grads[i], &m = bufs[i];
    TORCH_CHECK(p.device() == first.device() && g.device() == p.device() &&
                    m.device() == p.device() && (p.dim() == 2 || p.dim() == 3) &&
                    g.sizes() == p.sizes() && m.sizes() == p.sizes() && p.is_contiguous() &&
                    g.is_contiguous() && m.is_contiguous() &&
                    (p.scalar_type() == at::kBFloat16 || p.scalar_type() == at::kFloat) &&
                    g.scalar_type() == at::kBFloat16 && m.scalar_type() == at::kBFloat16,
                "parameter ", i, ": contiguous bf16 gradient and momentum beside it expected");
    const int64_t rows = p.size(-2), cols = p.size(-1);
    ps[i] = {p.mutable_data_ptr(),
             g.const_data_ptr(),
             m.mutable_data_ptr(),
             p.scalar_type() == at::kFloat,
             int32_t(p.dim() == 3 ? p.size(0) : 1),
             int32_t(rows),
             int32_t(cols),
             float(-lr * std::sqrt(std::max(1.0, double(rows) / double(cols))))};
  }
  const int32_t n = int32_t(ps.size());
  const Tensor norms = at::empty({3}, first.options().dtype(at::kFloat));
  const Tensor scratch = bytes_like(first, abi.muon_scratch_bytes(ps.data(), n));
  int32_t launched = 0;
  check(abi.muon_step(ps.data(), n, float(1.0 - momentum), float(momentum),
                      float(1.0 - lr * weight_decay), int32_t(steps), float(a), float(b), float(c),
                      float(eps), norms.mutable_data_ptr<float>(), scratch.mutable_data_ptr(),
                      size_t(scratch.numel()), &launched, status_word(first.get_device()),
                      c10::cuda::getCurrentCUDAStream().stream()),
        "moe_b200_muon_step");
  for (const auto* v : {&params, &bufs})
    for (const Tensor& t : *v) t.unsafeGetTensorImpl()->bump_version();
  n_launched += launched;
  return norms.narrow(0, 0, 2);
}

}  // namespace

PYBIND11_MODULE(_moe_shim, m) {
  m.def("bind", &bind);
  m.def("launches", [] { return n_launched.load(); });
  m.def("block", &block);
  m.def("sublayer", &sublayer);
  m.def("muon_step", &muon_step);
  py::class_<GraphedBlock, std::shared_ptr<GraphedBlock>>(m, "GraphedBlock")
      .def(py::init<const Tensor&, const Tensor&, const OptTensor&, const Tensor&, const Tensor&,
                    const OptTensor&, const OptTensor&, int64_t, bool, bool, double, int64_t, bool,
                    int64_t>())
      .def("run", &GraphedBlock::run);
}
