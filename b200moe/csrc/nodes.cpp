// Autograd nodes of the training step in C++: embedding, norm, the attention half of a block, the routed layer on one rank, and
// the LM head with its loss.  They do what the nodes of the same name in b200moe/ops do from Python, with the same kernels in
// the same order: what they save is the host's time, 20-30 us per launch and 30 per node of the backward pass (from Python's
// second thread), which is what a small layer costs.  A step of two blocks of width 512 took 4.7 ms for 1.5 ms of kernels.
//
// The functions at the end answer None where an operand is not what the node takes (type, layout, alignment, device); the
// caller then goes the general way.  Kernels come from the library that b200moe.ops.native has loaded (``bind``).
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <torch/csrc/autograd/graph_task.h>
#include <torch/extension.h>

#include <atomic>

#include "entries.h"

using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::variable_list;
using Tensor = at::Tensor;
using Optional = std::optional<Tensor>;

namespace {

std::atomic<long long> launches{0};

struct Library {
  decltype(&b2_layers_refused) layers_refused;
  decltype(&b2_attn_half_fwd) attn_half_fwd;
  decltype(&b2_attn_half_bwd) attn_half_bwd;
  decltype(&b2_moe_layer_fwd) moe_layer_fwd;
  decltype(&b2_moe_experts_bwd) moe_experts_bwd;
  decltype(&b2_moe_router_bwd) moe_router_bwd;
  decltype(&b2_moe_aux) moe_aux;
  decltype(&b2_rmsnorm_fwd) rmsnorm_fwd;
  decltype(&b2_rmsnorm_bwd) rmsnorm_bwd;
  decltype(&b2_rmsnorm_bwd_parts) rmsnorm_bwd_parts;
  decltype(&b2_swiglu_bwd_in_product) swiglu_bwd_in_product;
  decltype(&b2_head_chunk) head_chunk;
  decltype(&b2_scale_bf16) scale_bf16;
  decltype(&b2_embedding_fwd) embedding_fwd;
  decltype(&b2_embedding_bwd) embedding_bwd;
} lib;

void bind(const std::string& path) {
  void* const handle = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
  TORCH_CHECK(handle, "cannot load ", path, ": ", dlerror());
  auto resolve = [&](auto& entry, const char* name) {
    void* const symbol = dlsym(handle, name);
    TORCH_CHECK(symbol, path, " has no ", name);
    entry = reinterpret_cast<std::remove_reference_t<decltype(entry)>>(symbol);
  };
  resolve(lib.layers_refused, "b2_layers_refused");
  resolve(lib.attn_half_fwd, "b2_attn_half_fwd");
  resolve(lib.attn_half_bwd, "b2_attn_half_bwd");
  resolve(lib.moe_layer_fwd, "b2_moe_layer_fwd");
  resolve(lib.moe_experts_bwd, "b2_moe_experts_bwd");
  resolve(lib.moe_router_bwd, "b2_moe_router_bwd");
  resolve(lib.moe_aux, "b2_moe_aux");
  resolve(lib.rmsnorm_fwd, "b2_rmsnorm_fwd");
  resolve(lib.rmsnorm_bwd, "b2_rmsnorm_bwd");
  resolve(lib.rmsnorm_bwd_parts, "b2_rmsnorm_bwd_parts");
  resolve(lib.swiglu_bwd_in_product, "b2_swiglu_bwd_in_product");
  resolve(lib.head_chunk, "b2_head_chunk");
  resolve(lib.scale_bf16, "b2_scale_bf16");
  resolve(lib.embedding_fwd, "b2_embedding_fwd");
  resolve(lib.embedding_bwd, "b2_embedding_bwd");
}

cudaStream_t stream() { return c10::cuda::getCurrentCUDAStream().stream(); }
// Raises what b200moe.ops.native raises for a refused launch; ``name``: its entry point, null for a sequence of layers.cu.
void check(int code, const char* name, int count) {
  if (code != 0) {
    if (!name) name = lib.layers_refused();
    std::string detail;
    try {
      pybind11::gil_scoped_acquire gil;
      detail = pybind11::module_::import("b200moe.ops.native").attr("_failure_detail")(name, code).cast<std::string>();
    } catch (pybind11::error_already_set&) {      // the code alone, then
    }
    TORCH_CHECK(false, name, " failed with code ", code, detail);
  }
  launches += count;
}
// Addresses as the entry points type them; the tensors' types have been looked at by then.
struct Const {
  const void* at;
  template <typename T> operator const T*() const { return static_cast<const T*>(at); }
};
struct Mutable {
  void* at;
  template <typename T> operator T*() const { return static_cast<T*>(at); }
};
Const ptr(const Tensor& t) { return {t.defined() ? t.const_data_ptr() : nullptr}; }
Mutable mut(const Tensor& t) { return {t.defined() ? t.data_ptr() : nullptr}; }
Tensor fp32(at::IntArrayRef sizes, const Tensor& like) { return at::empty(sizes, like.options().dtype(at::kFloat)); }
Tensor bf16(at::IntArrayRef sizes, const Tensor& like) { return at::empty(sizes, like.options().dtype(at::kBFloat16)); }
Tensor int32(at::IntArrayRef sizes, const Tensor& like) { return at::empty(sizes, like.options().dtype(at::kInt)); }

bool aligned(const Tensor& t) { return reinterpret_cast<uintptr_t>(t.const_data_ptr()) % 16 == 0; }
bool plain(const Tensor& t, at::ScalarType type, const Tensor& beside) {
  return t.scalar_type() == type && t.is_contiguous() && t.device() == beside.device() && aligned(t);
}
// A bf16 weight and the buffer that its gradient is added to.
bool trained(const Tensor& weight, const Tensor& grad, const Tensor& beside) {
  return plain(weight, at::kBFloat16, beside) && plain(grad, at::kFloat, beside) && grad.sizes() == weight.sizes();
}
bool follows(std::initializer_list<Tensor> inputs) {
  if (!at::GradMode::is_enabled()) return false;
  for (const Tensor& t : inputs)
    if (t.defined() && t.requires_grad()) return true;
  return false;
}
// Scratch of one call, ``bytes`` per buffer (0: null).  Small calls take it as one allocation (1.3 us each); large ones buffer by
// buffer, as blocks that the allocator has use for elsewhere.
class Scratch {
 public:
  static constexpr int64_t TOGETHER = 16 << 20;
  Scratch(const Tensor& like, std::initializer_list<int64_t> bytes) {
    int64_t total = 0;
    for (int64_t b : bytes) total += (b + 255) / 256 * 256;
    const bool together = total <= TOGETHER;
    const auto options = like.options().dtype(at::kByte);
    if (together) held_.push_back(at::empty({total}, options));
    char* next = together ? static_cast<char*>(held_[0].data_ptr()) : nullptr;
    for (int64_t b : bytes) {
      if (together) {
        at_.push_back(b ? next : nullptr);
        next += (b + 255) / 256 * 256;
      } else {
        held_.push_back(b ? at::empty({b}, options) : Tensor());
        at_.push_back(mut(held_.back()).at);
      }
    }
  }
  Mutable operator[](size_t i) const { return {at_[i]}; }

 private:
  std::vector<Tensor> held_;
  std::vector<void*> at_;
};

// Where the gradient of a weight goes in a backward pass: the buffer that the weight carries then (its ``main_grad``; as in the
// Python nodes, one that took the place of the forward pass's is followed).  A buffer that the kernels do not take, or none,
// gets the sum afterwards.
class Gradient {
 public:
  Gradient(const Tensor& weight, const Tensor& buffer, at::ScalarType kind) : weight_(weight), buffer_(buffer) {
    const bool direct = buffer_.defined() && plain(buffer_, kind, weight) && buffer_.sizes() == weight.sizes();
    sum_ = direct ? buffer_ : at::zeros(weight.sizes(), weight.options().dtype(kind).requires_grad(false));
  }
  Mutable operator*() const { return {sum_.data_ptr()}; }
  // What autograd is told: nothing where there is a buffer.
  Tensor given() {
    if (buffer_.is_same(sum_)) return Tensor();
    if (buffer_.defined()) {
      buffer_.add_(sum_);
      return Tensor();
    }
    return weight_.requires_grad() ? sum_.to(weight_.scalar_type()) : Tensor();
  }
  // The buffers that ``count`` weights carry.
  static std::vector<Tensor> of(const std::vector<Tensor>& weights, size_t count) {
    std::vector<Tensor> buffers(count);
    pybind11::gil_scoped_acquire gil;
    static PyObject* const name = PyUnicode_InternFromString("main_grad");
    for (size_t i = 0; i < count; ++i) {
      const auto object = pybind11::reinterpret_steal<pybind11::object>(THPVariable_Wrap(weights[i]));
      const auto buffer = pybind11::reinterpret_steal<pybind11::object>(PyObject_GetAttr(object.ptr(), name));
      if (!buffer) PyErr_Clear();
      else if (THPVariable_Check(buffer.ptr())) buffers[i] = THPVariable_Unpack(buffer.ptr());
    }
    return buffers;
  }

 private:
  Tensor weight_, buffer_, sum_;
};

// What a node keeps beside the saved tensors: weights, as the Python nodes keep them.
void keep(AutogradContext* ctx, std::vector<Tensor> tensors) { ctx->saved_data["kept"] = std::move(tensors); }
std::vector<Tensor> kept(AutogradContext* ctx) { return ctx->saved_data["kept"].toTensorVector(); }

struct Embedding : public Function<Embedding> {
  static Tensor forward(AutogradContext* ctx, const Tensor& ids, const Tensor& table) {
    ctx->save_for_backward({ids});
    keep(ctx, {table});
    std::vector<int64_t> sizes = ids.sizes().vec();
    sizes.push_back(table.size(1));
    Tensor out = bf16(sizes, table);
    check(lib.embedding_fwd(ptr(ids), ptr(table), mut(out), ids.numel(), table.size(1), stream()), "b2_embedding_fwd", 1);
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const Tensor ids = ctx->get_saved_variables()[0], dy = grads[0].contiguous();
    const std::vector<Tensor> w = kept(ctx);
    TORCH_CHECK(dy.scalar_type() == at::kBFloat16, "expected bfloat16, got ", dy.scalar_type());
    Gradient grad(w[0], Gradient::of(w, 1)[0], at::kFloat);
    check(lib.embedding_bwd(ptr(ids), ptr(dy), *grad, ids.numel(), w[0].size(1), stream()), "b2_embedding_bwd", 1);
    return {Tensor(), grad.given()};
  }
};

struct RMSNorm : public Function<RMSNorm> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight, double eps, const Tensor& status) {
    const int D = x.size(-1), rows = x.numel() / D;
    Tensor y = at::empty_like(x), rstd = fp32({rows}, x);
    check(lib.rmsnorm_fwd(ptr(x), nullptr, ptr(weight), nullptr, mut(y), mut(rstd), rows, D, eps, mut(status), stream()),
          "b2_rmsnorm_fwd", 1);
    ctx->save_for_backward({x, weight, rstd});
    keep(ctx, {status});
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &weight = saved[1], &rstd = saved[2];
    const Tensor dy = grads[0].contiguous(), status = kept(ctx)[0];
    const int D = x.size(-1), rows = x.numel() / D;
    TORCH_CHECK(dy.scalar_type() == at::kBFloat16, "expected bfloat16, got ", dy.scalar_type());
    Tensor dx = at::empty_like(x), dw = fp32({D}, x), partial = fp32({lib.rmsnorm_bwd_parts(rows, D), D}, x);
    check(lib.rmsnorm_bwd(ptr(dy), ptr(x), ptr(weight), ptr(rstd), nullptr, mut(dx), mut(partial), mut(dw), rows, D, mut(status),
                          stream()), "b2_rmsnorm_bwd", 2);
    return {dx, dw, Tensor(), Tensor()};
  }
};

struct AttnHalf : public Function<AttnHalf> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& ln1, const Tensor& wqkv,
                               const Tensor& cos, const Tensor& sin, const Tensor& wo, const Tensor& ln2, const Tensor& status,
                               int64_t hq, int64_t hkv, double eps1, double eps2) {
    const int B = x.size(0), S = x.size(1);
    const int64_t T = x.size(0) * x.size(1);
    Tensor n1 = at::empty_like(x), a = at::empty_like(x), proj = at::empty_like(x), sum = at::empty_like(x), n2 = at::empty_like(x);
    Tensor qkv = bf16({T, 128 * (hq + 2 * hkv)}, x), stats = fp32({T * (2 + hq)}, x);
    check(lib.attn_half_fwd(ptr(x), ptr(ln1), ptr(wqkv), ptr(cos), ptr(sin), ptr(wo), ptr(ln2), mut(n1), mut(qkv), mut(a),
                            mut(proj), mut(sum), mut(n2), mut(stats), B, S, hq, hkv, eps1, eps2, mut(status), stream()),
          nullptr, 5);
    ctx->save_for_backward({x, ln1, ln2, cos, sin, n1, qkv, a, sum, stats});
    keep(ctx, {wqkv, wo, status});
    ctx->saved_data["heads"] = hq * 4096 + hkv;
    return {sum, n2};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &ln1 = saved[1], &ln2 = saved[2], &cos = saved[3], &sin = saved[4], &n1 = saved[5],
                 &qkv = saved[6], &a = saved[7], &sum = saved[8], &stats = saved[9];
    const std::vector<Tensor> w = kept(ctx);
    const int64_t heads = ctx->saved_data["heads"].toInt(), hq = heads / 4096, hkv = heads % 4096;
    const int B = x.size(0), S = x.size(1), D = x.size(2);
    const int64_t T = x.size(0) * x.size(1);
    const Tensor dsum = grads[0].contiguous(), dn2 = grads[1].contiguous();
    TORCH_CHECK(dsum.scalar_type() == at::kBFloat16 && dn2.scalar_type() == at::kBFloat16, "expected bfloat16 gradients");
    // The gradient of the first norm's output takes the place of the attention output's, which is used up by then, and dx that
    // of the sum's, which the first norm's kernel adds row by row before it stores the row: as much as the separate nodes hold.
    Tensor dx = at::empty_like(x), dln1 = fp32({D}, x), dln2 = fp32({D}, x);
    // da, dqkv, the norms' partial sums, the attention's row statistics
    const Scratch tmp(x, {2 * T * D, 2 * qkv.numel(), int64_t{4} * lib.rmsnorm_bwd_parts(T, D) * D, 8 * T * hq});
    const std::vector<Tensor> buffers = Gradient::of(w, 2);
    Gradient gqkv(w[0], buffers[0], at::kFloat), go(w[1], buffers[1], at::kFloat);
    check(lib.attn_half_bwd(ptr(dsum), ptr(dn2), ptr(x), ptr(ln1), ptr(w[0]), ptr(cos), ptr(sin), ptr(w[1]), ptr(ln2), ptr(n1),
                            ptr(qkv), ptr(a), ptr(sum), ptr(stats), *gqkv, *go, mut(dln1), mut(dln2), mut(dx), mut(dx), tmp[0],
                            tmp[0], tmp[1], tmp[2], tmp[3], B, S, hq, hkv, mut(w[2]), stream()),
          nullptr, 11);
    const Tensor none;
    return {dx, dln1, gqkv.given(), none, none, go.given(), dln2, none, none, none, none, none};
  }
};

struct MoELayer : public Function<MoELayer> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& router, const Tensor& w1, const Tensor& w3,
                               const Tensor& w2, const Optional& residual, const Tensor& status, int64_t cap, bool keeps,
                               bool balance) {
    ctx->set_materialize_grads(false);
    const int64_t D = x.size(-1), T = x.numel() / D, E = w1.size(0), F = w1.size(1);
    Tensor weights = fp32({T, 2}, x), probs = fp32({T, E}, x), idx = at::empty({T, 2}, x.options().dtype(at::kLong));
    Tensor tables = int32({2 * T + cap + 2 * E + cap / 128 + 4}, x);
    Tensor x_perm = bf16({cap, D}, x), y_perm = bf16({cap, D}, x), h = bf16({cap, F}, x), out = at::empty_like(x), gate, up;
    if (keeps) gate = at::empty_like(h), up = at::empty_like(h);
    check(lib.moe_layer_fwd(ptr(x), ptr(router), ptr(w1), ptr(w3), ptr(w2), ptr(residual ? *residual : Tensor()), mut(weights),
                            mut(idx), mut(probs), mut(tables), mut(x_perm), mut(h), mut(gate), mut(up), mut(y_perm), mut(out), T, D,
                            F, E, cap, mut(status), stream()), nullptr, 6);
    variable_list saved = {x, weights, idx, probs, tables, x_perm, y_perm};
    if (keeps) saved.insert(saved.end(), {gate, up});
    ctx->save_for_backward(std::move(saved));
    keep(ctx, {router, w1, w3, w2, status});
    ctx->saved_data["residual"] = residual.has_value();
    if (!balance) return {out};
    Tensor aux = fp32({}, x);
    check(lib.moe_aux(ptr(probs), tables.const_data_ptr<int>() + tables.numel() - E, mut(aux), T, E, stream()), "b2_moe_aux", 1);
    return {out, aux};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &weights = saved[1], &idx = saved[2], &probs = saved[3], &tables = saved[4], &x_perm = saved[5],
                 &y_perm = saved[6];
    const std::vector<Tensor> w = kept(ctx);
    const int64_t D = x.size(-1), T = x.numel() / D, E = w[1].size(0), F = w[1].size(1), cap = x_perm.size(0);
    const bool rebuild = saved.size() < 9;
    const Tensor dout = grads[0].defined() ? grads[0].contiguous() : at::zeros_like(x);
    TORCH_CHECK(dout.scalar_type() == at::kBFloat16, "expected bfloat16, got ", dout.scalar_type());
    Tensor daux = grads.size() > 1 && grads[1].defined() ? grads[1].to(x.device(), at::kFloat) : Tensor();
    const int64_t row = 2 * cap * D, wide = 2 * cap * F;
    const bool own = !lib.swiglu_bwd_in_product(cap, F, D);      // the SwiGLU backward is a kernel of its own
    const std::vector<Tensor> buffers = Gradient::of(w, 4);
    const at::ScalarType kind = buffers[1].defined() && buffers[1].scalar_type() == at::kBFloat16 ? at::kBFloat16 : at::kFloat;
    Gradient grouter(w[0], buffers[0], at::kFloat), g1(w[1], buffers[1], kind), g3(w[2], buffers[2], kind), g2(w[3], buffers[3], kind);
    // dx_perm takes the place of what is used up by then: dh, and gate and up where they are formed again.  dweights, dlogits.
    // Behind them dy_perm, dgu and h, which large calls hold no longer than the experts need them.
    const int64_t used_bytes = std::max(row, (own + 2 * rebuild) * wide);
    const int64_t few = used_bytes + row + 3 * wide <= Scratch::TOGETHER;
    const Scratch tmp(x, {used_bytes, 8 * T, 4 * T * E, few * row, few * 2 * wide, few * wide});
    char* const used = tmp[0];
    char* const formed = used + own * wide;
    {
      std::optional<Scratch> large;
      if (!few) large.emplace(x, std::initializer_list<int64_t>{row, 2 * wide, wide});
      const auto inner = [&](size_t i) { return few ? tmp[3 + i] : (*large)[i]; };
      check(lib.moe_experts_bwd(ptr(dout), ptr(w[1]), ptr(w[2]), ptr(w[3]), ptr(weights), mut(tables), ptr(x_perm), ptr(y_perm),
                                rebuild ? formed : mut(saved[7]).at, rebuild ? formed + wide : mut(saved[8]).at, rebuild, *g1, *g3,
                                *g2, kind == at::kFloat ? 1 : 2, inner(0), inner(1), inner(2), own ? used : nullptr, used, tmp[1],
                                T, D, F, E, cap, mut(w[4]), stream()), nullptr, 5 + own + rebuild);
    }
    Tensor dx = at::empty_like(x);
    check(lib.moe_router_bwd(ptr(x), ptr(w[0]), ptr(weights), ptr(idx), ptr(probs), mut(tables), ptr(daux), *grouter, used, tmp[1],
                             tmp[2], mut(dx), T, D, E, cap, stream()), nullptr, 2);
    const Tensor none;
    return {dx, grouter.given(), g1.given(), g3.given(), g2.given(), ctx->saved_data["residual"].toBool() ? grads[0] : none,
            none, none, none, none};
  }
};

// The head where the factor that will be back-propagated into the loss is known: b200moe/ops/loss.py.
struct Head : public Function<Head> {
  static Tensor forward(AutogradContext* ctx, const Tensor& hidden, const Tensor& weight, const Tensor& targets, const Tensor& grad,
                        double scale, int64_t chunk, const Tensor& status) {
    const int64_t V = weight.size(0), D = weight.size(1), T = hidden.numel() / D;
    Tensor loss = at::zeros({}, hidden.options().dtype(at::kDouble)), dh = at::empty_like(hidden);
    for (int64_t lo = 0; lo < T; lo += chunk) {
      const int64_t n = std::min(chunk, T - lo);
      Tensor logits = bf16({n, V}, hidden);
      check(lib.head_chunk(static_cast<const char*>(ptr(hidden).at) + 2 * lo * D, ptr(weight),
                           static_cast<const long long*>(ptr(targets)) + lo, mut(logits), mut(loss),
                           static_cast<char*>(mut(dh).at) + 2 * lo * D, mut(grad), n, V, D, 1.0 / T, scale / T, mut(status),
                           stream()),
            nullptr, 4);
    }
    ctx->save_for_backward({dh});
    ctx->saved_data["scale"] = scale;
    return loss.to(at::kFloat);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    Tensor dh = ctx->get_saved_variables()[0];
    if (torch::autograd::get_current_graph_task_keep_graph()) dh = dh.clone();
    const Tensor factor = (grads[0] / ctx->saved_data["scale"].toDouble()).to(dh.device(), at::kFloat);
    check(lib.scale_bf16(mut(dh), ptr(factor), dh.numel(), stream()), "b2_scale_bf16", 1);
    const Tensor none;
    return {dh, none, none, none, none, none, none};
  }
};

// ------------------------------------------------------------------ entry points
Optional embedding(const Tensor& ids, const Tensor& table, const Tensor& grad) {
  if (!(ids.scalar_type() == at::kLong && ids.is_contiguous() && ids.numel() > 0 && ids.numel() < INT_MAX && table.dim() == 2 &&
        table.size(1) % 8 == 0 && table.is_cuda() && ids.device() == table.device() && trained(table, grad, table)))
    return std::nullopt;
  return Embedding::apply(ids, table);
}

Optional rmsnorm(const Tensor& x, const Tensor& weight, double eps, const Tensor& status) {
  if (!(x.is_cuda() && x.dim() > 0 && x.numel() > 0 && plain(x, at::kBFloat16, x) && weight.dim() == 1 &&
        weight.size(0) == x.size(-1) && plain(weight, at::kFloat, x) && x.size(-1) % 8 == 0 && x.size(-1) <= 8192 &&
        x.numel() / x.size(-1) < INT_MAX))
    return std::nullopt;
  return RMSNorm::apply(x, weight, eps, status);
}

std::optional<variable_list> attn_half(const Tensor& x, const Tensor& ln1, const Tensor& wqkv, const Tensor& gqkv, const Tensor& cos,
                                       const Tensor& sin, const Tensor& wo, const Tensor& go, const Tensor& ln2,
                                       const Tensor& status, int64_t hq, int64_t hkv, double eps1, double eps2) {
  if (!(x.is_cuda() && x.dim() == 3 && x.numel() > 0 && plain(x, at::kBFloat16, x))) return std::nullopt;
  const int64_t S = x.size(1), D = x.size(2);
  if (!(S % 128 == 0 && D == 128 * hq && D <= 8192 && hkv > 0 && hq % hkv == 0 && x.size(0) * S * (hq + 2 * hkv) < INT_MAX / 128 &&
        wqkv.dim() == 2 && wqkv.size(0) == 128 * (hq + 2 * hkv) && wqkv.size(1) == D && trained(wqkv, gqkv, x) && wo.dim() == 2 &&
        wo.size(0) == D && wo.size(1) == D && trained(wo, go, x)))
    return std::nullopt;
  for (const Tensor& gain : {ln1, ln2})
    if (!(gain.dim() == 1 && gain.size(0) == D && plain(gain, at::kFloat, x))) return std::nullopt;
  for (const Tensor& table : {cos, sin})
    if (!(table.dim() == 2 && table.size(1) == 64 && table.size(0) >= S && plain(table, at::kFloat, x))) return std::nullopt;
  return AttnHalf::apply(x, ln1, wqkv, cos, sin, wo, ln2, status, hq, hkv, eps1, eps2);
}

std::optional<variable_list> moe_layer(const Tensor& x, const Tensor& router, const Tensor& w1, const Tensor& w3, const Tensor& w2,
                                       const Optional& residual, const Tensor& grouter, const Tensor& g1, const Tensor& g3,
                                       const Tensor& g2, const Tensor& status, int64_t align, bool recompute, bool balance) {
  if (!(x.is_cuda() && x.dim() >= 2 && x.numel() > 0 && plain(x, at::kBFloat16, x) && router.dim() == 2 && w1.dim() == 3))
    return std::nullopt;
  const int64_t E = w1.size(0), F = w1.size(1), D = x.size(-1), T = x.numel() / D;
  if (!(E >= 2 && E <= 16 && D % 64 == 0 && F % 128 == 0 && router.size(0) == E && router.size(1) == D && w1.size(2) == D &&
        w3.sizes() == w1.sizes() && w2.dim() == 3 && w2.size(0) == E && w2.size(1) == D && w2.size(2) == F &&
        E * D * 2 <= 200 * 1024 && T < (1 << 28) && trained(router, grouter, x)))
    return std::nullopt;
  const at::ScalarType kind = g1.scalar_type();
  if (kind != at::kFloat && kind != at::kBFloat16) return std::nullopt;
  const std::pair<const Tensor&, const Tensor&> experts[] = {{w1, g1}, {w3, g3}, {w2, g2}};
  for (const auto& [weight, grad] : experts)
    if (!(plain(weight, at::kBFloat16, x) && plain(grad, kind, x) && grad.sizes() == weight.sizes())) return std::nullopt;
  if (residual && !(plain(*residual, at::kBFloat16, x) && residual->sizes() == x.sizes())) return std::nullopt;
  const bool keeps = !recompute && follows({x, router, w1, w3, w2, residual ? *residual : Tensor()});
  const int64_t cap = (2 * T + E * (align - 1) + align - 1) / align * align;      // moe_fused.capacity_rows
  return MoELayer::apply(x, router, w1, w3, w2, residual, status, cap, keeps, balance);
}

Optional head(const Tensor& hidden, const Tensor& weight, const Tensor& targets, const Tensor& grad, double scale, int64_t chunk,
              const Tensor& status) {
  if (!(hidden.is_cuda() && hidden.dim() > 0 && hidden.numel() > 0 && plain(hidden, at::kBFloat16, hidden) && weight.dim() == 2 &&
        hidden.size(-1) == weight.size(1) && weight.size(1) % 64 == 0 && weight.size(0) % 64 == 0 && weight.size(0) > 16 &&
        weight.size(0) <= 32768 && trained(weight, grad, hidden) && targets.scalar_type() == at::kLong && targets.is_contiguous() &&
        targets.device() == hidden.device() && targets.numel() == hidden.numel() / weight.size(1) && scale != 0.0))
    return std::nullopt;
  if (!(at::GradMode::is_enabled() && hidden.requires_grad())) return std::nullopt;
  return Head::apply(hidden, weight, targets, grad, scale, chunk, status);
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  using Release = pybind11::call_guard<pybind11::gil_scoped_release>;
  m.def("bind", &bind);
  m.def("check", &check, Release());
  m.def("launches", [] { return launches.load(); });
  m.def("embedding", &embedding, Release());
  m.def("rmsnorm", &rmsnorm, Release());
  m.def("attn_half", &attn_half, Release());
  m.def("moe_layer", &moe_layer, Release());
  m.def("head", &head, Release());
}
