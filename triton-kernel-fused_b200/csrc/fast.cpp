// Autograd functions of the layer, of the experts on given picks and of the conv router as compiled code: the host side of the
// Python Functions of the same name (layer.py, moe.py, router.py) for plain calls.  Each function returns None for a call
// that is not plain (a tensor that would have to be cast or made contiguous, autocast, functorch transforms, forward-mode
// gradients, dispatch modes, tensor subclasses, a shape that is an error), and the caller then takes the Python Function, which
// casts, refuses or raises as it always did.
//
// Why: between two small passes the host was the bound.  A Python Function costs the caller 8 us to enter, its allocations and
// argument checks 15 to 30 more each way, and in the backward the autograd engine's thread waits for the interpreter lock before
// it can call it.  us a pass, Python / compiled: one token through 64 experts of 2048 x 1408 62 / 39; forward and backward of 512 tokens
// at width 256 237 / 148; conv router of 16 384 tokens 145 / 118.
//
// Nothing is kept between calls but what autograd saves (saved-tensor hooks see it); the workspace of a forward is a saved tensor.
#include <ATen/autocast_mode.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/extension.h>
#include <torch/version.h>

#include "../../include/b200moe.h"

namespace {

using at::Tensor;
using std::optional;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

void check(int rc) {
  if (rc == 0) return;
  const std::string msg = "b200moe error " + std::to_string(rc) + ": " + b200moe_last_error_string();
  if (rc == B200MOE_E_CUDA) TORCH_CHECK(false, msg);
  TORCH_CHECK_VALUE(false, msg);
}

// a contiguous CUDA tensor of its own memory that nothing wraps
bool plain(const Tensor& t, at::ScalarType type, c10::Device dev) {
  if (!t.defined() || t.scalar_type() != type || t.device() != dev || t.layout() != at::kStrided) return false;
  const auto ks = t.key_set();
  if (ks.has(c10::DispatchKey::Python) || ks.has(c10::DispatchKey::FuncTorchBatched) ||
      ks.has(c10::DispatchKey::FuncTorchGradWrapper) || ks.has(c10::DispatchKey::Functionalize))
    return false;
  return t.is_contiguous() && !t._fw_grad(0).defined();
}
bool plain_or_none(const optional<Tensor>& t, at::ScalarType type, c10::Device dev) { return !t.has_value() || plain(*t, type, dev); }

// no mode or transform that has to see the operations of this call
bool plain_call(const Tensor& x) {
  const auto tls = c10::impl::tls_local_dispatch_key_set();
  return x.is_cuda() && !tls.included_.has(c10::DispatchKey::FuncTorchDynamicLayerFrontMode) &&
         !c10::impl::TorchDispatchModeTLS::any_modes_set() && !at::autocast::is_autocast_enabled(at::kCUDA);
}

void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
void* ptr(const optional<Tensor>& t) { return t.has_value() ? t->data_ptr() : nullptr; }
b200moe_stream_t stream_of(const Tensor& t) { return reinterpret_cast<b200moe_stream_t>(c10::cuda::getCurrentCUDAStream(t.device().index()).stream()); }
Tensor bytes(size_t n, const Tensor& like) { return at::empty({static_cast<int64_t>(n)}, like.options().dtype(at::kByte)); }
Tensor grad_like(bool want, const Tensor& t) { return want ? at::empty(t.sizes(), t.options().dtype(at::kBFloat16)) : Tensor(); }
int32_t* status_ptr(const Tensor& t) { return t.data_ptr<int32_t>(); }

// ---------------------------------------------------------------------------- router and experts
struct LayerArgs {
  optional<Tensor> bias, codes, load;
  Tensor status;
  int64_t k, norm;
  double scale;
};

std::tuple<Tensor, Tensor, Tensor> layer_forward(const Tensor& x, const Tensor& gate, const Tensor& gate_up, const Tensor& down,
                                                 const LayerArgs& a, int keep) {
  const int64_t T = x.size(0), H = x.size(1), E = gate_up.size(0), I = down.size(2);
  Tensor ws = bytes(b200moe_layer_fwd_ws_bytes(T, H, I, E, a.k, keep), x);
  Tensor out = at::empty({T, H}, x.options()), counts = at::empty({E}, x.options().dtype(at::kInt));
  check(b200moe_layer_forward(ptr(x), ptr(gate), static_cast<const float*>(ptr(a.bias)), ptr(gate_up), ptr(down),
                              static_cast<const int32_t*>(ptr(a.codes)), T, H, I, E, a.k, a.norm, static_cast<float>(a.scale), keep, ptr(ws),
                              counts.data_ptr<int32_t>(), static_cast<int64_t*>(ptr(a.load)), ptr(out), status_ptr(a.status), stream_of(x)));
  return {out, counts, ws};
}

struct Layer : torch::autograd::Function<Layer> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& gate, const Tensor& gate_up, const Tensor& down,
                               const LayerArgs& a) {
    auto [out, counts, ws] = layer_forward(x, gate, gate_up, down, a, 1);
    variable_list saved{x, gate, gate_up, down, ws};
    if (a.codes.has_value()) saved.push_back(*a.codes);
    ctx->save_for_backward(std::move(saved));
    ctx->saved_data["status"] = a.status;
    ctx->saved_data["k"] = a.k;
    ctx->saved_data["norm"] = a.norm;
    ctx->saved_data["scale"] = a.scale;
    ctx->mark_non_differentiable({counts});
    ctx->set_materialize_grads(false);   // no zero-filled gradient for the counts
    return {out, counts};
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    variable_list res(5);
    if (!grads[0].defined()) return res;
    const variable_list s = ctx->get_saved_variables();
    const Tensor &x = s[0], &gate = s[1], &gate_up = s[2], &down = s[3], &ws = s[4];
    const Tensor codes = s.size() > 5 ? s[5] : Tensor(), status = ctx->saved_data["status"].toTensor();
    const int64_t T = x.size(0), H = x.size(1), E = gate_up.size(0), I = down.size(2), k = ctx->saved_data["k"].toInt();
    const c10::cuda::CUDAGuard guard(x.device());
    const Tensor go = grads[0].to(at::kBFloat16).contiguous();
    for (int i = 0; i < 4; ++i) res[i] = grad_like(ctx->needs_input_grad(i), s[i]);
    Tensor tmp = bytes(b200moe_layer_bwd_ws_bytes(T, H, I, E, k), x);
    check(b200moe_layer_backward(ptr(go), ptr(x), ptr(gate), ptr(gate_up), ptr(down), static_cast<const int32_t*>(ptr(codes)), T, H, I, E, k,
                                 ctx->saved_data["norm"].toInt(), static_cast<float>(ctx->saved_data["scale"].toDouble()), ptr(ws),
                                 ptr(tmp), ptr(res[0]), ptr(res[1]), ptr(res[2]), ptr(res[3]), status_ptr(status), stream_of(x)));
    return res;
  }
};

// (out (T,H), counts (E,) int32), or None
optional<std::tuple<Tensor, Tensor>> layer(const Tensor& x, const Tensor& gate, const optional<Tensor>& bias, const Tensor& gate_up,
                                           const Tensor& down, const optional<Tensor>& codes, const optional<Tensor>& load,
                                           const Tensor& status, int64_t k, int64_t norm, double scale) {
  if (!plain_call(x)) return std::nullopt;
  const auto dev = x.device();
  for (const Tensor* t : {&x, &gate, &gate_up, &down})
    if (!plain(*t, at::kBFloat16, dev)) return std::nullopt;
  if (!plain_or_none(bias, at::kFloat, dev) || !plain_or_none(codes, at::kInt, dev) || !plain_or_none(load, at::kLong, dev)) return std::nullopt;
  if (x.dim() != 2 || gate.dim() != 2 || gate_up.dim() != 3 || down.dim() != 3) return std::nullopt;
  const int64_t H = x.size(1), E = gate_up.size(0), I = down.size(2);
  if (x.size(0) == 0 || gate_up.size(1) != 2 * I || gate_up.size(2) != H || down.size(0) != E || down.size(1) != H || gate.size(0) != E ||
      gate.size(1) != H || (bias.has_value() && bias->numel() != E))
    return std::nullopt;
  const c10::cuda::CUDAGuard guard(dev);
  const LayerArgs a{bias, codes, load, status, k, norm, scale};
  if (at::GradMode::is_enabled() && (x.requires_grad() || gate.requires_grad() || gate_up.requires_grad() || down.requires_grad())) {
    variable_list r = Layer::apply(x, gate, gate_up, down, a);
    return std::make_tuple(r[0], r[1]);
  }
  auto [out, counts, ws] = layer_forward(x, gate, gate_up, down, a, 0);
  return std::make_tuple(out, counts);
}

// ---------------------------------------------------------------------------- experts on given picks
struct ExpertsArgs {
  Tensor idx;
  optional<Tensor> codes;
  Tensor status;
  int64_t E, row_kernels;
};

std::tuple<Tensor, Tensor> experts_forward(const Tensor& x, const Tensor& w, const Tensor& gate_up, const Tensor& down,
                                           const optional<Tensor>& params, const ExpertsArgs& a, int keep) {
  const int64_t T = x.size(0), H = x.size(1), n = gate_up.size(0), I = down.size(2), k = a.idx.size(1);
  Tensor ws = bytes(b200moe_moe_fwd_ws_bytes(T, H, I, a.E, n, k, keep, a.row_kernels), x), out = at::empty({T, H}, x.options());
  check(b200moe_moe_forward(ptr(x), a.idx.data_ptr<int64_t>(), w.data_ptr<float>(), ptr(gate_up), ptr(down),
                            static_cast<const int32_t*>(ptr(a.codes)), static_cast<const float*>(ptr(params)), T, H, I, a.E, n, k, keep,
                            a.row_kernels, ptr(ws), ptr(out), status_ptr(a.status), stream_of(x)));
  return {out, ws};
}

struct Experts : torch::autograd::Function<Experts> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, const Tensor& gate_up, const Tensor& down,
                        const optional<Tensor>& params, const ExpertsArgs& a) {
    auto [out, ws] = experts_forward(x, w, gate_up, down, params, a, 1);
    variable_list saved{ws, w, gate_up, down};
    if (a.codes.has_value()) saved.push_back(*a.codes);
    if (params.has_value()) saved.push_back(*params);
    ctx->save_for_backward(std::move(saved));
    ctx->saved_data["status"] = a.status;
    ctx->saved_data["has"] = static_cast<int64_t>((a.codes.has_value() ? 1 : 0) | (params.has_value() ? 2 : 0));
    ctx->saved_data["E"] = a.E;
    ctx->saved_data["rows"] = a.row_kernels;
    ctx->saved_data["H"] = x.size(1);
    return out;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list s = ctx->get_saved_variables();
    const Tensor &ws = s[0], &w = s[1], &gate_up = s[2], &down = s[3];
    const int64_t has = ctx->saved_data["has"].toInt(), E = ctx->saved_data["E"].toInt(), rows = ctx->saved_data["rows"].toInt();
    const Tensor codes = (has & 1) ? s[4] : Tensor(), params = (has & 2) ? s.back() : Tensor(), status = ctx->saved_data["status"].toTensor();
    const int64_t T = w.size(0), k = w.size(1), H = ctx->saved_data["H"].toInt(), n = gate_up.size(0), I = down.size(2);
    const c10::cuda::CUDAGuard guard(ws.device());
    const Tensor go = grads[0].to(at::kBFloat16).contiguous();
    const Tensor gw = at::empty_like(w);
    const Tensor gx = ctx->needs_input_grad(0) ? at::empty({T, H}, gate_up.options()) : Tensor();
    const Tensor ggu = grad_like(ctx->needs_input_grad(2), gate_up), gdn = grad_like(ctx->needs_input_grad(3), down);
    const Tensor gp = params.defined() && ctx->needs_input_grad(4) ? at::empty_like(params) : Tensor();
    Tensor tmp = bytes(b200moe_moe_bwd_ws_bytes(T, H, I, E, n, k, rows), ws);
    check(b200moe_moe_backward(ptr(go), w.data_ptr<float>(), ptr(gate_up), ptr(down), static_cast<const int32_t*>(ptr(codes)),
                               static_cast<const float*>(ptr(params)), T, H, I, E, n, k, rows, ptr(ws), ptr(tmp), ptr(gx), gw.data_ptr<float>(),
                               ptr(ggu), ptr(gdn), static_cast<float*>(ptr(gp)), status_ptr(status), stream_of(ws)));
    return {gx, ctx->needs_input_grad(1) ? gw : Tensor(), ggu, gdn, gp, Tensor()};
  }
};

// out (T,H), or None.  codes and params as the native call wants them: on the device, int32 and fp32
optional<Tensor> experts(const Tensor& x, const Tensor& idx, const Tensor& w, const Tensor& gate_up, const Tensor& down,
                         const optional<Tensor>& codes, const optional<Tensor>& params, const Tensor& status, int64_t E, int64_t n_glu,
                         int64_t row_kernels) {
  if (!plain_call(x)) return std::nullopt;
  const auto dev = x.device();
  for (const Tensor* t : {&x, &gate_up, &down})
    if (!plain(*t, at::kBFloat16, dev)) return std::nullopt;
  if (!plain(idx, at::kLong, dev) || !plain(w, at::kFloat, dev) || !plain_or_none(codes, at::kInt, dev) || !plain_or_none(params, at::kFloat, dev))
    return std::nullopt;
  if (x.dim() != 2 || idx.dim() != 2 || gate_up.dim() != 3 || down.dim() != 3 || x.size(0) == 0) return std::nullopt;
  const int64_t T = x.size(0), H = x.size(1), I = down.size(2);
  if (gate_up.size(0) != n_glu || gate_up.size(1) != 2 * I || gate_up.size(2) != H || down.size(0) != n_glu || down.size(1) != H ||
      idx.size(0) != T || w.sizes() != idx.sizes() || (codes.has_value() && codes->numel() != E) ||
      (params.has_value() && (params->dim() != 2 || params->size(0) != E || params->size(1) != 2)))
    return std::nullopt;
  const c10::cuda::CUDAGuard guard(dev);
  const ExpertsArgs a{idx, codes, status, E, row_kernels};
  if (at::GradMode::is_enabled() && (x.requires_grad() || w.requires_grad() || gate_up.requires_grad() || down.requires_grad() ||
                                     (params.has_value() && params->requires_grad())))
    return Experts::apply(x, w, gate_up, down, params, a);
  return std::get<0>(experts_forward(x, w, gate_up, down, params, a, row_kernels ? 1 : 0));
}

// ---------------------------------------------------------------------------- conv router
struct ConvArgs {
  optional<Tensor> bias;
  Tensor status;
  int64_t k, norm;
  double scale;
};

struct ConvRouter : torch::autograd::Function<ConvRouter> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight, const ConvArgs& a) {
    const int64_t B = x.size(0), S = x.size(1), H = x.size(2), E = weight.size(0), taps = weight.size(2);
    Tensor wt = at::empty({taps * E, H}, x.options()), logits = at::empty({B * S, E}, x.options());
    Tensor idx = at::empty({B, S, a.k}, x.options().dtype(at::kLong)), w = at::empty({B, S, a.k}, x.options().dtype(at::kFloat));
    Tensor counts = at::empty({E}, x.options().dtype(at::kInt)), ws = bytes(b200moe_conv_router_fwd_ws_bytes(B, S, H, E, taps), x);
    check(b200moe_conv_router_forward(ptr(x), ptr(weight), static_cast<const float*>(ptr(a.bias)), B, S, H, E, taps, a.k, a.norm,
                                      static_cast<float>(a.scale), ptr(ws), ptr(wt), ptr(logits), idx.data_ptr<int64_t>(),
                                      w.data_ptr<float>(), counts.data_ptr<int32_t>(), status_ptr(a.status), stream_of(x)));
    ctx->save_for_backward({x, wt, logits, idx});
    ctx->saved_data["status"] = a.status;
    ctx->saved_data["taps"] = taps;
    ctx->saved_data["norm"] = a.norm;
    ctx->saved_data["scale"] = a.scale;
    ctx->mark_non_differentiable({idx, counts});
    ctx->set_materialize_grads(false);
    return {idx, w, counts};
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    variable_list res(3);
    if (!grads[1].defined()) return res;
    const variable_list s = ctx->get_saved_variables();
    const Tensor &x = s[0], &wt = s[1], &logits = s[2], &idx = s[3];
    const Tensor status = ctx->saved_data["status"].toTensor();
    const int64_t taps = ctx->saved_data["taps"].toInt(), B = x.size(0), S = x.size(1), H = x.size(2), E = logits.size(1);
    const c10::cuda::CUDAGuard guard(x.device());
    const Tensor gw = grads[1].contiguous().to(at::kFloat);
    res[0] = grad_like(ctx->needs_input_grad(0), x);
    res[1] = ctx->needs_input_grad(1) ? at::empty({E, H, taps}, x.options()) : Tensor();
    Tensor ws = bytes(b200moe_conv_router_bwd_ws_bytes(B, S, H, E, taps), x);
    check(b200moe_conv_router_backward(ptr(x), ptr(wt), ptr(logits), idx.data_ptr<int64_t>(), gw.data_ptr<float>(), B, S, H, E, taps,
                                       idx.size(2), ctx->saved_data["norm"].toInt(), static_cast<float>(ctx->saved_data["scale"].toDouble()),
                                       ptr(ws), ptr(res[0]), ptr(res[1]), status_ptr(status), stream_of(x)));
    return res;
  }
};

// (idx (B,S,k) int64, weights (B,S,k) fp32, counts (E,) int32), or None
optional<std::tuple<Tensor, Tensor, Tensor>> conv_router(const Tensor& x, const Tensor& weight, const optional<Tensor>& bias,
                                                         const Tensor& status, int64_t k, int64_t experts, int64_t norm, double scale) {
  if (!plain_call(x)) return std::nullopt;
  const auto dev = x.device();
  if (!plain(x, at::kBFloat16, dev) || !plain(weight, at::kBFloat16, dev) || !plain_or_none(bias, at::kFloat, dev)) return std::nullopt;
  if (x.dim() != 3 || weight.dim() != 3 || weight.size(1) != x.size(2) || weight.size(0) != experts || x.numel() == 0 || k < 1 ||
      (bias.has_value() && bias->numel() != experts))
    return std::nullopt;
  const c10::cuda::CUDAGuard guard(dev);
  variable_list r = ConvRouter::apply(x, weight, ConvArgs{bias, status, k, norm, scale});
  return std::make_tuple(r[0], r[1], r[2]);
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.attr("torch_version") = TORCH_VERSION;
  m.def("layer", torch::wrap_pybind_function_no_gil(layer));
  m.def("experts", torch::wrap_pybind_function_no_gil(experts));
  m.def("conv_router", torch::wrap_pybind_function_no_gil(conv_router));
}
