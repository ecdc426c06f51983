// Graph nodes of the training path in C++: the operators of ops/functional.py and ops/gated_mlp.py with a graph, and whole blocks of them in one call.
//
// An autograd function in Python costs 25 to 45 us forward and about as much backward (its own apply, views, checks, the dispatch of every kernel), more than
// most kernels of a training block take up to some thousand tokens: a T5 decoder block of 16 x 128 tokens took 1200 us of which the GPU worked 420 (host time now 540).  Here
// a node is a torch::autograd::Function that launches the same kernels in the same order and saves the same tensors through save_for_backward, so
// saved-tensor hooks, checkpointing, retain_graph and the checks of versions see what they saw.  With create_graph the gradients are what they are without and have no graph, as
// those of the Python functions have none (kernels record nothing); only SplitAttention alone differentiates the unfused form then, for q, k and v that come from elsewhere.  Whatever transforms a call (vmap, forward-mode, traces) takes the
// Python functions as before; the caller decides (`_graph_node`).  Nothing is kept from one call for the next.
//
// Weight gradients go to `param.main_grad` where the parameter has one, which is a Python attribute that may come and go between forward and backward
// (sharded optimizers), so it is asked for in the backward pass.
#include <torch/csrc/autograd/autograd.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/pybind.h>
#include <torch/library.h>

#include <atomic>
#include <string>

#include "ops.h"

namespace lb_nodes {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::variable_list;
using Opt = std::optional<Tensor>;

std::atomic<int64_t> launches{0};       // kernels launched from here and by the blocks without a graph (ops.launch_count())
void count(int64_t n) { launches.fetch_add(n, std::memory_order_relaxed); }

// ---- attributes of parameters -----------------------------------------------------------------------------------
// p.main_grad, or undefined where there is none (with the GIL held, as the next)
Tensor main_grad(const Tensor& p) {
  static PyObject* const name = PyUnicode_InternFromString("main_grad");
  const auto obj = pybind11::reinterpret_steal<pybind11::object>(THPVariable_Wrap(p));
  const auto g = pybind11::reinterpret_steal<pybind11::object>(PyObject_GetAttr(obj.ptr(), name));
  if (g) return g.is_none() ? Tensor() : g.cast<Tensor>();
  if (!PyErr_ExceptionMatches(PyExc_AttributeError)) throw pybind11::error_already_set();
  PyErr_Clear();
  return {};
}
void mark_added(const Tensor& p) {
  static PyObject* const name = PyUnicode_InternFromString("grad_added_to_main_grad");
  const auto obj = pybind11::reinterpret_steal<pybind11::object>(THPVariable_Wrap(p));
  if (PyObject_SetAttr(obj.ptr(), name, Py_True) != 0) throw pybind11::error_already_set();
}
template <size_t N>
std::array<Tensor, N> main_grads(const std::array<const Tensor*, N>& params) {
  pybind11::gil_scoped_acquire gil;
  std::array<Tensor, N> grads;
  for (size_t i = 0; i < N; ++i)
    if (params[i]->defined()) grads[i] = main_grad(*params[i]);
  return grads;
}
template <size_t N>
void added_to_main_grad(const std::array<const Tensor*, N>& params) {
  pybind11::gil_scoped_acquire gil;
  for (const Tensor* p : params)
    if (p->defined()) mark_added(*p);
}
bool fp32(const Tensor& t) { return t.defined() && t.scalar_type() == at::kFloat; }

// ---- pieces ---------------------------------------------------------------------------------------------------------
Tensor rows(const Tensor& t) { return t.reshape({-1, t.size(-1)}).contiguous(); }
std::vector<int64_t> with_last(const Tensor& x, int64_t n) {
  std::vector<int64_t> s(x.sizes().begin(), x.sizes().end());
  s.back() = n;
  return s;
}
Opt opt(const Tensor& t) { return t.defined() ? Opt(t) : Opt(); }
bool requires_grad(const Opt& t) { return t.has_value() && t->defined() && t->requires_grad(); }
// which of a node's inputs want gradients, as the forward pass found them
int64_t bits(std::initializer_list<bool> need) {
  int64_t m = 0, i = 0;
  for (bool b : need) m |= static_cast<int64_t>(b) << i++;
  return m;
}
// A block's parameters themselves, whose main_grad is asked for: what is unpacked may be a copy (checkpointing, saved-tensor hooks).  As with the Python functions only the weights of
// norms and linear layers are saved tensors too; biases, and the weights of a gated MLP, which have to lie in one buffer, do not go through hooks.
void hold_parameters(AutogradContext* ctx, at::TensorList p) { ctx->saved_data["params"] = c10::List<Tensor>(p); }
std::vector<Tensor> held_parameters(AutogradContext* ctx) { return ctx->saved_data["params"].toTensorVector(); }
bool wants(AutogradContext* ctx, int i) { return (ctx->saved_data["need"].toInt() >> i) & 1; }
Tensor held(AutogradContext* ctx, const char* name) {
  const auto it = ctx->saved_data.find(name);
  return it == ctx->saved_data.end() ? Tensor() : it->second.toTensor();
}
// gᵀ x into main_grad, or as a tensor
Tensor weight_grad(const Tensor& g, const Tensor& x, const Tensor& w, const Tensor& main_grad) {
  count(1);
  if (main_grad.defined()) {
    lb_ops::gemm(g, x, 2, {}, main_grad, true, at::kFloat);
    added_to_main_grad<1>({&w});
    return {};
  }
  return lb_ops::gemm(g, x, 2, {}, {}, false, at::kFloat).to(w.scalar_type());
}
Tensor bias_grad(const Tensor& g, const Tensor& bias, const Tensor& main_grad) {
  count(1);
  if (fp32(main_grad)) {
    lb_ops::colsum(g, main_grad);
    added_to_main_grad<1>({&bias});
    return {};
  }
  return lb_ops::colsum(g, {}).to(bias.scalar_type());
}

// ---- nodes ----------------------------------------------------------------------------------------------------------
// (norm(x)[, x]): the gradient of the second output joins inside the norm's backward kernel
struct Norm : Function<Norm> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, const Opt& b, double eps, bool rms, bool with_skip) {
    const Tensor x2 = rows(x);
    auto [y, mean, rstd] = lb_ops::norm_fwd(x2, w, b, eps, rms);
    count(1);
    ctx->save_for_backward({x2, w, mean, rstd});
    ctx->saved_data["rms"] = rms;
    if (b.has_value() && b->defined()) ctx->saved_data["bias"] = *b;
    variable_list out{y.view(x.sizes())};
    if (with_skip) out.push_back(x.view_as(x));
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto s = ctx->get_saved_variables();
    const Tensor &x2 = s[0], &w = s[1], bias = held(ctx, "bias"), g2 = rows(g[0]);
    const bool rms = ctx->saved_data["rms"].toBool(), has_bias = bias.defined();
    const Opt skip = g.size() > 1 && g[1].defined() ? Opt(rows(g[1])) : Opt();
    count(2);
    const auto mg = main_grads<2>({&w, &bias});
    if (fp32(mg[0]) && (!has_bias || mg[1].defined())) {
      const Tensor gx = std::get<0>(lb_ops::norm_bwd(g2, x2, w, s[2], s[3], rms, has_bias, mg[0], opt(mg[1]), skip));
      added_to_main_grad<2>({&w, &bias});
      return {gx.view(g[0].sizes()), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
    }
    auto [gx, gw, gb] = lb_ops::norm_bwd(g2, x2, w, s[2], s[3], rms, has_bias, {}, {}, skip);
    return {gx.view(g[0].sizes()), gw.to(w.scalar_type()), has_bias ? gb.to(w.scalar_type()) : Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

// act(x wᵀ + b)
struct Linear : Function<Linear> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, const Opt& b, int64_t act) {
    const Tensor x2 = rows(x);
    const bool need_pre = act != 0 && (x.requires_grad() || w.requires_grad() || requires_grad(b));
    auto [y, pre] = lb_ops::linear_fwd(x2, w, b, act, need_pre);
    count(1);
    ctx->save_for_backward({x2, w, need_pre ? pre : Tensor()});
    ctx->saved_data["act"] = act;
    ctx->saved_data["need"] = bits({x.requires_grad(), w.requires_grad(), requires_grad(b)});
    ctx->saved_data["shape"] = x.sizes().vec();
    if (b.has_value() && b->defined()) ctx->saved_data["bias"] = *b;
    return y.view(with_last(x, w.size(0)));
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto s = ctx->get_saved_variables();
    const Tensor &x2 = s[0], &w = s[1], bias = held(ctx, "bias");
    const int64_t act = ctx->saved_data["act"].toInt();
    Tensor g2 = rows(g[0]), gx, gw, gb;
    if (act != 0) {
      g2 = lb_ops::act_bwd(g2, s[2], act);
      count(1);
    }
    const auto mg = main_grads<2>({&w, &bias});
    if (wants(ctx, 0)) {
      gx = lb_ops::gemm(g2, w, 1, {}, {}, false, at::kBFloat16).view(ctx->saved_data["shape"].toIntVector());
      count(1);
    }
    if (wants(ctx, 1)) gw = weight_grad(g2, x2, w, mg[0]);
    if (wants(ctx, 2)) gb = bias_grad(g2, bias, mg[1]);
    return {gx, gw, gb, Tensor()};
  }
};

// x wᵀ + b + residual
struct LinearResidual : Function<LinearResidual> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, const Opt& b, const Tensor& residual) {
    const Tensor x2 = rows(x);
    const Tensor y = lb_ops::linear_bias_residual(x2, w, b, residual.reshape({-1, w.size(0)}).contiguous());
    count(1);
    ctx->save_for_backward({x2, w});
    ctx->saved_data["need"] = bits({x.requires_grad(), w.requires_grad(), requires_grad(b)});
    ctx->saved_data["shape"] = x.sizes().vec();
    if (b.has_value() && b->defined()) ctx->saved_data["bias"] = *b;
    return y.view(with_last(x, w.size(0)));
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto s = ctx->get_saved_variables();
    const Tensor &x2 = s[0], &w = s[1], bias = held(ctx, "bias"), g2 = rows(g[0]);
    Tensor gx, gw, gb;
    const auto mg = main_grads<2>({&w, &bias});
    if (wants(ctx, 0)) {
      gx = lb_ops::gemm(g2, w, 1, {}, {}, false, at::kBFloat16).view(ctx->saved_data["shape"].toIntVector());
      count(1);
    }
    if (wants(ctx, 1)) gw = weight_grad(g2, x2, w, mg[0]);
    if (wants(ctx, 2)) gb = bias_grad(g2, bias, mg[1]);
    return {gx, gw, gb, g[0]};
  }
};

// act(x w1ᵀ + b1) w2ᵀ [+ b2 + residual]; the activation's derivative rides in the epilogue of the second layer's input gradient, with `fuse_bias` the
// column sums for b1 too
struct Mlp : Function<Mlp> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w1, const Opt& b1, const Tensor& w2, int64_t act, const Opt& b2, const Opt& residual,
                        bool fuse_bias) {
    const Tensor x2 = rows(x);
    const bool need[] = {x.requires_grad(), w1.requires_grad(), requires_grad(b1), w2.requires_grad(), requires_grad(b2), requires_grad(residual)};
    const bool any = need[0] || need[1] || need[2] || need[3] || need[4] || need[5];
    auto [h, pre] = lb_ops::linear_fwd(x2, w1, b1, act, any);
    const bool has_res = residual.has_value() && residual->defined();
    const Tensor y = has_res ? lb_ops::linear_bias_residual(h, w2, b2, residual->reshape({-1, w2.size(0)}).contiguous())
                             : std::get<0>(lb_ops::linear_fwd(h, w2, b2, 0, false));
    count(2);
    ctx->save_for_backward({x2, w1, w2, pre, h});
    ctx->saved_data["act"] = act;
    ctx->saved_data["fuse"] = fuse_bias;
    ctx->saved_data["res"] = has_res;
    ctx->saved_data["need"] = bits({need[0], need[1], need[2], need[3], need[4]});
    ctx->saved_data["shape"] = x.sizes().vec();
    if (b1.has_value() && b1->defined()) ctx->saved_data["b1"] = *b1;
    if (b2.has_value() && b2->defined()) ctx->saved_data["b2"] = *b2;
    return y.view(with_last(x, w2.size(0)));
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto s = ctx->get_saved_variables();
    const Tensor &x2 = s[0], &w1 = s[1], &w2 = s[2], &pre = s[3], &h = s[4], b1 = held(ctx, "b1"), b2 = held(ctx, "b2"), g2 = rows(g[0]);
    const auto mg = main_grads<4>({&w1, &b1, &w2, &b2});
    const bool fused = wants(ctx, 2) && ctx->saved_data["fuse"].toBool() && fp32(mg[1]) && mg[1].is_contiguous();
    const Tensor dpre = lb_ops::dgrad_actgrad(g2, w2, pre, ctx->saved_data["act"].toInt(), fused ? Opt(mg[1]) : Opt());
    count(1);
    Tensor gx, gw1, gw2, gb1, gb2;
    if (wants(ctx, 3)) gw2 = weight_grad(g2, h, w2, mg[2]);
    if (wants(ctx, 1)) gw1 = weight_grad(dpre, x2, w1, mg[0]);
    if (fused) added_to_main_grad<1>({&b1});
    else if (wants(ctx, 2)) gb1 = bias_grad(dpre, b1, mg[1]);
    if (wants(ctx, 0)) {
      gx = lb_ops::gemm(dpre, w1, 1, {}, {}, false, at::kBFloat16).view(ctx->saved_data["shape"].toIntVector());
      count(1);
    }
    if (wants(ctx, 4)) gb2 = bias_grad(g2, b2, mg[3]);
    return {gx, gw1, gb1, gw2, Tensor(), gb2, ctx->saved_data["res"].toBool() ? g[0] : Tensor(), Tensor()};
  }
};

// two weights that lie one behind the other in one buffer, as one [2 F, K] matrix (undefined where they do not)
Tensor stacked(const Tensor& a, const Tensor& b) {
  if (!a.defined() || !b.defined() || a.dim() != 2 || a.sizes() != b.sizes() || a.scalar_type() != b.scalar_type() || !a.is_contiguous() || !b.is_contiguous() ||
      a.storage().data() != b.storage().data() || b.data_ptr() != static_cast<char*>(a.data_ptr()) + a.nbytes())
    return {};
  return a.detach().as_strided({2 * a.size(0), a.size(1)}, {a.size(1), 1});
}
// (silu(x Wgᵀ) * (x Wuᵀ)) Wdᵀ [+ residual]
struct GatedMlp : Function<GatedMlp> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& wg, const Tensor& wu, const Tensor& wd, const Opt& residual) {
    const Tensor w = stacked(wg, wu), x2 = rows(x);
    TORCH_CHECK(w.defined(), "gated_mlp: gate and up weights of one buffer");
    const Tensor gu = lb_ops::gemm(x2, w, 0, {}, {}, false, at::kBFloat16), h = lb_ops::swiglu_packed_fwd(gu);
    const bool has_res = residual.has_value() && residual->defined();
    const Tensor y = has_res ? lb_ops::linear_bias_residual(h, wd, {}, residual->reshape({-1, wd.size(0)}).contiguous())
                             : lb_ops::gemm(h, wd, 0, {}, {}, false, at::kBFloat16);
    count(3);
    ctx->save_for_backward({x2, gu, h});
    ctx->saved_data["wg"] = wg;
    ctx->saved_data["wu"] = wu;
    ctx->saved_data["wd"] = wd;
    ctx->saved_data["res"] = has_res;
    ctx->saved_data["need"] = bits({x.requires_grad(), wg.requires_grad(), wu.requires_grad(), wd.requires_grad()});
    return y.view(with_last(x, wd.size(0)));
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto s = ctx->get_saved_variables();
    const Tensor &x2 = s[0], &gu = s[1], &h = s[2], wg = held(ctx, "wg"), wu = held(ctx, "wu"), wd = held(ctx, "wd"), g2 = rows(g[0]), w = stacked(wg, wu);
    TORCH_CHECK(w.defined(), "gated_mlp: gate and up weights of one buffer");
    const auto mg = main_grads<3>({&wg, &wu, &wd});
    const Tensor joint = fp32(mg[0]) ? stacked(mg[0], mg[1]) : Tensor();
    const Tensor dh = lb_ops::gemm(g2, wd, 1, {}, {}, false, at::kBFloat16);
    Tensor gx, gwg, gwu, gwd;
    if (wants(ctx, 3)) gwd = weight_grad(g2, h, wd, mg[2]);
    const Tensor dgu = lb_ops::swiglu_packed_bwd(dh, gu);
    if (wants(ctx, 0)) gx = lb_ops::gemm(dgu, w, 1, {}, {}, false, at::kBFloat16).view(with_last(g[0], x2.size(1)));
    if (wants(ctx, 1) || wants(ctx, 2)) {
      count(1);
      if (joint.defined()) {
        lb_ops::gemm(dgu, x2, 2, {}, joint, true, at::kFloat);
        added_to_main_grad<2>({&wg, &wu});
      } else {
        const Tensor out = lb_ops::gemm(dgu, x2, 2, {}, {}, false, at::kFloat);
        const int64_t f = wg.size(0);
        gwg = out.narrow(0, 0, f).to(wg.scalar_type());
        gwu = out.narrow(0, f, f).to(wu.scalar_type());
      }
    }
    count(3);
    return {gx, gwg, gwu, gwd, ctx->saved_data["res"].toBool() ? g[0] : Tensor()};
  }
};

// attention of the packed projection [b, s, a, 3 d] -> [b, s, a, d] (flash kernels)
struct FlashPacked : Function<FlashPacked> {
  static std::array<Tensor, 3> parts(const Tensor& qkv) {
    const int64_t d = qkv.size(-1) / 3;
    const Tensor v4 = qkv.permute({0, 2, 1, 3});
    return {v4.narrow(3, 0, d), v4.narrow(3, d, d), v4.slice(3, 2 * d)};
  }
  static Tensor forward(AutogradContext* ctx, const Tensor& qkv, bool causal, double scale, const Opt& kv_lens, double p_drop, const Opt& slopes, int64_t salt) {
    const auto [q, k, v] = parts(qkv);
    auto [o, lse, rng] = lb_ops::attn_fwd(q, k, v, causal, scale, kv_lens, {}, slopes, p_drop, salt);
    count(1);
    ctx->save_for_backward({qkv, o, lse, kv_lens.value_or(Tensor()), rng, slopes.value_or(Tensor())});
    ctx->saved_data["causal"] = causal;
    ctx->saved_data["scale"] = scale;
    ctx->saved_data["p_drop"] = p_drop;
    return o.permute({0, 2, 1, 3});
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto s = ctx->get_saved_variables();
    const auto [q, k, v] = parts(s[0]);
    const double p_drop = ctx->saved_data["p_drop"].toDouble();
    const Tensor dqkv = std::get<3>(lb_ops::attn_bwd(g[0].permute({0, 2, 1, 3}), q, k, v, s[1], s[2], ctx->saved_data["causal"].toBool(),
                                                     ctx->saved_data["scale"].toDouble(), opt(s[3]), {}, opt(s[5]), {}, p_drop, p_drop > 0 ? opt(s[4]) : Opt()));
    count(3);
    return {dqkv.view(s[0].sizes()), Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

// attention with 32-bit probabilities; layout 0: [b, s, a, 3 d], 1: [b, s, a, d] and [b, sk, a, 2 d], 2: q, k, v [b, a, s, d]
struct SplitAttention : Function<SplitAttention> {
  static std::array<Tensor, 3> parts(int64_t layout, const Tensor& t0, const Tensor& t1, const Tensor& t2) {
    if (layout == 2) return {t0, t1, t2};
    if (layout == 1) {
      const auto kv = t1.permute({0, 2, 1, 3}).chunk(2, -1);
      return {t0.permute({0, 2, 1, 3}), kv[0], kv[1]};
    }
    const auto c = t0.permute({0, 2, 1, 3}).chunk(3, -1);
    return {c[0], c[1], c[2]};
  }
  static Tensor forward(AutogradContext* ctx, const Tensor& t0, const Opt& t1, const Opt& t2, int64_t layout, bool causal, double scale, const Opt& mask) {
    const Tensor a1 = t1.value_or(Tensor()), a2 = t2.value_or(Tensor());
    const auto [q, k, v] = parts(layout, t0, a1, a2);
    Tensor words, fill;
    const bool masked = mask.has_value() && mask->defined();
    if (masked) {
      Tensor m = *mask;
      while (m.dim() < 4) m = m.unsqueeze(0);
      std::tie(words, fill) = lb_ops::attn_mask_pack(m.expand({m.size(0), m.size(1), q.size(2), k.size(2)}), causal);
      count(1);
    }
    const bool train = t0.requires_grad() || requires_grad(t1) || requires_grad(t2);
    auto [o, o32, lse] = lb_ops::attn_split_fwd(q, k, v, causal && !masked, scale, opt(words), opt(fill), train);
    count(1);
    if (train) {
      ctx->save_for_backward({o32, lse, words, fill, t0, a1, a2});
      ctx->saved_data["layout"] = layout;
      ctx->saved_data["causal"] = causal;
      ctx->saved_data["scale"] = scale;
      ctx->saved_data["need"] = bits({t0.requires_grad(), requires_grad(t1), requires_grad(t2)});
      if (masked) ctx->saved_data["mask"] = *mask;
    }
    return layout == 2 ? o : o.permute({0, 2, 1, 3});
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto s = ctx->get_saved_variables();
    const int64_t layout = ctx->saved_data["layout"].toInt();
    const bool causal = ctx->saved_data["causal"].toBool();
    const double scale = ctx->saved_data["scale"].toDouble();
    const int n = layout == 2 ? 3 : layout == 1 ? 2 : 1;
    variable_list grads(7);
    if (at::GradMode::is_enabled()) {    // a graph of the gradients is wanted: the unfused form is differentiated
      pybind11::gil_scoped_acquire gil;
      static const char* const names[] = {"qkv", "q_kv", "q_k_v"};
      pybind11::list ts, need;
      for (int i = 0; i < n; ++i) {
        ts.append(s[4 + i]);
        need.append(pybind11::bool_(wants(ctx, i)));
      }
      const Tensor mask = held(ctx, "mask");
      const pybind11::list got = pybind11::module_::import("libai_b200.ops.functional").attr("_split_graph_backward")(
          g[0], names[layout], causal, scale, mask.defined() ? pybind11::cast(mask) : pybind11::none(), ts, need);
      for (int i = 0; i < n; ++i)
        if (!got[i].is_none()) grads[i] = got[i].cast<Tensor>();
      return grads;
    }
    const auto [q, k, v] = parts(layout, s[4], s[5], s[6]);
    Tensor go = g[0];
    for (int i = 0; i < n; ++i) {
      const Tensor& t = s[4 + i];
      // (gradients backed by [b, s, a, d], as the projections around an attention read them)
      grads[i] = layout == 2 ? at::empty({t.size(0), t.size(2), t.size(1), t.size(3)}, t.options()).permute({0, 2, 1, 3}) : at::empty(t.sizes(), t.options());
    }
    if (layout != 2) go = go.permute({0, 2, 1, 3});
    const auto [gq, gk, gv] = parts(layout, grads[0], grads[1], grads[2]);
    lb_ops::attn_split_bwd(go, q, k, v, s[0], s[1], gq, gk, gv, causal && !s[2].defined(), scale, opt(s[2]), opt(s[3]));
    count(3);
    return grads;
  }
};

// rotary embedding on q and k of the packed projection; the gradient is rotated back in place
struct RopeQkv : Function<RopeQkv> {
  static Tensor forward(AutogradContext* ctx, const Tensor& qkv, const Tensor& cos, const Tensor& sin, int64_t at) {
    ctx->save_for_backward({cos, sin});
    ctx->saved_data["at"] = at;
    count(1);
    return lb_ops::rope_qkv(qkv, cos, sin, at, false, false);
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto s = ctx->get_saved_variables();
    count(1);
    return {lb_ops::rope_qkv(g[0].contiguous(), s[0], s[1], ctx->saved_data["at"].toInt(), true, true), Tensor(), Tensor(), Tensor()};
  }
};

// loss per token over the whole vocabulary; the gradient takes the place of the logits
struct CrossEntropy : Function<CrossEntropy> {
  static Tensor forward(AutogradContext* ctx, const Tensor& logits, const Tensor& labels, int64_t start) {
    auto [mx, se, tgt] = lb_ops::ce_stats(logits, labels, start);
    count(1);
    const Tensor lse = mx + se.log();
    ctx->save_for_backward({logits, labels, lse});
    ctx->saved_data["start"] = start;
    return lse - tgt;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto s = ctx->get_saved_variables();
    count(1);
    return {lb_ops::ce_bwd(s[0], s[1], s[2], g[0].contiguous().to(at::kFloat), ctx->saved_data["start"].toInt()), Tensor(), Tensor()};
  }
};

// ---- operators --------------------------------------------------------------------------------------------------------
Tensor norm(const Tensor& x, const Tensor& w, const Opt& b, double eps, bool rms) { return Norm::apply(x, w, b, eps, rms, false)[0]; }
std::tuple<Tensor, Tensor> norm_skip(const Tensor& x, const Tensor& w, const Opt& b, double eps, bool rms) {
  auto y = Norm::apply(x, w, b, eps, rms, true);
  return std::make_tuple(y[0], y[1]);
}
Tensor linear(const Tensor& x, const Tensor& w, const Opt& b, int64_t act) { return Linear::apply(x, w, b, act); }
Tensor linear_residual(const Tensor& x, const Tensor& w, const Opt& b, const Tensor& residual) { return LinearResidual::apply(x, w, b, residual); }
Tensor mlp(const Tensor& x, const Tensor& w1, const Opt& b1, const Tensor& w2, int64_t act, const Opt& b2, const Opt& residual, bool fuse_bias) {
  return Mlp::apply(x, w1, b1, w2, act, b2, residual, fuse_bias);
}
Tensor gated_mlp(const Tensor& x, const Tensor& wg, const Tensor& wu, const Tensor& wd, const Opt& residual) { return GatedMlp::apply(x, wg, wu, wd, residual); }
Tensor flash_packed(const Tensor& qkv, bool causal, double scale, const Opt& kv_lens, double p_drop, const Opt& slopes, int64_t salt) {
  return FlashPacked::apply(qkv, causal, scale, kv_lens, p_drop, slopes, salt);
}
Tensor split_attention(const std::vector<Tensor>& ts, bool causal, double scale, const Opt& mask, int64_t layout) {
  TORCH_CHECK(layout >= 0 && layout <= 2 && ts.size() == static_cast<size_t>(layout) + 1, "split attention: one tensor packed, two or three");
  return SplitAttention::apply(ts[0], ts.size() > 1 ? Opt(ts[1]) : Opt(), ts.size() > 2 ? Opt(ts[2]) : Opt(), layout, causal, scale, mask);
}
Tensor rope_qkv(const Tensor& qkv, const Tensor& cos, const Tensor& sin, int64_t at) { return RopeQkv::apply(qkv, cos, sin, at); }
Tensor cross_entropy(const Tensor& logits, const Tensor& labels, int64_t start) { return CrossEntropy::apply(logits, labels, start); }

// ---- whole blocks ---------------------------------------------------------------------------------------------------------
// A pre-norm block's parameters: norm weight, bias; qkv weight, bias; projection weight, bias; [norm weight, bias; query weight, bias; key and value weight, bias;
// projection weight, bias of the cross attention;] norm weight, bias; h->4h weight, bias; 4h->h weight, bias.
struct BlockArgs {
  int64_t heads;
  std::vector<double> eps;
  double scale, cross_scale;
  bool causal, fuse_bias;               // causal: the triangle alone (a mask stands in its place, lengths stand beside it)
  Opt kv_lens, mask, cross_mask;
};

// (norm(x), x), with the skip connection's gradient joined where x has one
std::tuple<Tensor, Tensor> norm_and_skip(const Tensor& x, const Tensor& w, const Opt& b, double eps, bool rms) {
  if (x.requires_grad()) return norm_skip(x, w, b, eps, rms);
  return std::make_tuple(norm(x, w, b, eps, rms), x);
}
bool has(const Opt& t) { return t.has_value() && t->defined(); }
bool flash(const BlockArgs& a, int64_t d) { return !has(a.mask) && (d == 64 || d == 128); }

// the nodes above in the order in which the modules make them
Tensor block_of_nodes(const Tensor& x, at::TensorList p, const Opt& enc, const BlockArgs& a) {
  const int64_t B = x.size(0), ad = p[2].size(0) / 3, d = ad / a.heads;
  const size_t m = has(enc) ? 14 : 6;
  auto [ln, skip] = norm_and_skip(x, p[0], p[1], a.eps[0], false);
  const Tensor qkv = Linear::apply(ln, p[2], Opt(p[3]), 0).view({B, -1, a.heads, 3 * d});
  const Tensor c = flash(a, d) ? FlashPacked::apply(qkv, a.causal, a.scale, a.kv_lens, 0.0, Opt(), 0)
                               : SplitAttention::apply(qkv, Opt(), Opt(), 0, a.causal, a.scale, a.mask);
  Tensor y = LinearResidual::apply(c.reshape({B, -1, ad}), p[4], Opt(p[5]), skip);
  if (has(enc)) {
    std::tie(ln, skip) = norm_and_skip(y, p[6], p[7], a.eps[1], false);
    const Tensor q = Linear::apply(ln, p[8], Opt(p[9]), 0).view({B, -1, a.heads, d}), kv = Linear::apply(*enc, p[10], Opt(p[11]), 0).view({B, -1, a.heads, 2 * d});
    const Tensor o = SplitAttention::apply(q, Opt(kv), Opt(), 1, false, a.cross_scale, a.cross_mask);
    y = LinearResidual::apply(o.reshape({B, -1, ad}), p[12], Opt(p[13]), skip);
  }
  std::tie(ln, skip) = norm_and_skip(y, p[m], p[m + 1], a.eps.back(), false);
  return Mlp::apply(ln, p[m + 2], Opt(p[m + 3]), p[m + 4], 1 /* GELU */, Opt(p[m + 5]), Opt(skip), a.fuse_bias);
}
Tensor llama_of_nodes(const Tensor& x, at::TensorList p, const Opt& bias, const Tensor& cos, const Tensor& sin, int64_t heads, double eps1, double eps2,
                      double scale) {
  const int64_t B = x.size(0), ad = p[1].size(0) / 3, d = ad / heads;
  auto [ln, skip] = norm_and_skip(x, p[0], Opt(), eps1, true);
  const Tensor qkv = RopeQkv::apply(Linear::apply(ln, p[1], bias, 0).view({B, -1, heads, 3 * d}), cos, sin, 0);
  const Tensor y = LinearResidual::apply(FlashPacked::apply(qkv, true, scale, Opt(), 0.0, Opt(), 0).reshape({B, -1, ad}), p[2], Opt(), skip);
  std::tie(ln, skip) = norm_and_skip(y, p[3], Opt(), eps2, true);
  return GatedMlp::apply(ln, p[4], p[5], p[6], Opt(skip));
}

// One node for a block all of whose parameters want gradients: between the nodes above, the engine and the views cost as much as the launches do
// (GPT-2 like block of 864 tokens x 256, forward and backward: 745 us of host time with the Python functions, 454 with a node per operator, 309 with one; the GPU works 131).
struct Gradients {                        // of the parameters, by index
  std::vector<Tensor> main, out;          // main_grad, or undefined; what goes back to the engine
  std::vector<char> added;
  const std::vector<Tensor>& params;
  explicit Gradients(const std::vector<Tensor>& p) : main(p.size()), out(p.size()), added(p.size(), 0), params(p) {
    pybind11::gil_scoped_acquire gil;
    for (size_t i = 0; i < p.size(); ++i) main[i] = main_grad(p[i]);
  }
  void weight(size_t i, const Tensor& g, const Tensor& x) {
    count(1);
    if (main[i].defined()) {
      lb_ops::gemm(g, x, 2, {}, main[i], true, at::kFloat);
      added[i] = 1;
    } else {
      out[i] = lb_ops::gemm(g, x, 2, {}, {}, false, at::kFloat).to(params[i].scalar_type());
    }
  }
  void bias(size_t i, const Tensor& g) {
    if (added[i]) return;
    count(1);
    if (fp32(main[i])) {
      lb_ops::colsum(g, main[i]);
      added[i] = 1;
    } else {
      out[i] = lb_ops::colsum(g, {}).to(params[i].scalar_type());
    }
  }
  // gradient of the norm's input, `skip` added; the norm's parameters are i and, with has_bias, i + 1
  Tensor norm(size_t i, const Tensor& g, const Tensor& x, const Tensor& w, const Tensor& mean, const Tensor& rstd, bool rms, bool has_bias, const Tensor& skip) {
    count(2);
    if (fp32(main[i]) && (!has_bias || main[i + 1].defined())) {
      added[i] = 1;
      if (has_bias) added[i + 1] = 1;
      return std::get<0>(lb_ops::norm_bwd(g, x, w, mean, rstd, rms, has_bias, main[i], has_bias ? Opt(main[i + 1]) : Opt(), skip));
    }
    auto [gx, gw, gb] = lb_ops::norm_bwd(g, x, w, mean, rstd, rms, has_bias, {}, {}, skip);
    out[i] = gw.to(w.scalar_type());
    if (has_bias) out[i + 1] = gb.to(w.scalar_type());
    return gx;
  }
  // the same of a layer norm, with the gradients of the biases around it: `before` that of the layer that made its input (column sums of the result), `behind` that of the
  // layer whose output the skip connection joined (column sums of `skip`; -1: not asked for).  Those that it has not made are left to bias().
  Tensor norm_and_biases(size_t i, const Tensor& g, const Tensor& x, const Tensor& w, const Tensor& mean, const Tensor& rstd, const Tensor& skip, int before, int behind) {
    if (fp32(main[i]) && fp32(main[i + 1]) && fp32(main[before]) && (behind < 0 || fp32(main[behind]))) {
      const Tensor gx = lb_ops::norm_bwd_sums(g, x, w, mean, rstd, main[i], main[i + 1], skip, behind < 0 ? Tensor() : main[behind], main[before]);
      if (gx.defined()) {
        count(1);
        added[i] = added[i + 1] = added[before] = 1;
        if (behind >= 0) added[behind] = 1;
        return gx;
      }
    }
    return norm(i, g, x, w, mean, rstd, false, true, skip);
  }
  void mark() const {
    pybind11::gil_scoped_acquire gil;
    for (size_t i = 0; i < params.size(); ++i)
      if (added[i]) mark_added(params[i]);
  }
};
Tensor input_grad(const Tensor& g, const Tensor& w) {
  count(1);
  return lb_ops::gemm(g, w, 1, {}, {}, false, at::kBFloat16);
}

// What a block's backward pass needs of its forward pass.  A tensor goes through saved-tensor hooks and the check of its version as save_for_backward sends it, but alone and as
// soon as it is there: hooks that take it elsewhere free it then, and the backward pass unpacks it where it is used and, unless the graph is kept, lets go of it behind that, as the
// engine does between the nodes of single operators.  Peak of a step of 4 x 1024 tokens, MiB, all saved at once and unpacked at once -> so (a node per operator): GPT-2 block of width
// 1024 233 -> 168 (176), 16 heads of 48 271 -> 174 (174), T5 decoder 313 -> 179 (185), Llama block 272 -> 182 (212); forward under checkpointing hooks 128 -> 80 (88).
struct Kept : torch::CustomClassHolder {
  std::vector<torch::autograd::SavedVariable> at;
};
class Keep {
 public:
  Keep(AutogradContext* ctx, size_t n) : kept_(c10::make_intrusive<Kept>()), outside_(c10::impl::tls_local_dispatch_key_set()) {
    kept_->at.resize(n);
    ctx->saved_data["kept"] = c10::IValue::make_capsule(kept_);
  }
  const Tensor& operator()(size_t i, const Tensor& t) {
    c10::impl::ForceDispatchKeyGuard as_outside(outside_);              // (hooks run whatever they like)
    kept_->at[i] = torch::autograd::SavedVariable(t, /*is_output=*/false);
    return t;
  }

 private:
  c10::intrusive_ptr<Kept> kept_;
  const c10::impl::LocalDispatchKeySet outside_;
};
class Take {
 public:
  explicit Take(AutogradContext* ctx)
      : kept_(c10::static_intrusive_pointer_cast<Kept>(ctx->saved_data["kept"].toCapsule())), outside_(c10::impl::tls_local_dispatch_key_set()),
        keep_graph_(torch::autograd::get_current_graph_task_keep_graph()) {
    ctx->get_saved_variables();                                         // (none; raises where an earlier pass has let go of what was kept)
  }
  Tensor operator()(size_t i) {                                         // once per pass: checkpointing hooks allow no more
    c10::impl::ForceDispatchKeyGuard as_outside(outside_);
    Tensor t = kept_->at[i].unpack();
    if (!keep_graph_) kept_->at[i].reset_data();
    return t;
  }

 private:
  const c10::intrusive_ptr<Kept> kept_;
  const c10::impl::LocalDispatchKeySet outside_;
  const bool keep_graph_;
};

struct Block : Function<Block> {
  // a norm's weight, result, mean and reciprocal deviation; the weights of products with what they read; attention: o32, log-sum-exp, mask words and fill, or of the flash
  // kernels log-sum-exp and lengths
  enum : size_t {
    X, ENC, NORM1, QKV_W = NORM1 + 4, QKV, ATT, CTX = ATT + 4, O_W, Y1, NORMC, Q_W = NORMC + 4, Q, KV_W, KV, CATT, CCTX = CATT + 4, CO_W, Y2, NORM2, FF1_W = NORM2 + 4, PRE, FF2_W, ACT, KEPT
  };
  static Tensor forward(AutogradContext* ctx, const Tensor& x, at::TensorList p, const Opt& enc, const BlockArgs& a) {
    const int64_t B = x.size(0), S = x.size(1), h = x.size(2), T = B * S, ad = p[2].size(0) / 3, d = ad / a.heads;
    const size_t m = has(enc) ? 14 : 6;
    Keep keep(ctx, KEPT);
    keep(X, x);
    Tensor y;
    {
      at::AutoDispatchBelowADInplaceOrView guard;
      auto norm = [&](const Tensor& t, size_t i, double eps, size_t to) {
        auto [ln, mean, rstd] = lb_ops::norm_fwd(t, p[i], p[i + 1], eps, false);
        keep(to, p[i]);
        keep(to + 1, ln);
        keep(to + 2, mean);
        keep(to + 3, rstd);
        return ln;
      };
      auto linear = [&](const Tensor& t, size_t i, size_t to) { return keep(to + 1, std::get<0>(lb_ops::linear_fwd(t, keep(to, p[i]), p[i + 1], 0, false))); };
      auto attend = [&](const Tensor& q, const Tensor& k, const Tensor& v, bool causal, double scale, const Opt& mask, size_t to) {
        Tensor words, fill;
        if (has(mask)) {
          Tensor w = *mask;
          while (w.dim() < 4) w = w.unsqueeze(0);
          std::tie(words, fill) = lb_ops::attn_mask_pack(w.expand({w.size(0), w.size(1), q.size(2), k.size(2)}), causal);
          count(1);
        }
        auto [o, o32, lse] = lb_ops::attn_split_fwd(q, k, v, causal && !has(mask), scale, opt(words), opt(fill), true);
        keep(to, o32);
        keep(to + 1, lse);
        keep(to + 2, words);
        keep(to + 3, fill);
        return o;
      };
      const Tensor x2 = x.view({T, h});
      {
        const Tensor qkv = linear(norm(x2, 0, a.eps[0], NORM1), 2, QKV_W).view({B, S, a.heads, 3 * d});
        Tensor o;
        if (flash(a, d)) {
          const auto [q, k, v] = FlashPacked::parts(qkv);
          auto [f, lse, rng] = lb_ops::attn_fwd(q, k, v, a.causal, a.scale, a.kv_lens, {}, {}, 0.0, 0);
          keep(ATT, lse);
          if (has(a.kv_lens)) keep(ATT + 1, *a.kv_lens);
          o = f;
        } else {
          const auto [q, k, v] = SplitAttention::parts(0, qkv, {}, {});
          o = attend(q, k, v, a.causal, a.scale, a.mask, ATT);
        }
        const Tensor c = keep(CTX, o.permute({0, 2, 1, 3}).view({T, ad}));
        y = keep(Y1, lb_ops::linear_bias_residual(c, keep(O_W, p[4]), p[5], x2));
      }
      if (has(enc)) {
        Tensor cc;
        {
          const Tensor q = linear(norm(y, 6, a.eps[1], NORMC), 8, Q_W).view({B, S, a.heads, d});
          const Tensor kv = linear(keep(ENC, *enc).view({-1, h}), 10, KV_W).view({B, -1, a.heads, 2 * d});
          const auto [q4, k4, v4] = SplitAttention::parts(1, q, kv, {});
          cc = keep(CCTX, attend(q4, k4, v4, false, a.cross_scale, a.cross_mask, CATT).permute({0, 2, 1, 3}).view({T, ad}));
        }
        y = keep(Y2, lb_ops::linear_bias_residual(cc, keep(CO_W, p[12]), p[13], y));
        count(5);
      }
      auto [act, pre] = lb_ops::linear_fwd(norm(y, m, a.eps.back(), NORM2), keep(FF1_W, p[m + 2]), p[m + 3], 1 /* GELU */, true);
      keep(PRE, pre);
      keep(ACT, act);
      pre = Tensor();
      y = lb_ops::linear_bias_residual(act, keep(FF2_W, p[m + 4]), p[m + 5], y);
      count(7);
    }
    hold_parameters(ctx, p);
    ctx->saved_data["heads"] = a.heads;
    ctx->saved_data["scales"] = std::vector<double>{a.scale, a.cross_scale};
    ctx->saved_data["flags"] = bits({a.causal, a.fuse_bias, has(enc), requires_grad(enc), flash(a, d)});
    return y.view(x.sizes());
  }

  static variable_list backward(AutogradContext* ctx, variable_list grad) {
    Take take(ctx);
    const int64_t flags = ctx->saved_data["flags"].toInt(), heads = ctx->saved_data["heads"].toInt();
    const bool causal = flags & 1, fuse = flags & 2, cross = flags & 4, by_flash = flags & 16;
    const size_t m = cross ? 14 : 6;
    const auto scales = ctx->saved_data["scales"].toDoubleVector();
    const std::vector<Tensor> p = held_parameters(ctx);
    const std::vector<int64_t> sizes = grad[0].sizes().vec();
    Gradients g(p);
    Tensor gx, genc;
    {
      at::AutoDispatchBelowADInplaceOrView guard;
      const int64_t B = sizes[0], S = sizes[1], h = sizes[2], T = B * S, ad = p[2].size(0) / 3, d = ad / heads;
      Tensor gy = rows(grad[0]), dln;
      grad.clear();
      {
        const bool fused = fuse && fp32(g.main[m + 3]) && g.main[m + 3].is_contiguous();
        const Tensor dpre = lb_ops::dgrad_actgrad(gy, take(FF2_W), take(PRE), 1, fused ? Opt(g.main[m + 3]) : Opt());
        count(1);
        g.weight(m + 4, gy, take(ACT));
        g.weight(m + 2, dpre, take(NORM2 + 1));
        if (fused) g.added[m + 3] = 1;
        else g.bias(m + 3, dpre);
        dln = input_grad(dpre, take(FF1_W));
      }
      Tensor dy = g.norm_and_biases(m, dln, take(cross ? Y2 : Y1), take(NORM2), take(NORM2 + 2), take(NORM2 + 3), gy, cross ? 13 : 5, static_cast<int>(m) + 5);
      g.bias(m + 5, gy);
      gy = dln = Tensor();
      auto attend_back = [&](int64_t layout, const Tensor& t0, const Tensor& t1, const Tensor& dctx, size_t kept, bool causal_, double scale, Tensor& g0, Tensor& g1) {
        g0 = at::empty(t0.sizes(), t0.options());
        if (layout == 1) g1 = at::empty(t1.sizes(), t1.options());
        const auto [q, kk, v] = SplitAttention::parts(layout, t0, t1, {});
        const auto [gq, gk, gv] = SplitAttention::parts(layout, g0, g1, {});
        const Tensor words = take(kept + 2);
        lb_ops::attn_split_bwd(dctx.view({B, S, heads, d}).permute({0, 2, 1, 3}), q, kk, v, take(kept), take(kept + 1), gq, gk, gv, causal_ && !words.defined(), scale,
                               opt(words), opt(take(kept + 3)));
        count(3);
      };
      if (cross) {
        Tensor gq, gkv;
        {
          const Tensor dctx = input_grad(dy, take(CO_W));
          g.weight(12, dy, take(CCTX));
          g.bias(13, dy);
          attend_back(1, take(Q).view({B, S, heads, d}), take(KV).view({B, -1, heads, 2 * d}), dctx, CATT, false, scales[1], gq, gkv);
        }
        gq = gq.view({T, ad});
        gkv = gkv.view({-1, 2 * ad});
        const Tensor kv_w = take(KV_W);
        if (flags & 8) genc = input_grad(gkv, kv_w).view({B, -1, h});
        g.weight(10, gkv, take(ENC).view({-1, h}));
        g.bias(11, gkv);
        gkv = Tensor();
        dln = input_grad(gq, take(Q_W));
        g.weight(8, gq, take(NORMC + 1));
        g.bias(9, gq);
        gq = Tensor();
        dy = g.norm_and_biases(6, dln, take(Y1), take(NORMC), take(NORMC + 2), take(NORMC + 3), dy, 5, -1);
        dln = Tensor();
      }
      Tensor dqkv, none;
      {
        const Tensor dctx = input_grad(dy, take(O_W));
        Tensor c = take(CTX);
        g.weight(4, dy, c);
        g.bias(5, dy);
        if (!by_flash) c = Tensor();
        const Tensor qkv = take(QKV).view({B, S, heads, 3 * d});
        if (by_flash) {
          const auto [q, kk, v] = FlashPacked::parts(qkv);
          dqkv = std::get<3>(lb_ops::attn_bwd(dctx.view({B, S, heads, d}).permute({0, 2, 1, 3}), q, kk, v, c.view({B, S, heads, d}).permute({0, 2, 1, 3}), take(ATT), causal,
                                              scales[0], opt(take(ATT + 1)), {}, {}, {}, 0.0, {}));
          count(3);
        } else {
          attend_back(0, qkv, {}, dctx, ATT, causal, scales[0], dqkv, none);
        }
      }
      dqkv = dqkv.view({T, 3 * ad});
      dln = input_grad(dqkv, take(QKV_W));
      g.weight(2, dqkv, take(NORM1 + 1));
      g.bias(3, dqkv);
      dqkv = Tensor();
      gx = g.norm(0, dln, take(X).view({T, h}), take(NORM1), take(NORM1 + 2), take(NORM1 + 3), false, true, dy);
    }
    g.mark();
    const size_t n = p.size();
    variable_list out(n + 3);              // x, parameters, enc, arguments
    out[0] = gx.view(sizes);
    for (size_t i = 0; i < n; ++i) out[1 + i] = g.out[i];
    out[1 + n] = genc;
    return out;
  }
};

// Llama block, head dim 64 or 128: parameters norm; qkv; projection; norm; gate, up (one behind the other in memory), down[; bias of qkv]
struct LlamaBlock : Function<LlamaBlock> {
  enum : size_t { X, COS, SIN, NORM1, QKV_W = NORM1 + 4, QKV, LSE, CTX, O_W, Y1, NORM2, GU = NORM2 + 4, ACT, KEPT };       // (norms as in Block)
  static Tensor forward(AutogradContext* ctx, const Tensor& x, at::TensorList p, const Tensor& cos, const Tensor& sin, int64_t heads, double eps1, double eps2,
                        double scale) {
    const int64_t B = x.size(0), S = x.size(1), h = x.size(2), T = B * S, ad = p[1].size(0) / 3, d = ad / heads;
    Keep keep(ctx, KEPT);
    keep(X, x);
    keep(COS, cos);
    keep(SIN, sin);
    Tensor y;
    {
      at::AutoDispatchBelowADInplaceOrView guard;
      auto norm = [&](const Tensor& t, size_t i, double eps, size_t to) {
        auto [ln, mean, rstd] = lb_ops::norm_fwd(t, p[i], {}, eps, true);
        keep(to, p[i]);
        keep(to + 1, ln);
        keep(to + 2, mean);
        keep(to + 3, rstd);
        return ln;
      };
      const Tensor x2 = x.view({T, h});
      Tensor y1, act;
      {
        Tensor qkv = std::get<0>(lb_ops::linear_fwd(norm(x2, 0, eps1, NORM1), keep(QKV_W, p[1]), p.size() > 7 ? Opt(p[7]) : Opt(), 0, false)).view({B, S, heads, 3 * d});
        qkv = keep(QKV, lb_ops::rope_qkv(qkv, cos, sin, 0, false, false));
        const auto [q, k, v] = FlashPacked::parts(qkv);
        auto [o, lse, rng] = lb_ops::attn_fwd(q, k, v, true, scale, {}, {}, {}, 0.0, 0);
        keep(LSE, lse);
        y1 = keep(Y1, lb_ops::linear_bias_residual(keep(CTX, o.permute({0, 2, 1, 3}).view({T, ad})), keep(O_W, p[2]), {}, x2));
      }
      {
        const Tensor gu = keep(GU, lb_ops::gemm(norm(y1, 3, eps2, NORM2), stacked(p[4], p[5]), 0, {}, {}, false, at::kBFloat16));
        act = keep(ACT, lb_ops::swiglu_packed_fwd(gu));
      }
      y = lb_ops::linear_bias_residual(act, p[6], {}, y1);
      count(9);
    }
    hold_parameters(ctx, p);
    ctx->saved_data["heads"] = heads;
    ctx->saved_data["scale"] = scale;
    return y.view(x.sizes());
  }
  static variable_list backward(AutogradContext* ctx, variable_list grad) {
    Take take(ctx);
    const int64_t heads = ctx->saved_data["heads"].toInt();
    const double scale = ctx->saved_data["scale"].toDouble();
    const std::vector<Tensor> p = held_parameters(ctx);
    const std::vector<int64_t> sizes = grad[0].sizes().vec();
    const size_t n = p.size();
    Gradients g(p);
    Tensor gx;
    {
      at::AutoDispatchBelowADInplaceOrView guard;
      const int64_t B = sizes[0], S = sizes[1], h = sizes[2], T = B * S, ad = p[1].size(0) / 3, d = ad / heads, f = p[4].size(0);
      const Tensor w = stacked(p[4], p[5]);
      TORCH_CHECK(w.defined(), "llama block: gate and up weights of one buffer");
      Tensor gy = rows(grad[0]), dln;
      grad.clear();
      {
        const Tensor joint = fp32(g.main[4]) ? stacked(g.main[4], g.main[5]) : Tensor();
        Tensor dh = input_grad(gy, p[6]);
        g.weight(6, gy, take(ACT));
        const Tensor dgu = lb_ops::swiglu_packed_bwd(dh, take(GU));
        dh = Tensor();
        dln = input_grad(dgu, w);
        const Tensor ln = take(NORM2 + 1);
        if (joint.defined()) {
          lb_ops::gemm(dgu, ln, 2, {}, joint, true, at::kFloat);
          g.added[4] = g.added[5] = 1;
        } else {
          const Tensor both = lb_ops::gemm(dgu, ln, 2, {}, {}, false, at::kFloat);
          g.out[4] = both.narrow(0, 0, f).to(p[4].scalar_type());
          g.out[5] = both.narrow(0, f, f).to(p[5].scalar_type());
        }
      }
      const Tensor dy = g.norm(3, dln, take(Y1), take(NORM2), take(NORM2 + 2), take(NORM2 + 3), true, false, gy);
      gy = dln = Tensor();
      const Tensor cos = take(COS), sin = take(SIN);
      Tensor dqkv;
      {
        const Tensor dctx = input_grad(dy, take(O_W)), c = take(CTX);
        g.weight(2, dy, c);
        const auto [q, kk, v] = FlashPacked::parts(take(QKV));
        dqkv = std::get<3>(lb_ops::attn_bwd(dctx.view({B, S, heads, d}).permute({0, 2, 1, 3}), q, kk, v, c.view({B, S, heads, d}).permute({0, 2, 1, 3}), take(LSE), true, scale,
                                            {}, {}, {}, {}, 0.0, {}));
      }
      dqkv = lb_ops::rope_qkv(dqkv.view({B, S, heads, 3 * d}), cos, sin, 0, true, true).view({T, 3 * ad});
      dln = input_grad(dqkv, take(QKV_W));
      g.weight(1, dqkv, take(NORM1 + 1));
      if (n > 7) g.bias(7, dqkv);
      dqkv = Tensor();
      gx = g.norm(0, dln, take(X).view({T, h}), take(NORM1), take(NORM1 + 2), take(NORM1 + 3), true, false, dy);
      count(6);                            // attention, rotation, SwiGLU, gate and up weights
    }
    g.mark();
    variable_list out(n + 7);              // x, parameters, cos, sin, heads, eps, eps, scale
    out[0] = gx.view(sizes);
    for (size_t i = 0; i < n; ++i) out[1 + i] = g.out[i];
    return out;
  }
};

bool all_want_gradients(at::TensorList p) {
  for (const Tensor& t : p)
    if (!t.requires_grad()) return false;
  return true;
}

// An empty answer of these two: not of the form that they take, the caller's modules run.
std::vector<Tensor> block(const Tensor& x, const std::vector<Tensor>& p, int64_t heads, at::ArrayRef<double> eps, double scale, bool causal, const Opt& kv_lens,
                          const Opt& mask, const Opt& enc, const Opt& cross_mask, double cross_scale, bool fuse_bias) {
  const bool cross = has(enc);
  const size_t m = cross ? 14 : 6;                       // first of the feed-forward's parameters
  if (p.size() != m + 6 || eps.size() != (cross ? 3u : 2u) || x.dim() != 3 || !lb_ops::block_tensor(x, x) || x.numel() == 0 || heads <= 0 || p[2].dim() != 2 ||
      p[m + 2].dim() != 2)
    return {};
  const int64_t B = x.size(0), h = x.size(2), ad = p[2].size(0) / 3, d = ad / heads, f = p[m + 2].size(0);
  auto linear_ok = [&](size_t i, int64_t n, int64_t k) { return lb_ops::block_matrix(p[i], x, n, k) && lb_ops::block_vector(p[i + 1], x, n); };
  auto norm_ok = [&](size_t i) { return lb_ops::block_vector(p[i], x, h) && lb_ops::block_vector(p[i + 1], x, h); };
  if (p[2].size(0) != 3 * heads * d || d % 8 || !norm_ok(0) || !linear_ok(2, 3 * ad, h) || !linear_ok(4, h, ad) || !norm_ok(m) || !linear_ok(m + 2, f, h) ||
      !linear_ok(m + 4, h, f))
    return {};
  if (cross && (enc->dim() != 3 || !lb_ops::block_tensor(*enc, x) || enc->numel() == 0 || enc->size(0) != B || enc->size(2) != h || !norm_ok(6) ||
                !linear_ok(8, ad, h) || !linear_ok(10, 2 * ad, h) || !linear_ok(12, h, ad)))
    return {};
  const BlockArgs a{heads, eps.vec(), scale, cross_scale, causal && !has(mask), fuse_bias, kv_lens, mask, cross_mask};
  return {all_want_gradients(p) ? Block::apply(x, at::TensorList(p), enc, a) : block_of_nodes(x, p, enc, a)};
}

std::vector<Tensor> llama_block(const Tensor& x, const std::vector<Tensor>& p, const Opt& bias, const Tensor& cos, const Tensor& sin, int64_t heads, double eps1,
                                double eps2, double scale) {
  if (p.size() != 7 || x.dim() != 3 || !lb_ops::block_tensor(x, x) || x.numel() == 0 || heads <= 0 || p[1].dim() != 2 || p[4].dim() != 2) return {};
  const int64_t S = x.size(1), h = x.size(2), ad = p[1].size(0) / 3, d = ad / heads, f = p[4].size(0);
  if (p[1].size(0) != 3 * heads * d || (d != 64 && d != 128) || !lb_ops::block_vector(p[0], x, h) || !lb_ops::block_matrix(p[1], x, 3 * ad, h) ||
      !lb_ops::block_matrix(p[2], x, h, ad) || !lb_ops::block_vector(p[3], x, h) || !lb_ops::block_matrix(p[4], x, f, h) || !lb_ops::block_matrix(p[5], x, f, h) ||
      !lb_ops::block_matrix(p[6], x, h, f) || !stacked(p[4], p[5]).defined() || (has(bias) && !lb_ops::block_vector(*bias, x, 3 * ad)))
    return {};
  for (const Tensor* t : {&cos, &sin})
    if (!(t->defined() && t->is_cuda() && t->device() == x.device() && t->scalar_type() == at::kFloat && t->dim() == 2 && t->is_contiguous() && t->size(0) >= S &&
          t->size(1) == d && !t->requires_grad()))
      return {};
  if (cos.sizes() != sin.sizes()) return {};
  std::vector<Tensor> all(p);
  if (has(bias)) all.push_back(*bias);
  return {all_want_gradients(all) ? LlamaBlock::apply(x, at::TensorList(all), cos, sin, heads, eps1, eps2, scale)
                                  : llama_of_nodes(x, p, bias, cos, sin, heads, eps1, eps2, scale)};
}

int64_t launched(bool reset) { return reset ? launches.exchange(0) : launches.load(); }

}  // namespace lb_nodes

TORCH_LIBRARY_FRAGMENT(libai_b200, m) {
  m.def("norm_node(Tensor x, Tensor weight, Tensor? bias, float eps, bool rms) -> Tensor", &lb_nodes::norm);
  m.def("norm_skip_node(Tensor x, Tensor weight, Tensor? bias, float eps, bool rms) -> (Tensor, Tensor)", &lb_nodes::norm_skip);
  m.def("linear_node(Tensor x, Tensor w, Tensor? bias, int act) -> Tensor", &lb_nodes::linear);
  m.def("linear_residual_node(Tensor x, Tensor w, Tensor? bias, Tensor residual) -> Tensor", &lb_nodes::linear_residual);
  m.def("mlp_node(Tensor x, Tensor w1, Tensor? b1, Tensor w2, int act, Tensor? b2, Tensor? residual, bool fuse_bias) -> Tensor", &lb_nodes::mlp);
  m.def("gated_mlp_node(Tensor x, Tensor wg, Tensor wu, Tensor wd, Tensor? residual) -> Tensor", &lb_nodes::gated_mlp);
  m.def("flash_packed_node(Tensor qkv, bool causal, float scale, Tensor? kv_lens, float p_drop, Tensor? slopes, int salt) -> Tensor", &lb_nodes::flash_packed);
  m.def("split_attention_node(Tensor[] ts, bool causal, float scale, Tensor? mask, int layout) -> Tensor", &lb_nodes::split_attention);
  m.def("rope_qkv_node(Tensor qkv, Tensor cos, Tensor sin, int at) -> Tensor", &lb_nodes::rope_qkv);
  m.def("cross_entropy_node(Tensor logits, Tensor labels, int start) -> Tensor", &lb_nodes::cross_entropy);
  m.def("block_nodes(Tensor x, Tensor[] params, int heads, float[] eps, float scale, bool causal, Tensor? kv_lens, Tensor? mask, Tensor? enc, Tensor? cross_mask, float cross_scale, bool fuse_bias) -> Tensor[]", &lb_nodes::block);
  m.def("llama_block_nodes(Tensor x, Tensor[] params, Tensor? bias, Tensor cos, Tensor sin, int heads, float eps1, float eps2, float scale) -> Tensor[]", &lb_nodes::llama_block);
  m.def("launched(bool reset) -> int", &lb_nodes::launched);
}
