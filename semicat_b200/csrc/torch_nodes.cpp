// The library's ops as native autograd nodes, for the two situations that the training and sampling passes are made of: no
// forward-mode level at all, and exactly one torch.func.jvp around plain CUDA tensors.
//
// An op is entered from Python through one function of the module below, whose first argument says which of the two it is
// (`semicat_b200._nodes.native`).  Its inputs are looked at next (`fits`); in any other situation (vmap, nested transforms,
// forward_ad duals without a transform, tracing, dispatch or function modes, tensor subclasses, shapes that the kernels do
// not take) it returns None and the caller goes the general way, through the torch.autograd.Function classes in Python.
//
// Under torch.func.jvp an op is two dispatcher ops.  The outer one runs on the transform's wrappers: it takes the tangents off
// the inputs, calls the inner one on primals and tangents, and hangs the returned tangents on the returned primals.  The inner
// one has left the transform's level by the time its autograd kernel runs (the dispatcher unwraps on the way), so its
// node is an ordinary reverse-mode node on ordinary tensors: (primals, tangents) -> (outputs, output tangents).  In Python
// the same thing is a class built per call, a transform of a custom function and a node whose backward needs the
// interpreter: forward and gradient of one attention call took 780-900 us of host time that way for 22-50 us of kernels.
#include <ATen/autocast_mode.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/extension.h>

#include <atomic>

#include "../../include/jvpattn.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::variable_list;
using Opt = std::optional<Tensor>;

std::atomic<int> g_kernels{JVPATTN_KERNELS_AUTO};

// A failed call raises what semicat_b200._lib.check raises; the node may run on an engine thread.
void check(int rc, const char *where) {
  if (rc == JVPATTN_OK) return;
  pybind11::gil_scoped_acquire gil;
  try {
    pybind11::module_::import("semicat_b200._lib").attr("check")(rc, where);
  } catch (pybind11::error_already_set &e) {
    e.restore();
    python_error err;
    err.persist();
    throw err;
  }
}

void *stream_of(const Tensor &t) { return c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }
void *ptr(const Tensor &t) { return t.defined() ? t.data_ptr() : nullptr; }
Tensor unit(const Tensor &t) { return !t.defined() || t.stride(-1) == 1 ? t : t.contiguous(); }
Tensor dense(const Tensor &t) { return t.defined() ? t.contiguous() : t; }
// an absent tangent and a symbolic zero are the same
Tensor value(const Opt &t) { return t.has_value() && t->defined() && !t->_is_zerotensor() ? *t : Tensor(); }
Opt opt(const Tensor &t) { return t.defined() ? Opt(t) : std::nullopt; }
bool any_grad(std::initializer_list<const Tensor *> ts) {
  if (!at::GradMode::is_enabled()) return false;
  for (const Tensor *t : ts)
    if (t->defined() && t->requires_grad()) return true;
  return false;
}

// Gradients of a node that may be passed once only (as torch.autograd.function.once_differentiable has it).
variable_list once(const variable_list &cotangents, variable_list grads) {
  if (!at::GradMode::is_enabled()) return grads;
  bool again = false;
  for (const Tensor &g : cotangents) again = again || (g.defined() && g.requires_grad());
  if (!again) return grads;
  std::vector<size_t> live;
  variable_list in;
  for (size_t i = 0; i < grads.size(); ++i)
    if (grads[i].defined()) live.push_back(i), in.push_back(grads[i].detach().requires_grad_());
  auto error = std::make_shared<torch::autograd::DelayedError>(
      "trying to differentiate twice a function that was marked with @once_differentiable", (int64_t)in.size());
  variable_list out = (*error)(std::move(in));
  for (size_t k = 0; k < live.size(); ++k) grads[live[k]] = out[k];
  return grads;
}

// ------------------------------------------------------------------------------------------------ attention
jvpattn_tensor t4(const Tensor &t, bool bshd) {
  return {ptr(t), {t.stride(0), t.stride(bshd ? 2 : 1), t.stride(bshd ? 1 : 2), t.stride(3)}};
}

// (what is made anew has the memory order that it would have from (B, H, S, D) views)
Tensor unit(const Tensor &t, bool bshd) {
  return !bshd || !t.defined() || t.stride(-1) == 1 ? unit(t) : t.transpose(1, 2).contiguous().transpose(1, 2);
}
Tensor like_input(const Tensor &x, bool bshd) {
  if (bshd && !x.is_non_overlapping_and_dense()) return like_input(x.transpose(1, 2), false).transpose(1, 2);
  Tensor out = at::empty_like(x);
  return out.stride(-1) == 1 ? out : at::empty(x.sizes(), x.options());
}

struct Heads {
  int64_t B, H, Lq, Lk, D, rows;
  Heads(const Tensor &q, const Tensor &k, bool bshd)
      : B(q.size(0)), H(q.size(bshd ? 2 : 1)), Lq(q.size(bshd ? 1 : 2)), Lk(k.size(bshd ? 1 : 2)), D(q.size(3)),
        rows((Lq + 127) / 128 * 128) {}
  jvpattn_problem problem(const Tensor &q) const {
    return {(int32_t)B, (int32_t)H, (int32_t)Lq, (int32_t)Lk, (int32_t)D, (int32_t)rows,
            q.scalar_type() == at::kBFloat16 ? JVPATTN_BF16 : JVPATTN_FP16, g_kernels.load(), 0.f};
  }
};

// -> y, ty, lse, mu (ty and mu undefined without tangents).  The outputs are (B, S, H, D)-contiguous memory either way.
std::array<Tensor, 4> attention_forward(const Tensor &q, const Tensor &k, const Tensor &v, Tensor tq, Tensor tk, Tensor tv, bool bshd) {
  c10::cuda::CUDAGuard guard(q.device());
  const Heads n(q, k, bshd);
  const bool dual = tq.defined() || tk.defined() || tv.defined();
  Tensor y = at::empty({n.B, n.Lq, n.H, n.D}, q.options()), ty, mu;
  Tensor lse = at::empty({n.B, n.H, n.rows}, q.options().dtype(at::kFloat));
  const Tensor qu = unit(q, bshd), ku = unit(k, bshd), vu = unit(v, bshd);
  if (dual) {
    ty = at::empty_like(y);
    mu = n.rows == n.Lq ? at::empty_like(lse) : at::zeros_like(lse);
    // an input without a tangent has tangent zero
    tq = tq.defined() ? unit(tq, bshd) : at::zeros_like(qu);
    tk = tk.defined() ? unit(tk, bshd) : at::zeros_like(ku);
    tv = tv.defined() ? unit(tv, bshd) : at::zeros_like(vu);
  }
  const jvpattn_problem p = n.problem(q);
  const jvpattn_tensor q4 = t4(qu, bshd), k4 = t4(ku, bshd), v4 = t4(vu, bshd), y4 = t4(y, true);
  jvpattn_tensor tq4, tk4, tv4, ty4;
  if (dual) tq4 = t4(tq, bshd), tk4 = t4(tk, bshd), tv4 = t4(tv, bshd), ty4 = t4(ty, true);
  check(jvpattn_fwd(&p, &q4, &k4, &v4, dual ? &tq4 : nullptr, dual ? &tk4 : nullptr, dual ? &tv4 : nullptr, &y4, dual ? &ty4 : nullptr,
                    lse.data_ptr<float>(), dual ? mu.data_ptr<float>() : nullptr, nullptr, stream_of(q)),
        "jvpattn_fwd");
  if (!bshd) y = y.transpose(1, 2), ty = dual ? ty.transpose(1, 2) : ty;
  return {y, ty, lse, mu};
}

// Without g_ty (plain attention backward) the tangents get no gradient.
std::array<Tensor, 6> attention_backward(Tensor q, Tensor k, Tensor v, Tensor tq, Tensor tk, Tensor tv, const Tensor &y, const Tensor &ty,
                                         const Tensor &lse, const Tensor &mu, Tensor gy, Tensor gty, bool bshd) {
  c10::cuda::CUDAGuard guard(q.device());
  const bool dual = gty.defined();
  q = unit(q, bshd), k = unit(k, bshd), v = unit(v, bshd), gy = unit(gy, bshd), gty = unit(gty, bshd);
  if (dual) {
    tq = tq.defined() ? unit(tq, bshd) : at::zeros_like(q);
    tk = tk.defined() ? unit(tk, bshd) : at::zeros_like(k);
    tv = tv.defined() ? unit(tv, bshd) : at::zeros_like(v);
  }
  const Heads n(q, k, bshd);
  const jvpattn_problem p = n.problem(q);
  const size_t need = jvpattn_bwd_workspace_bytes(&p);
  Tensor workspace = need ? at::empty({(int64_t)need}, q.options().dtype(at::kByte)) : Tensor();
  std::array<Tensor, 6> grads = {like_input(q, bshd), like_input(k, bshd), like_input(v, bshd)};
  if (dual) grads[3] = like_input(tq, bshd), grads[4] = like_input(tk, bshd), grads[5] = like_input(tv, bshd);
  const Tensor *given[16] = {&q, &k, &v, &tq, &tk, &tv, &y, &ty, &gy, &gty, &grads[0], &grads[1], &grads[2], &grads[3], &grads[4], &grads[5]};
  jvpattn_tensor t[16];
  const jvpattn_tensor *a[16];
  for (int i = 0; i < 16; ++i) {
    const bool tangent = (i >= 3 && i < 6) || i == 7 || i >= 13;
    a[i] = given[i]->defined() && (dual || !tangent) ? &(t[i] = t4(*given[i], bshd)) : nullptr;
  }
  check(jvpattn_bwd(&p, a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7], a[8], a[9], lse.data_ptr<float>(),
                    dual ? mu.data_ptr<float>() : nullptr, a[10], a[11], a[12], a[13], a[14], a[15], ptr(workspace), need, stream_of(q)),
        "jvpattn_bwd");
  return grads;
}

// (q, k, v, tq, tk, tv) -> (y, ty): a reverse pass meets one node with whichever cotangents exist and makes one library call.
struct AttentionPair : Function<AttentionPair> {
  static variable_list forward(AutogradContext *ctx, const Tensor &q, const Tensor &k, const Tensor &v, const Opt &tq_, const Opt &tk_,
                               const Opt &tv_, bool bshd) {
    at::AutoDispatchBelowADInplaceOrView below;
    const Tensor tq = value(tq_), tk = value(tk_), tv = value(tv_);
    auto [y, ty, lse, mu] = attention_forward(q, k, v, tq, tk, tv, bshd);
    ctx->save_for_backward({q, k, v, tq, tk, tv, y, ty, lse, mu});
    ctx->set_materialize_grads(false);
    ctx->saved_data["bshd"] = bshd;
    return {y, ty};
  }
  static variable_list backward(AutogradContext *ctx, const variable_list &g) {
    if (!g[0].defined() && !g[1].defined()) return variable_list(7);
    const auto s = ctx->get_saved_variables();
    std::array<Tensor, 6> d;
    {
      at::AutoDispatchBelowADInplaceOrView below;
      at::NoGradGuard off;
      d = attention_backward(s[0], s[1], s[2], s[3], s[4], s[5], s[6], s[7], s[8], s[9], g[0], g[1], ctx->saved_data["bshd"].toBool());
    }
    for (int i = 3; i < 6; ++i)
      if (!s[i].defined()) d[i] = Tensor();
    return once(g, {d[0], d[1], d[2], d[3], d[4], d[5], Tensor()});
  }
};

struct AttentionPrimal : Function<AttentionPrimal> {
  static Tensor forward(AutogradContext *ctx, const Tensor &q, const Tensor &k, const Tensor &v, bool bshd) {
    at::AutoDispatchBelowADInplaceOrView below;
    auto [y, ty, lse, mu] = attention_forward(q, k, v, {}, {}, {}, bshd);
    ctx->save_for_backward({q, k, v, y, lse});
    ctx->set_materialize_grads(false);
    ctx->saved_data["bshd"] = bshd;
    return y;
  }
  static variable_list backward(AutogradContext *ctx, const variable_list &g) {
    if (!g[0].defined()) return variable_list(4);
    const auto s = ctx->get_saved_variables();
    std::array<Tensor, 6> d;
    {
      at::AutoDispatchBelowADInplaceOrView below;
      at::NoGradGuard off;
      d = attention_backward(s[0], s[1], s[2], {}, {}, {}, s[3], {}, s[4], {}, g[0], {}, ctx->saved_data["bshd"].toBool());
    }
    return once(g, {d[0], d[1], d[2], Tensor()});
  }
};

std::tuple<Tensor, Tensor> attention_pair(const Tensor &q, const Tensor &k, const Tensor &v, const Opt &tq, const Opt &tk, const Opt &tv,
                                          bool bshd) {
  auto out = attention_forward(q, k, v, value(tq), value(tk), value(tv), bshd);
  if (!out[1].defined()) out[1] = at::zeros_like(out[0]);  // every tangent was a symbolic zero
  return {out[0], out[1]};
}
std::tuple<Tensor, Tensor> attention_pair_autograd(const Tensor &q, const Tensor &k, const Tensor &v, const Opt &tq, const Opt &tk,
                                                   const Opt &tv, bool bshd) {
  const Tensor t[3] = {value(tq), value(tk), value(tv)};
  if (any_grad({&q, &k, &v, &t[0], &t[1], &t[2]}) && (t[0].defined() || t[1].defined() || t[2].defined())) {
    auto out = AttentionPair::apply(q, k, v, tq, tk, tv, bshd);
    return {out[0], out[1]};
  }
  if (any_grad({&q, &k, &v})) {
    Tensor y = AttentionPrimal::apply(q, k, v, bshd);
    return {y, at::zeros_like(y)};
  }
  at::AutoDispatchBelowADInplaceOrView below;
  return attention_pair(q, k, v, tq, tk, tv, bshd);
}
Tensor attention_primal(const Tensor &q, const Tensor &k, const Tensor &v, bool bshd) {
  return attention_forward(q, k, v, {}, {}, {}, bshd)[0];
}
Tensor attention_primal_autograd(const Tensor &q, const Tensor &k, const Tensor &v, bool bshd) {
  if (any_grad({&q, &k, &v})) return AttentionPrimal::apply(q, k, v, bshd);
  at::AutoDispatchBelowADInplaceOrView below;
  return attention_primal(q, k, v, bshd);
}

// ------------------------------------------------------------------------------------------------ LayerNorm + modulation
int code(const Tensor &t) { return t.scalar_type() == at::kBFloat16 ? JVPATTN_BF16 : JVPATTN_FP32; }
const float *fptr(const Tensor &t) { return t.defined() ? t.data_ptr<float>() : nullptr; }
float *fmut(const Tensor &t) { return t.defined() ? t.data_ptr<float>() : nullptr; }

// A (B, 1, C) or (B, C) modulation tensor as (B, C) rows of unit stride that start on 16 bytes.
Tensor mod_rows(const Tensor &t) {
  if (!t.defined()) return t;
  Tensor r = t.dim() == 3 ? t.select(1, 0) : t;
  const bool ok = r.stride(1) == 1 && r.stride(0) % 8 == 0 && reinterpret_cast<uintptr_t>(r.data_ptr()) % 16 == 0;
  return ok ? r : r.contiguous();
}
int64_t pitch(const Tensor &a, const Tensor &b) { return a.defined() ? a.stride(0) : b.defined() ? b.stride(0) : 0; }
// two of them with one row pitch
void equal_pitch(Tensor &a, Tensor &b) {
  if (a.defined() && b.defined() && a.stride(0) != b.stride(0)) a = a.contiguous(), b = b.contiguous();
}

struct LnInputs {
  Tensor x, tx, gamma, beta, shift, scale, tshift, tscale;
  double eps;
  bool exact;
};
struct LnRows {
  Tensor sh, sc, tsh, tsc;
  explicit LnRows(const LnInputs &a) : sh(mod_rows(a.shift)), sc(mod_rows(a.scale)), tsh(mod_rows(a.tshift)), tsc(mod_rows(a.tscale)) {
    equal_pitch(sh, sc);
    equal_pitch(tsh, tsc);
  }
};

void ln_launch(int which, const LnInputs &a, const LnRows &m, const Tensor &tx, const Tensor &mean, const Tensor &rstd, const Tensor &out,
               const Tensor &g, const Tensor &dx, const Tensor &dtx, float *sums, int exact) {
  const Tensor &x = a.x;
  check(jvpattn_ln_modulate(which, ptr(x), ptr(tx), fptr(a.gamma), fptr(a.beta), ptr(m.sh), ptr(m.sc), ptr(m.tsh), ptr(m.tsc),
                            pitch(m.sc, m.sh), pitch(m.tsc, m.tsh), fmut(mean), fmut(rstd), ptr(out), ptr(g), ptr(dx), ptr(dtx), sums,
                            (int)x.size(0), (int)x.size(1), (int)x.size(2), (float)a.eps, exact, code(x), stream_of(x)),
        "jvpattn_ln_modulate");
}
void ln_dual_launch(int which, const LnInputs &a, const LnRows &m, const Tensor &mean, const Tensor &rstd, const Tensor &y, const Tensor &ty,
                    const Tensor &g, const Tensor &gt, const Tensor &dx, const Tensor &dtx, float *sums) {
  const Tensor &x = a.x;
  check(jvpattn_ln_modulate_dual(which, ptr(x), ptr(a.tx), fptr(a.gamma), fptr(a.beta), ptr(m.sh), ptr(m.sc), ptr(m.tsh), ptr(m.tsc),
                                 pitch(m.sc, m.sh), pitch(m.tsc, m.tsh), fmut(mean), fmut(rstd), ptr(y), ptr(ty), ptr(g), ptr(gt),
                                 ptr(dx), ptr(dtx), sums, (int)x.size(0), (int)x.size(1), (int)x.size(2), (float)a.eps, (int)a.exact,
                                 code(x), stream_of(x)),
        "jvpattn_ln_modulate_dual");
}

// -> y, ty (undefined unless `dual`), mean, rstd; `a.x` and `a.tx` contiguous
std::array<Tensor, 4> ln_forward(const LnInputs &a, bool dual) {
  c10::cuda::CUDAGuard guard(a.x.device());
  Tensor y = at::empty_like(a.x), ty = dual ? at::empty_like(a.x) : Tensor();
  Tensor stats = at::empty({2, a.x.size(0) * a.x.size(1)}, a.x.options().dtype(at::kFloat));
  const Tensor mean = stats[0], rstd = stats[1];
  const LnRows m(a);
  if (!dual) {
    LnRows primal = m;
    primal.tsh = primal.tsc = Tensor();
    ln_launch(0, a, primal, {}, mean, rstd, y, {}, {}, {}, nullptr, a.exact);
  } else if (a.x.scalar_type() == at::kBFloat16) {
    ln_dual_launch(0, a, m, mean, rstd, y, ty, {}, {}, {}, {}, nullptr);
  } else {
    LnRows primal = m, tangent = m;
    primal.tsh = primal.tsc = tangent.sh = Tensor();
    ln_launch(0, a, primal, {}, mean, rstd, y, {}, {}, {}, nullptr, a.exact);
    ln_launch(1, a, tangent, a.tx.defined() ? a.tx : at::zeros_like(a.x), mean, rstd, ty, {}, {}, {}, nullptr, a.exact);
  }
  return {y, ty, mean, rstd};
}

// -> dx, d_gamma, d_beta, d_shift, d_scale, dtx, d_tshift, d_tscale
std::array<Tensor, 8> ln_backward(const LnInputs &a, const Tensor &mean, const Tensor &rstd, const Tensor &gy, const Tensor &gty) {
  c10::cuda::CUDAGuard guard(a.x.device());
  const int64_t B = a.x.size(0), C = a.x.size(2), nsum = gty.defined() ? 5 : 2;
  std::array<Tensor, 8> d;
  d[0] = at::empty_like(a.x);
  if (gty.defined()) d[5] = at::empty_like(a.x);
  // one fill for everything that is added to
  Tensor zeros = at::zeros({nsum * B * C + 2 * C}, a.x.options().dtype(at::kFloat));
  float *sums = zeros.data_ptr<float>();
  Tensor params = zeros.narrow(0, nsum * B * C, 2 * C).view({2, C});
  LnRows m(a);
  m.sh = m.tsh = Tensor();
  float *sums_y = gy.defined() ? sums : nullptr, *sums_ty = gty.defined() ? sums + 2 * B * C : nullptr;
  if (gy.defined() && gty.defined() && a.x.scalar_type() == at::kBFloat16) {
    ln_dual_launch(1, a, m, mean, rstd, {}, {}, gy, gty, d[0], d[5], sums);
  } else {
    LnRows primal = m;
    primal.tsc = Tensor();
    if (gy.defined()) ln_launch(2, a, primal, {}, mean, rstd, {}, gy, d[0], {}, sums_y, a.exact);
    if (gty.defined())
      ln_launch(3, a, m, a.tx.defined() ? a.tx : at::zeros_like(a.x), mean, rstd, {}, gty, d[0], d[5], sums_ty,
                (int)a.exact | (gy.defined() ? 2 : 0));
  }
  const auto fresh = at::TensorOptions(a.scale.options());
  if (gy.defined()) d[3] = at::empty({B, C}, fresh);
  d[4] = at::empty({B, C}, fresh);
  if (gty.defined() && a.tshift.defined()) d[6] = at::empty({B, C}, fresh);
  if (gty.defined() && a.tscale.defined()) d[7] = at::empty({B, C}, fresh);
  d[1] = params[0];
  if (a.beta.defined()) d[2] = params[1];
  check(jvpattn_ln_finalize(sums_y, sums_ty, fptr(a.gamma), fptr(a.beta), ptr(m.sc), ptr(m.tsc), pitch(m.sc, {}), pitch(m.tsc, {}), ptr(d[3]),
                            ptr(d[4]), ptr(d[6]), ptr(d[7]), fmut(d[1]), fmut(d[2]), (int)B, (int)C, code(a.x), stream_of(a.x)),
        "jvpattn_ln_finalize");
  auto shaped = [](Tensor &t, const Tensor &like) {
    if (t.defined()) t = t.reshape(like.sizes());
  };
  shaped(d[3], a.shift), shaped(d[4], a.scale), shaped(d[6], a.tshift), shaped(d[7], a.tscale);
  if (!a.tx.defined()) d[5] = Tensor();
  return d;
}

struct LnPair : Function<LnPair> {
  static variable_list forward(AutogradContext *ctx, const Tensor &x, const Tensor &gamma, const Opt &beta, const Tensor &shift,
                               const Tensor &scale, const Opt &tx, const Opt &tshift, const Opt &tscale, double eps, bool exact, bool dual) {
    at::AutoDispatchBelowADInplaceOrView below;
    const LnInputs a{dense(x), dense(value(tx)), gamma, value(beta), shift, scale, value(tshift), value(tscale), eps, exact};
    auto [y, ty, mean, rstd] = ln_forward(a, dual);
    ctx->save_for_backward({a.x, a.tx, a.gamma, a.beta, a.shift, a.scale, a.tshift, a.tscale, mean, rstd});
    ctx->set_materialize_grads(false);
    ctx->saved_data["eps"] = eps;
    ctx->saved_data["exact"] = exact;
    return dual ? variable_list{y, ty} : variable_list{y};
  }
  static variable_list backward(AutogradContext *ctx, const variable_list &g) {
    const Tensor gy = g[0], gty = g.size() > 1 ? g[1] : Tensor();
    if (!gy.defined() && !gty.defined()) return variable_list(11);
    const auto s = ctx->get_saved_variables();
    std::array<Tensor, 8> d;
    {
      at::AutoDispatchBelowADInplaceOrView below;
      at::NoGradGuard off;
      const LnInputs a{s[0], s[1], s[2], s[3], s[4], s[5], s[6], s[7], ctx->saved_data["eps"].toDouble(), ctx->saved_data["exact"].toBool()};
      d = ln_backward(a, s[8], s[9], dense(gy), dense(gty));
    }
    return once(g, {d[0], d[1], d[2], d[3], d[4], d[5], d[6], d[7], Tensor(), Tensor(), Tensor()});
  }
};

std::tuple<Tensor, Tensor> ln_pair(const Tensor &x, const Tensor &gamma, const Opt &beta, const Tensor &shift, const Tensor &scale, const Opt &tx,
                                   const Opt &tshift, const Opt &tscale, double eps, bool exact) {
  const LnInputs a{dense(x), dense(value(tx)), gamma, value(beta), shift, scale, value(tshift), value(tscale), eps, exact};
  auto out = ln_forward(a, true);
  return {out[0], out[1]};
}
std::tuple<Tensor, Tensor> ln_pair_autograd(const Tensor &x, const Tensor &gamma, const Opt &beta, const Tensor &shift, const Tensor &scale,
                                            const Opt &tx, const Opt &tshift, const Opt &tscale, double eps, bool exact) {
  const Tensor b = value(beta), t[3] = {value(tx), value(tshift), value(tscale)};
  if (any_grad({&x, &gamma, &b, &shift, &scale, &t[0], &t[1], &t[2]})) {
    auto out = LnPair::apply(x, gamma, beta, shift, scale, tx, tshift, tscale, eps, exact, true);
    return {out[0], out[1]};
  }
  at::AutoDispatchBelowADInplaceOrView below;
  return ln_pair(x, gamma, beta, shift, scale, tx, tshift, tscale, eps, exact);
}
Tensor ln_primal(const Tensor &x, const Tensor &gamma, const Opt &beta, const Tensor &shift, const Tensor &scale, double eps, bool exact) {
  return ln_forward({dense(x), {}, gamma, value(beta), shift, scale, {}, {}, eps, exact}, false)[0];
}
Tensor ln_primal_autograd(const Tensor &x, const Tensor &gamma, const Opt &beta, const Tensor &shift, const Tensor &scale, double eps,
                          bool exact) {
  const Tensor b = value(beta);
  if (any_grad({&x, &gamma, &b, &shift, &scale}))
    return LnPair::apply(x, gamma, beta, shift, scale, Opt(), Opt(), Opt(), eps, exact, false)[0];
  at::AutoDispatchBelowADInplaceOrView below;
  return ln_primal(x, gamma, beta, shift, scale, eps, exact);
}

// ------------------------------------------------------------------------------------------------ gated residual
struct GateInputs {
  Tensor x, y, gate, seed, tx, ty, tgate;
  int64_t call;
  double p;
  jvpattn_dropout drop() const { return {static_cast<const uint64_t *>(ptr(seed)), (uint32_t)call, (float)p}; }
};

void gate_dual_launch(int which, const GateInputs &a, const Tensor &z, const Tensor &tz, const Tensor &gz, const Tensor &gtz, const Tensor &dy,
                      const Tensor &dty, const Tensor &sums) {
  const Tensor g = mod_rows(a.gate), tg = mod_rows(a.tgate);
  const jvpattn_dropout drop = a.drop();
  const Tensor &y = a.y;
  check(jvpattn_gated_residual_dual(which, ptr(a.x), ptr(a.tx), ptr(y), ptr(a.ty), ptr(g), ptr(tg), nullptr, pitch(g, {}), pitch(tg, {}), ptr(z),
                                    ptr(tz), ptr(gz), ptr(gtz), ptr(dy), ptr(dty), fmut(sums), (int)y.size(0), (int)y.size(1), (int)y.size(2),
                                    code(y), a.seed.defined() ? &drop : nullptr, stream_of(y)),
        "jvpattn_gated_residual_dual");
}

std::array<Tensor, 2> gate_forward(const GateInputs &a, bool dual) {
  c10::cuda::CUDAGuard guard(a.y.device());
  Tensor z = at::empty_like(a.y), tz;
  if (dual) {
    tz = at::empty_like(a.y);
    gate_dual_launch(0, a, z, tz, {}, {}, {}, {}, {});
  } else {
    const Tensor g = mod_rows(a.gate);
    const jvpattn_dropout drop = a.drop();
    check(jvpattn_gated_residual(ptr(a.x), ptr(a.y), ptr(g), nullptr, pitch(g, {}), ptr(z), (int)a.y.size(0), (int)a.y.size(1),
                                 (int)a.y.size(2), code(a.y), a.seed.defined() ? &drop : nullptr, stream_of(a.y)),
          "jvpattn_gated_residual");
  }
  return {z, tz};
}

struct GatePair : Function<GatePair> {
  static variable_list forward(AutogradContext *ctx, const Tensor &x, const Tensor &y, const Tensor &gate, const Opt &seed, const Opt &tx,
                               const Opt &ty, const Opt &tgate, int64_t call, double p, bool dual) {
    at::AutoDispatchBelowADInplaceOrView below;
    const GateInputs a{dense(x), dense(y), gate, value(seed), dense(value(tx)), dense(value(ty)), value(tgate), call, p};
    auto [z, tz] = gate_forward(a, dual);
    ctx->save_for_backward({a.y, a.gate, a.seed, a.ty, a.tgate});
    ctx->set_materialize_grads(false);
    ctx->saved_data["call"] = call;
    ctx->saved_data["p"] = p;
    ctx->saved_data["has_tx"] = a.tx.defined();
    return dual ? variable_list{z, tz} : variable_list{z};
  }
  static variable_list backward(AutogradContext *ctx, const variable_list &g) {
    if (!g[0].defined() && !(g.size() > 1 && g[1].defined())) return variable_list(10);
    const auto s = ctx->get_saved_variables();
    variable_list d(10);
    {
      at::AutoDispatchBelowADInplaceOrView below;
      at::NoGradGuard off;
      const Tensor gz = dense(g[0]), gtz = g.size() > 1 ? dense(g[1]) : Tensor();
      const GateInputs a{{}, s[0], s[1], s[2], {}, s[3], s[4], ctx->saved_data["call"].toInt(), ctx->saved_data["p"].toDouble()};
      c10::cuda::CUDAGuard guard(a.y.device());
      Tensor dy = at::empty_like(a.y), dty = gtz.defined() ? at::empty_like(a.y) : Tensor();
      Tensor sums = at::zeros({2, a.y.size(0), a.y.size(2)}, a.y.options().dtype(at::kFloat));
      gate_dual_launch(1, a, {}, {}, gz, gtz, dy, dty, sums);
      d[0] = gz;
      d[1] = dy;
      d[2] = sums[0].to(a.gate.scalar_type()).reshape(a.gate.sizes());
      if (ctx->saved_data["has_tx"].toBool()) d[4] = gtz;
      if (a.ty.defined()) d[5] = dty;
      if (a.tgate.defined() && gtz.defined()) d[6] = sums[1].to(a.tgate.scalar_type()).reshape(a.tgate.sizes());
    }
    return once(g, d);
  }
};

std::tuple<Tensor, Tensor> gate_pair(const Tensor &x, const Tensor &y, const Tensor &gate, const Opt &seed, const Opt &tx, const Opt &ty,
                                     const Opt &tgate, int64_t call, double p) {
  auto out = gate_forward({dense(x), dense(y), gate, value(seed), dense(value(tx)), dense(value(ty)), value(tgate), call, p}, true);
  return {out[0], out[1]};
}
std::tuple<Tensor, Tensor> gate_pair_autograd(const Tensor &x, const Tensor &y, const Tensor &gate, const Opt &seed, const Opt &tx,
                                              const Opt &ty, const Opt &tgate, int64_t call, double p) {
  const Tensor t[3] = {value(tx), value(ty), value(tgate)};
  if (any_grad({&x, &y, &gate, &t[0], &t[1], &t[2]})) {
    auto out = GatePair::apply(x, y, gate, seed, tx, ty, tgate, call, p, true);
    return {out[0], out[1]};
  }
  at::AutoDispatchBelowADInplaceOrView below;
  return gate_pair(x, y, gate, seed, tx, ty, tgate, call, p);
}
Tensor gate_primal(const Tensor &x, const Tensor &y, const Tensor &gate, const Opt &seed, int64_t call, double p) {
  return gate_forward({dense(x), dense(y), gate, value(seed), {}, {}, {}, call, p}, false)[0];
}
Tensor gate_primal_autograd(const Tensor &x, const Tensor &y, const Tensor &gate, const Opt &seed, int64_t call, double p) {
  if (any_grad({&x, &y, &gate})) return GatePair::apply(x, y, gate, seed, Opt(), Opt(), Opt(), call, p, false)[0];
  at::AutoDispatchBelowADInplaceOrView below;
  return gate_primal(x, y, gate, seed, call, p);
}

// ------------------------------------------------------------------------------------------------ GELU (tanh form)
void gelu_launch(int mode, const Tensor &h, const Tensor &v, const Tensor &w, const Tensor &u, const Tensor &out, const Tensor &out2) {
  c10::cuda::CUDAGuard guard(h.device());
  check(jvpattn_gelu_dual(mode, ptr(h), ptr(v), ptr(w), ptr(u), ptr(out), ptr(out2), h.numel(), code(h), stream_of(h)), "jvpattn_gelu_dual");
}

std::tuple<Tensor, Tensor> gelu_pair(const Tensor &h, const Tensor &th_) {
  const Tensor th = th_._is_zerotensor() ? at::zeros_like(h) : th_.contiguous();
  Tensor y = at::empty_like(h), ty = at::empty_like(h);
  gelu_launch(3, h, th, {}, {}, y, ty);
  return {y, ty};
}
Tensor gelu_primal(const Tensor &h) {
  Tensor y = at::empty_like(h);
  gelu_launch(0, h, {}, {}, {}, y, {});
  return y;
}

struct GeluPair : Function<GeluPair> {
  static variable_list forward(AutogradContext *ctx, const Tensor &h, const Opt &th) {
    at::AutoDispatchBelowADInplaceOrView below;
    ctx->set_materialize_grads(false);
    if (!th.has_value()) {
      ctx->save_for_backward({h, Tensor()});
      return {gelu_primal(h)};
    }
    auto [y, ty] = gelu_pair(h, *th);
    ctx->save_for_backward({h, th->_is_zerotensor() ? at::zeros_like(h) : *th});
    return {y, ty};
  }
  static variable_list backward(AutogradContext *ctx, const variable_list &g) {
    const Tensor gy = g[0], gty = g.size() > 1 ? g[1] : Tensor();
    if (!gy.defined() && !gty.defined()) return variable_list(2);
    const auto s = ctx->get_saved_variables();
    const Tensor h = s[0], th = s[1];
    variable_list d(2);
    {
      at::AutoDispatchBelowADInplaceOrView below;
      at::NoGradGuard off;
      d[0] = at::empty_like(h);
      if (gty.defined()) d[1] = at::empty_like(h);
      if (!gty.defined()) gelu_launch(1, h, gy.contiguous(), {}, {}, d[0], {});
      else if (!gy.defined()) gelu_launch(2, h, gty.contiguous(), th.contiguous(), {}, d[1], d[0]);
      else gelu_launch(4, h, gy.contiguous(), th.contiguous(), gty.contiguous(), d[0], d[1]);
    }
    return once(g, d);
  }
};

std::tuple<Tensor, Tensor> gelu_pair_autograd(const Tensor &h, const Tensor &th) {
  if (any_grad({&h, &th})) {
    auto out = GeluPair::apply(h, Opt(th));
    return {out[0], out[1]};
  }
  at::AutoDispatchBelowADInplaceOrView below;
  return gelu_pair(h, th);
}
Tensor gelu_primal_autograd(const Tensor &h) {
  if (any_grad({&h})) return GeluPair::apply(h, Opt())[0];
  at::AutoDispatchBelowADInplaceOrView below;
  return gelu_primal(h);
}

// ------------------------------------------------------------------------------------------------ linear layer
std::tuple<Tensor, Tensor> linear_pair(const Tensor &x, const Tensor &tx, const Tensor &w, const Opt &b) {
  return {at::linear(x, w, b), at::linear(tx, w)};
}

// The sum of a matrix over its rows: by the library's kernel for plain bf16 values, by torch's reduction for whatever else a backward
// pass may be given (batched, dual or recorded cotangents, other types), and for a single row or 8 columns, where that is faster
// (1 x 768 2.3 against 2.7 us; 262144 x 8 10.4 against 12.8, of 16 columns 14.5 against 13.1).
Tensor column_sum(const Tensor &g) {
  const auto keys = g.key_set();
  if (g.scalar_type() != at::kBFloat16 || !g.is_cuda() || g.layout() != at::kStrided || keys.has(c10::DispatchKey::Python) ||
      keys.has(c10::DispatchKey::Functionalize) || keys.has(c10::DispatchKey::FuncTorchBatched) || keys.has(c10::DispatchKey::Batched) ||
      keys.has(c10::DispatchKey::FuncTorchGradWrapper) || !g.has_storage() || g.is_neg() || c10::impl::TorchDispatchModeTLS::any_modes_set() ||
      (at::GradMode::is_enabled() && g.requires_grad()) || g._fw_grad(0).defined() || g.size(1) % 8 || g.size(0) < 2 || g.size(1) < 16 || g.stride(1) != 1 ||
      g.stride(0) % 8 || g.stride(0) < g.size(1) || (g.storage_offset() * 2) % 16)
    return g.sum(0);
  at::AutoDispatchBelowADInplaceOrView below;
  c10::cuda::CUDAGuard guard(g.device());
  Tensor out = at::empty({g.size(1)}, g.options());
  const int64_t bytes = jvpattn_column_sum_workspace_bytes(g.size(0), (int)g.size(1));
  const Tensor workspace = at::empty({bytes}, g.options().dtype(at::kByte));
  check(jvpattn_column_sum(ptr(g), g.size(0), (int)g.size(1), g.stride(0), ptr(out), JVPATTN_BF16, ptr(workspace), bytes, stream_of(g)), "jvpattn_column_sum");
  return out;
}

// Without a tangent: torch's own layer, but for the gradient of the bias.  (Differentiable again, as torch's is.)
struct LinearPrimal : Function<LinearPrimal> {
  static Tensor forward(AutogradContext *ctx, const Tensor &x, const Tensor &w, const Tensor &b) {
    at::AutoDispatchBelowADInplaceOrView below;
    // (only what the backward reads: the rest may be freed, or written to)
    ctx->save_for_backward({w.requires_grad() ? x : Tensor(), x.requires_grad() ? w : Tensor()});
    ctx->saved_data["x"] = x.sizes().vec();
    return at::linear(x, w, b);
  }
  static variable_list backward(AutogradContext *ctx, const variable_list &g) {
    const auto s = ctx->get_saved_variables();
    const std::vector<int64_t> shape = ctx->saved_data["x"].toIntVector();
    const Tensor x = s[0], w = s[1], g2 = g[0].reshape({-1, g[0].size(-1)});
    variable_list d(3);
    if (ctx->needs_input_grad(0)) d[0] = at::mm(g2, w).view(shape);
    if (ctx->needs_input_grad(1)) d[1] = at::mm(g2.t(), x.reshape({-1, shape.back()}));
    if (ctx->needs_input_grad(2)) d[2] = column_sum(g2);
    return d;
  }
};

// Two GEMMs forward; backward two for dx / dtx, two for dw (the second adds to the first in its epilogue), one reduction for db.
struct LinearPair : Function<LinearPair> {
  static variable_list forward(AutogradContext *ctx, const Tensor &x, const Tensor &tx_, const Tensor &w, const Opt &b) {
    at::AutoDispatchBelowADInplaceOrView below;
    const Tensor tx = tx_._is_zerotensor() ? at::zeros_like(x) : tx_;
    auto [y, ty] = linear_pair(x, tx, w, b);
    ctx->save_for_backward({x, tx, w});
    ctx->saved_data["bias"] = b.has_value() && b->defined();
    ctx->set_materialize_grads(false);
    return {y, ty};
  }
  static variable_list backward(AutogradContext *ctx, const variable_list &g) {
    const auto s = ctx->get_saved_variables();
    const Tensor x = s[0], tx = s[1], w = s[2];
    variable_list d(4);
    {
      at::AutoDispatchBelowADInplaceOrView below;
      at::NoGradGuard off;
      const int64_t K = w.size(1), N = w.size(0);
      if (g[0].defined()) {
        const Tensor g2 = g[0].reshape({-1, N});
        if (ctx->needs_input_grad(0)) d[0] = at::mm(g2, w).view(x.sizes());
        if (ctx->needs_input_grad(2)) d[2] = at::mm(g2.t(), x.reshape({-1, K}));
        if (ctx->saved_data["bias"].toBool() && ctx->needs_input_grad(3)) d[3] = column_sum(g2);
      }
      if (g[1].defined()) {
        const Tensor t2 = g[1].reshape({-1, N});
        if (ctx->needs_input_grad(1)) d[1] = at::mm(t2, w).view(tx.sizes());
        if (ctx->needs_input_grad(2))
          d[2] = d[2].defined() ? at::addmm(d[2], t2.t(), tx.reshape({-1, K})) : at::mm(t2.t(), tx.reshape({-1, K}));
      }
    }
    return once(g, d);
  }
};

std::tuple<Tensor, Tensor> linear_pair_autograd(const Tensor &x, const Tensor &tx, const Tensor &w, const Opt &b) {
  const Tensor bias = value(b);
  if (any_grad({&x, &tx, &w, &bias})) {
    auto out = LinearPair::apply(x, tx, w, b);
    return {out[0], out[1]};
  }
  at::AutoDispatchBelowADInplaceOrView below;
  return linear_pair(x, tx, w, b);
}

// ------------------------------------------------------------------------------------------------ rotary embedding
void rotary_launch(const std::array<Tensor, 3> &in, const std::array<Tensor, 3> &out, const Tensor &cos, const Tensor &sin, bool transpose) {
  const void *ip[3];
  void *op[3];
  int64_t is[9], os[9];
  for (int t = 0; t < 3; ++t) {
    ip[t] = in[t].data_ptr(), op[t] = out[t].data_ptr();
    for (int k = 0; k < 3; ++k) is[3 * t + k] = in[t].stride(k), os[3 * t + k] = out[t].stride(k);
  }
  c10::cuda::CUDAGuard guard(in[0].device());
  check(jvpattn_rotary_qkv(ip, is, code(in[0]), op, os, code(out[0]), cos.data_ptr<float>(), sin.data_ptr<float>(), (int)in[0].size(0),
                           (int)in[0].size(1), (int)in[0].size(2), (int)in[0].size(3), transpose, stream_of(in[0])),
        "jvpattn_rotary_qkv");
}
std::array<Tensor, 3> thirds(const Tensor &qkv) { return {qkv.select(2, 0), qkv.select(2, 1), qkv.select(2, 2)}; }

std::array<Tensor, 3> rotary_split(const Tensor &qkv, const Tensor &cos, const Tensor &sin, at::ScalarType dtype) {
  std::array<Tensor, 3> out;
  for (Tensor &t : out) t = at::empty({qkv.size(0), qkv.size(1), qkv.size(3), qkv.size(4)}, qkv.options().dtype(dtype));
  rotary_launch(thirds(qkv), out, cos, sin, false);
  return out;
}
// (dq, dk, dv) -> the gradient of the (B, S, 3, H, D) projection, written in place by one launch
Tensor rotary_merge(std::array<Tensor, 3> g, at::IntArrayRef shape, at::ScalarType dtype, const Tensor &cos, const Tensor &sin) {
  const Tensor &any = g[0].defined() ? g[0] : g[1].defined() ? g[1] : g[2];
  if (!any.defined()) return {};
  const auto options = any.options().dtype(dtype);
  for (Tensor &t : g) t = !t.defined() ? at::zeros({shape[0], shape[1], shape[3], shape[4]}, options) : unit(t);
  const at::ScalarType first = g[0].scalar_type();
  if (g[1].scalar_type() != first || g[2].scalar_type() != first || (first != at::kBFloat16 && first != at::kFloat))
    for (Tensor &t : g) t = t.to(dtype);
  Tensor d = at::empty(shape, options);
  rotary_launch(g, thirds(d), cos, sin, true);
  return d;
}

struct RotaryPair : Function<RotaryPair> {
  static variable_list forward(AutogradContext *ctx, const Tensor &qkv, const Opt &tqkv, const Tensor &cos, const Tensor &sin, int64_t dtype) {
    at::AutoDispatchBelowADInplaceOrView below;
    const auto out_type = (at::ScalarType)dtype;
    auto p = rotary_split(qkv, cos, sin, out_type);
    variable_list out(p.begin(), p.end());
    if (tqkv.has_value()) {
      auto t = rotary_split(tqkv->_is_zerotensor() ? at::zeros_like(qkv) : *tqkv, cos, sin, out_type);
      out.insert(out.end(), t.begin(), t.end());
    }
    // (constants of the op: read again in the backward, never differentiated)
    ctx->saved_data["cos"] = cos;
    ctx->saved_data["sin"] = sin;
    ctx->saved_data["shape"] = qkv.sizes().vec();
    ctx->saved_data["dtype"] = (int64_t)qkv.scalar_type();
    ctx->set_materialize_grads(false);
    return out;
  }
  static variable_list backward(AutogradContext *ctx, const variable_list &g) {
    const Tensor cos = ctx->saved_data["cos"].toTensor(), sin = ctx->saved_data["sin"].toTensor();
    const std::vector<int64_t> shape = ctx->saved_data["shape"].toIntVector();
    const auto dtype = (at::ScalarType)ctx->saved_data["dtype"].toInt();
    variable_list d(5);
    {
      at::AutoDispatchBelowADInplaceOrView below;
      at::NoGradGuard off;
      d[0] = rotary_merge({g[0], g[1], g[2]}, shape, dtype, cos, sin);
      if (g.size() > 3) d[1] = rotary_merge({g[3], g[4], g[5]}, shape, dtype, cos, sin);
    }
    return once(g, d);
  }
};

std::vector<Tensor> rotary_pair(const Tensor &qkv, const Opt &tqkv, const Tensor &cos, const Tensor &sin, int64_t dtype) {
  auto p = rotary_split(qkv, cos, sin, (at::ScalarType)dtype);
  std::vector<Tensor> out(p.begin(), p.end());
  if (tqkv.has_value()) {
    auto t = rotary_split(tqkv->_is_zerotensor() ? at::zeros_like(qkv) : *tqkv, cos, sin, (at::ScalarType)dtype);
    out.insert(out.end(), t.begin(), t.end());
  }
  return out;
}
std::vector<Tensor> rotary_pair_autograd(const Tensor &qkv, const Opt &tqkv, const Tensor &cos, const Tensor &sin, int64_t dtype) {
  const Tensor t = tqkv.value_or(Tensor());
  if (any_grad({&qkv, &t})) return RotaryPair::apply(qkv, tqkv, cos, sin, dtype);
  at::AutoDispatchBelowADInplaceOrView below;
  return rotary_pair(qkv, tqkv, cos, sin, dtype);
}

// ------------------------------------------------------------------------------------------------ under torch.func.jvp
// (Of the op that F implements: one per function, since several have the same signature.)
template <auto *F>
const auto &handle(const char *name) {
  static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow(name, "").typed<std::remove_pointer_t<decltype(F)>>();
  return op;
}
Opt tangent(const Tensor &t) { return opt(t._fw_grad(/*level=*/0)); }
Tensor dual(const Tensor &y, const Tensor &ty) {
  y._set_fw_grad(ty, /*level=*/0, /*is_inplace_op=*/false);
  return y;
}

Tensor attention_jvp(const Tensor &q, const Tensor &k, const Tensor &v, bool bshd) {
  const Opt tq = tangent(q), tk = tangent(k), tv = tangent(v);
  std::tuple<Tensor, Tensor> out;
  {
    at::AutoDispatchBelowADInplaceOrView below;  // the op leaves the transform's level here
    if (!tq && !tk && !tv) return handle<attention_primal>("jvpattn::attention_primal").call(q, k, v, bshd);
    out = handle<attention_pair>("jvpattn::attention_pair").call(q, k, v, tq, tk, tv, bshd);
  }
  return dual(std::get<0>(out), std::get<1>(out));
}
Tensor ln_jvp(const Tensor &x, const Tensor &gamma, const Opt &beta, const Tensor &shift, const Tensor &scale, double eps, bool exact) {
  const Opt tx = tangent(x), tsh = tangent(shift), tsc = tangent(scale);
  std::tuple<Tensor, Tensor> out;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    if (!tx && !tsh && !tsc) return handle<ln_primal>("jvpattn::ln_primal").call(x, gamma, beta, shift, scale, eps, exact);
    out = handle<ln_pair>("jvpattn::ln_pair").call(x, gamma, beta, shift, scale, tx, tsh, tsc, eps, exact);
  }
  return dual(std::get<0>(out), std::get<1>(out));
}
Tensor gate_jvp(const Tensor &x, const Tensor &y, const Tensor &gate, const Opt &seed, int64_t call, double p) {
  const Opt tx = tangent(x), ty = tangent(y), tg = tangent(gate);
  std::tuple<Tensor, Tensor> out;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    if (!tx && !ty && !tg) return handle<gate_primal>("jvpattn::gate_primal").call(x, y, gate, seed, call, p);
    out = handle<gate_pair>("jvpattn::gate_pair").call(x, y, gate, seed, tx, ty, tg, call, p);
  }
  return dual(std::get<0>(out), std::get<1>(out));
}
Tensor gelu_jvp(const Tensor &h) {
  const Opt th = tangent(h);
  std::tuple<Tensor, Tensor> out;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    if (!th) return handle<gelu_primal>("jvpattn::gelu_primal").call(h);
    out = handle<gelu_pair>("jvpattn::gelu_pair").call(h, *th);
  }
  return dual(std::get<0>(out), std::get<1>(out));
}
Tensor linear_jvp(const Tensor &x, const Tensor &w, const Opt &b) {
  const Opt tx = tangent(x);
  std::tuple<Tensor, Tensor> out;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    out = handle<linear_pair>("jvpattn::linear_pair").call(x, *tx, w, b);
  }
  return dual(std::get<0>(out), std::get<1>(out));
}
std::vector<Tensor> rotary_jvp(const Tensor &qkv, const Tensor &cos, const Tensor &sin, int64_t dtype) {
  const Opt t = tangent(qkv);
  std::vector<Tensor> out;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    out = handle<rotary_pair>("jvpattn::rotary_pair").call(qkv, t, cos, sin, dtype);
  }
  if (!t) return out;
  return {dual(out[0], out[3]), dual(out[1], out[4]), dual(out[2], out[5])};
}

TORCH_LIBRARY(jvpattn, m) {
  m.def("attention(Tensor q, Tensor k, Tensor v, bool bshd) -> Tensor", attention_jvp);
  m.def("attention_pair(Tensor q, Tensor k, Tensor v, Tensor? tq, Tensor? tk, Tensor? tv, bool bshd) -> (Tensor, Tensor)");
  m.def("attention_primal(Tensor q, Tensor k, Tensor v, bool bshd) -> Tensor");
  m.def("ln(Tensor x, Tensor gamma, Tensor? beta, Tensor shift, Tensor scale, float eps, bool exact) -> Tensor", ln_jvp);
  m.def("ln_pair(Tensor x, Tensor gamma, Tensor? beta, Tensor shift, Tensor scale, Tensor? tx, Tensor? tshift, Tensor? tscale, "
        "float eps, bool exact) -> (Tensor, Tensor)");
  m.def("ln_primal(Tensor x, Tensor gamma, Tensor? beta, Tensor shift, Tensor scale, float eps, bool exact) -> Tensor");
  m.def("gate(Tensor x, Tensor y, Tensor gate, Tensor? seed, int call, float p) -> Tensor", gate_jvp);
  m.def("gate_pair(Tensor x, Tensor y, Tensor gate, Tensor? seed, Tensor? tx, Tensor? ty, Tensor? tgate, int call, float p) -> "
        "(Tensor, Tensor)");
  m.def("gate_primal(Tensor x, Tensor y, Tensor gate, Tensor? seed, int call, float p) -> Tensor");
  m.def("gelu(Tensor h) -> Tensor", gelu_jvp);
  m.def("gelu_pair(Tensor h, Tensor th) -> (Tensor, Tensor)");
  m.def("gelu_primal(Tensor h) -> Tensor");
  m.def("linear(Tensor x, Tensor w, Tensor? b) -> Tensor", linear_jvp);
  m.def("linear_pair(Tensor x, Tensor tx, Tensor w, Tensor? b) -> (Tensor, Tensor)");
  m.def("rotary(Tensor qkv, Tensor cos, Tensor sin, int dtype) -> Tensor[]", rotary_jvp);
  m.def("rotary_pair(Tensor qkv, Tensor? tqkv, Tensor cos, Tensor sin, int dtype) -> Tensor[]");
}
TORCH_LIBRARY_IMPL(jvpattn, Autograd, m) {
  m.impl("attention_pair", attention_pair_autograd);
  m.impl("attention_primal", attention_primal_autograd);
  m.impl("ln_pair", ln_pair_autograd);
  m.impl("ln_primal", ln_primal_autograd);
  m.impl("gate_pair", gate_pair_autograd);
  m.impl("gate_primal", gate_primal_autograd);
  m.impl("gelu_pair", gelu_pair_autograd);
  m.impl("gelu_primal", gelu_primal_autograd);
  m.impl("linear_pair", linear_pair_autograd);
  m.impl("rotary_pair", rotary_pair_autograd);
}
TORCH_LIBRARY_IMPL(jvpattn, CUDA, m) {
  m.impl("attention_pair", attention_pair);
  m.impl("attention_primal", attention_primal);
  m.impl("ln_pair", ln_pair);
  m.impl("ln_primal", ln_primal);
  m.impl("gate_pair", gate_pair);
  m.impl("gate_primal", gate_primal);
  m.impl("gelu_pair", gelu_pair);
  m.impl("gelu_primal", gelu_primal);
  m.impl("linear_pair", linear_pair);
  m.impl("rotary_pair", rotary_pair);
}

// ------------------------------------------------------------------------------------------------ entry from Python
namespace py = pybind11;

// A tensor as given from Python: undefined where it is None; `exact` is false for anything but Tensor and Parameter.
struct Arg {
  Tensor t;
  bool ok;
  explicit Arg(py::handle h) : ok(h.is_none() || THPVariable_CheckExact(h.ptr())) {
    if (ok && !h.is_none()) t = THPVariable_Unpack(h.ptr());
  }
};

// A tangent may be of another type or on another device than its primal (torch.func.jvp hands it on as given): the kernels read
// it with the primal's, so it must be a plain tensor of the same kind.
bool tangent_fits(const Tensor &t, const Tensor &p) {
  const auto keys = t.key_set();
  return t.scalar_type() == p.scalar_type() && t.device() == p.device() && t.layout() == at::kStrided && t.sizes() == p.sizes() &&
         !keys.has(c10::DispatchKey::Python) && !keys.has(c10::DispatchKey::Functionalize) && !keys.has(c10::DispatchKey::FuncTorchBatched) &&
         !t.is_conj() && !t.is_neg();
}

bool watched() {
  return c10::impl::TorchDispatchModeTLS::any_modes_set() || at::impl::torch_function_mode_enabled() || torch::jit::tracer::isTracing();
}

// `jvp`: one torch.func.jvp is open and no other transform; else none is.
bool fits(bool jvp, std::initializer_list<const Arg *> args) {
  if (watched()) return false;
  for (const Arg *a : args) {
    if (!a->ok) return false;
    if (!a->t.defined()) continue;
    const auto keys = a->t.key_set();
    if (!a->t.is_cuda() || a->t.layout() != at::kStrided || keys.has(c10::DispatchKey::Python) || keys.has(c10::DispatchKey::Functionalize) ||
        keys.has(c10::DispatchKey::FuncTorchBatched) || a->t.is_conj() || a->t.is_neg())
      return false;
    const Tensor &t = a->t._fw_grad(/*level=*/0);
    if (keys.has(c10::DispatchKey::FuncTorchGradWrapper)) {
      if (!jvp || a->t.requires_grad()) return false;  // (reverse mode inside the transform)
      if (t.defined() && !tangent_fits(t, a->t)) return false;
    } else if (t.defined()) {
      return false;  // a dual of a plain forward_ad level
    }
  }
  return true;
}

py::object attention_py(bool jvp, py::handle q_, py::handle k_, py::handle v_, bool bshd) {
  const Arg q(q_), k(k_), v(v_);
  if (!fits(jvp, {&q, &k, &v}) || !q.t.defined() || !k.t.defined() || !v.t.defined() || q.t.dim() != 4 || k.t.dim() != 4) return py::none();
  const int64_t D = q.t.size(3), h = bshd ? 2 : 1;
  const auto dt = q.t.scalar_type();
  if (v.t.sizes() != k.t.sizes() || k.t.size(0) != q.t.size(0) || k.t.size(h) != q.t.size(h) || k.t.size(3) != D || D < 16 || D > 128 ||
      (dt != at::kBFloat16 && dt != at::kHalf) || k.t.scalar_type() != dt || v.t.scalar_type() != dt || k.t.device() != q.t.device() ||
      v.t.device() != q.t.device())
    return py::none();
  if (jvp) return py::cast(handle<attention_jvp>("jvpattn::attention").call(q.t, k.t, v.t, bshd));
  return py::cast(attention_primal_autograd(q.t, k.t, v.t, bshd));
}

bool modulation_ok(const Tensor &m, const Tensor &x) {
  const int64_t B = x.size(0), C = x.size(2);
  return m.defined() && m.scalar_type() == x.scalar_type() && m.device() == x.device() &&
         ((m.dim() == 3 && m.size(0) == B && m.size(1) == 1 && m.size(2) == C) || (m.dim() == 2 && m.size(0) == B && m.size(1) == C));
}
bool rows_ok(const Tensor &x) {
  if (!x.defined() || x.dim() != 3 || (x.scalar_type() != at::kBFloat16 && x.scalar_type() != at::kFloat)) return false;
  const int64_t C = x.size(2);
  return C == 256 || C == 512 || C == 768 || C == 1024;
}

// (A parameter with a tangent of its own is refused by the classes: the terms it would add are not formed here.)
bool param_ok(const Tensor &p, const Tensor &x) {
  return !p._fw_grad(0).defined() && p.scalar_type() == at::kFloat && p.dim() == 1 && p.size(0) == x.size(2) && p.is_contiguous() && p.device() == x.device();
}

py::object ln_py(bool jvp, py::handle x_, py::handle w_, py::handle b_, py::handle shift_, py::handle scale_, double eps, bool exact) {
  const Arg x(x_), w(w_), b(b_), shift(shift_), scale(scale_);
  if (!fits(jvp, {&x, &w, &b, &shift, &scale}) || !rows_ok(x.t) || !modulation_ok(shift.t, x.t) || !modulation_ok(scale.t, x.t)) return py::none();
  if (!w.t.defined() || !param_ok(w.t, x.t) || (b.t.defined() && !param_ok(b.t, x.t))) return py::none();
  if (jvp)
    return py::cast(handle<ln_jvp>("jvpattn::ln").call(x.t, w.t, opt(b.t), shift.t, scale.t, eps, exact));
  return py::cast(ln_primal_autograd(x.t, w.t, opt(b.t), shift.t, scale.t, eps, exact));
}

py::object gate_py(bool jvp, py::handle x_, py::handle y_, py::handle gate_, py::handle seed_, int64_t call, double p) {
  const Arg x(x_), y(y_), gate(gate_), seed(seed_);
  if (!fits(jvp, {&x, &y, &gate, &seed}) || !rows_ok(y.t) || !x.t.defined() || x.t.sizes() != y.t.sizes() || x.t.scalar_type() != y.t.scalar_type() ||
      x.t.device() != y.t.device() || !modulation_ok(gate.t, y.t))
    return py::none();
  if (jvp) return py::cast(handle<gate_jvp>("jvpattn::gate").call(x.t, y.t, gate.t, opt(seed.t), call, p));
  return py::cast(gate_primal_autograd(x.t, y.t, gate.t, opt(seed.t), call, p));
}

// gated_residual and ln_modulate of its result, where nothing is recorded: (z, h).
py::object gate_ln_py(py::handle x_, py::handle y_, py::handle gate_, py::handle w_, py::handle b_, py::handle shift_, py::handle scale_,
                      double eps) {
  const Arg x(x_), y(y_), gate(gate_), w(w_), b(b_), shift(shift_), scale(scale_);
  if (!fits(false, {&x, &y, &gate, &w, &b, &shift, &scale}) || !rows_ok(y.t) || !x.t.defined() || x.t.sizes() != y.t.sizes() ||
      x.t.scalar_type() != y.t.scalar_type() || x.t.device() != y.t.device() || !modulation_ok(gate.t, y.t) || !modulation_ok(shift.t, y.t) ||
      !modulation_ok(scale.t, y.t) || !w.t.defined() || !param_ok(w.t, y.t) || (b.t.defined() && !param_ok(b.t, y.t)))
    return py::none();
  at::AutoDispatchBelowADInplaceOrView below;
  c10::cuda::CUDAGuard guard(y.t.device());
  const Tensor xc = dense(x.t), yc = dense(y.t), g = mod_rows(gate.t);
  Tensor sh = mod_rows(shift.t), sc = mod_rows(scale.t);
  equal_pitch(sh, sc);
  Tensor z = at::empty_like(yc), h = at::empty_like(yc);
  check(jvpattn_gate_ln(ptr(xc), ptr(yc), ptr(g), pitch(g, {}), fptr(w.t), fptr(b.t), ptr(sh), ptr(sc), pitch(sc, {}), ptr(z), ptr(h),
                        (int)yc.size(0), (int)yc.size(1), (int)yc.size(2), (float)eps, code(yc), stream_of(yc)),
        "jvpattn_gate_ln");
  return py::make_tuple(z, h);
}

py::object gelu_py(bool jvp, py::handle h_) {
  const Arg h(h_);
  if (!fits(jvp, {&h}) || !h.t.defined() || (h.t.scalar_type() != at::kBFloat16 && h.t.scalar_type() != at::kFloat) || !h.t.is_contiguous() ||
      h.t.numel() % 8 || (h.t.storage_offset() * h.t.element_size()) % 16)
    return py::none();
  if (jvp) return py::cast(handle<gelu_jvp>("jvpattn::gelu").call(h.t));
  return py::cast(gelu_primal_autograd(h.t));
}

// Without a tangent on x the layer is torch's own, but where a bf16 bias wants its gradient; with one on a parameter it is refused
// by the class.
py::object linear_py(bool jvp, py::handle x_, py::handle w_, py::handle b_) {
  const Arg x(x_), w(w_), b(b_);
  if (!fits(jvp, {&x, &w, &b}) || !x.t.defined() || !w.t.defined() ||
      (jvp && (!x.t._fw_grad(0).defined() || w.t._fw_grad(0).defined() || (b.t.defined() && b.t._fw_grad(0).defined()))))
    return py::none();
  const auto dt = x.t.scalar_type();
  if (w.t.scalar_type() != dt || w.t.dim() != 2 || (b.t.defined() && b.t.scalar_type() != dt) ||
      (at::autocast::is_autocast_enabled(at::kCUDA) && at::autocast::get_autocast_dtype(at::kCUDA) != dt))
    return py::none();
  if (!jvp) {
    if (dt != at::kBFloat16 || !b.t.defined() || !any_grad({&b.t}) || b.t.dim() != 1 || x.t.dim() < 2 || x.t.numel() == 0 || x.t.size(-1) != w.t.size(1) ||
        b.t.size(0) != w.t.size(0) || w.t.size(0) % 8 || w.t.device() != x.t.device() || b.t.device() != x.t.device())
      return py::none();
    return py::cast(LinearPrimal::apply(x.t, w.t, b.t));
  }
  return py::cast(handle<linear_jvp>("jvpattn::linear").call(x.t, w.t, opt(b.t)));
}

py::object rotary_py(bool jvp, py::handle qkv_, py::handle cos_, py::handle sin_, bool bf16) {
  const Arg qkv(qkv_), cos(cos_), sin(sin_);
  if (!fits(jvp, {&qkv, &cos, &sin}) || !qkv.t.defined() || qkv.t.dim() != 5 || qkv.t.size(2) != 3 || !cos.t.defined() || !sin.t.defined()) return py::none();
  const Tensor &x = qkv.t;
  auto layout_ok = [](const Tensor &t) {
    for (int i = 0; i < 4; ++i)
      if (t.stride(i) % 8) return false;
    return t.stride(4) == 1 && (t.storage_offset() * t.element_size()) % 16 == 0;
  };
  auto table_ok = [&](const Tensor &t) {
    return t.scalar_type() == at::kFloat && t.is_contiguous() && t.device() == x.device() && t.dim() == 2 && t.size(0) == x.size(1) &&
           t.size(1) * 2 == x.size(4) && !t.requires_grad() && !t._fw_grad(0).defined() && (t.storage_offset() * 4) % 16 == 0;
  };
  if ((x.scalar_type() != at::kBFloat16 && x.scalar_type() != at::kFloat) || x.size(4) % 16 || !layout_ok(x) || !table_ok(cos.t) || !table_ok(sin.t))
    return py::none();
  const Tensor &t = x._fw_grad(0);
  if (t.defined() && (t.strides() != x.strides() || !layout_ok(t))) return py::none();
  const int64_t dtype = (int64_t)(bf16 ? at::kBFloat16 : at::kFloat);
  const std::vector<Tensor> out = jvp ? handle<rotary_jvp>("jvpattn::rotary").call(x, cos.t, sin.t, dtype)
                                                   : rotary_pair_autograd(x, Opt(), cos.t, sin.t, dtype);
  return py::make_tuple(out[0], out[1], out[2]);
}

// 16-bit copies of contiguous fp32 CUDA parameters, side by side in one buffer (each from 16 bytes on): of a matrix as it is, or
// (`align`) with rows and columns padded to multiples of 8; times `scale`.  None where they are not all of that kind, and under a
// dispatch or function mode or a trace, which would not see the kernel's writes.
py::object cast_params(const std::vector<Tensor> &params, const std::vector<double> &scale, const std::vector<bool> &align, bool bf16) {
  if (params.empty() || scale.size() != params.size() || align.size() != params.size() || watched()) return py::none();
  const Tensor &p0 = params[0];
  std::vector<jvpattn_cast> e(params.size());
  std::vector<int64_t> offset(params.size());
  int64_t total = 0;
  for (size_t i = 0; i < params.size(); ++i) {
    const Tensor &p = params[i];
    if (!p.is_cuda() || p.device() != p0.device() || p.layout() != at::kStrided || p.scalar_type() != at::kFloat || p.dim() < 1 || p.dim() > 2 ||
        !p.is_contiguous() || p.key_set().has(c10::DispatchKey::Python) || p.size(0) > INT32_MAX - 8 || p.size(-1) > INT32_MAX - 8)
      return py::none();
    const int64_t rows = p.dim() == 2 ? p.size(0) : 1, cols = p.size(-1);
    const auto up = [&](int64_t n) { return align[i] ? (n + 7) / 8 * 8 : n; };
    e[i] = {p.data_ptr<float>(), nullptr, (int32_t)rows, (int32_t)cols, (int32_t)(p.dim() == 2 ? up(rows) : 1), (int32_t)up(cols), (float)scale[i]};
    offset[i] = total;
    total += ((int64_t)e[i].rows_out * e[i].cols_out + 7) / 8 * 8;
  }
  c10::cuda::CUDAGuard guard(p0.device());
  at::AutoDispatchBelowADInplaceOrView below;
  const Tensor flat = at::empty({total}, p0.options().dtype(bf16 ? at::kBFloat16 : at::kHalf));
  std::vector<Tensor> out(params.size());
  for (size_t i = 0; i < params.size(); ++i) {
    e[i].dst = static_cast<char *>(flat.data_ptr()) + 2 * offset[i];
    out[i] = params[i].dim() == 2 ? flat.as_strided({e[i].rows_out, e[i].cols_out}, {e[i].cols_out, 1}, offset[i])
                                  : flat.as_strided({e[i].cols_out}, {1}, offset[i]);
  }
  check(jvpattn_cast_params(e.data(), (int)e.size(), bf16 ? JVPATTN_BF16 : JVPATTN_FP16, stream_of(p0)), "jvpattn_cast_params");
  return py::cast(out);
}

}  // namespace

PYBIND11_MODULE(_native, m) {
  py::register_exception_translator([](std::exception_ptr p) {
    try {
      if (p) std::rethrow_exception(p);
    } catch (python_error &e) {
      e.restore();
    }
  });
  m.def("set_kernels", [](int kind) { g_kernels.store(kind); });
  m.def("cast_params", cast_params);
  m.def("attention", attention_py);
  m.def("ln_modulate", ln_py);
  m.def("gated_residual", gate_py);
  m.def("gate_ln", gate_ln_py);
  m.def("gelu", gelu_py);
  m.def("linear", linear_py);
  m.def("rotary_qkv", rotary_py);
}
