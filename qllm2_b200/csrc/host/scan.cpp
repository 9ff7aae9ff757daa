// pam_scan: argument checks, autograd nodes and launches of the chunked scan.
#include "common.h"

namespace qhost {
namespace {

using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::variable_list;

struct Config {
  double q_scale, eps;
  int64_t chunk;
};

qpam_scan_args scan_args(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& gamma, const Tensor& coef, const Tensor& s0, const Tensor& cu,
                         const Tensor& y, const Tensor& s_final, const Config& c) {
  qpam_scan_args a{};
  a.q = q.data_ptr(); a.k = k.data_ptr(); a.v = v.data_ptr();
  a.gamma = fptr(gamma); a.coef = fptr(coef); a.s0 = fptr(s0);
  a.cu_seqlens = static_cast<int32_t*>(ptr(cu));
  a.y = ptr(y); a.s_final = fptr(s_final);
  a.B = (int32_t)q.size(0); a.H = (int32_t)q.size(1); a.T = (int32_t)q.size(2); a.d = (int32_t)q.size(3);
  a.K = (int32_t)gamma.size(0);
  a.S = cu.defined() ? (int32_t)cu.numel() - 1 : a.B;
  a.chunk = (int32_t)c.chunk; a.io_dtype = dtype_code(q.scalar_type());
  a.q_scale = (float)c.q_scale; a.gamma_eps = (float)c.eps;
  return a;
}
void set_workspace(qpam_scan_args& a, const Tensor& ws) {
  a.workspace = ws.data_ptr();
  a.workspace_bytes = (size_t)ws.numel();
}
Tensor final_states(const qpam_scan_args& a, const Tensor& q) {
  return at::empty({a.K, a.S, a.H, a.d, a.d, 2}, q.options().dtype(at::kFloat));
}
Tensor grad_states(const Tensor& ds, const qpam_scan_args& a) {
  if (!ds.defined()) return ds;
  QH_REQUIRE(ds.numel() == (int64_t)a.K * a.S * a.H * a.d * a.d * 2, "ds_final has the wrong number of elements");
  return dense(ds.to(at::kFloat));
}

// One scan (all K states in its kernels).  Inputs contiguous, gamma / coef / s0 fp32.
struct Scan : Function<Scan> {
  static variable_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& gamma, const OptTensor& coef_,
                               const OptTensor& s0_, const OptTensor& cu_, double q_scale, double eps, int64_t chunk, bool save_states) {
    const Tensor coef = value(coef_), s0 = value(s0_), cu = value(cu_);
    const Config c{q_scale, eps, chunk};
    Tensor y = at::empty_like(q);
    qpam_scan_args a = scan_args(q, k, v, gamma, coef, s0, cu, y, Tensor(), c);
    Tensor s_final = final_states(a, q);
    a.s_final = fptr(s_final);
    const bool bwd = needs_grad(q) || needs_grad(k) || needs_grad(v) || needs_grad(gamma) || needs_grad(coef) || needs_grad(s0);
    const bool keep = bwd && save_states;
    Tensor ws = workspace(qpam_scan_workspace_bytes(&a, keep ? 1 : 0), q);
    set_workspace(a, ws);
    check(qpam_scan_fwd(&a, stream()), "qpam_scan_fwd");
    ctx->save_for_backward({q, k, v, gamma, coef, s0, cu, keep ? ws : Tensor()});
    ctx->saved_data["q_scale"] = q_scale;
    ctx->saved_data["eps"] = eps;
    ctx->saved_data["chunk"] = chunk;
    ctx->saved_data["ds0"] = needs_grad(s0);
    ctx->set_materialize_grads(false);
    return {y, s_final};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const Tensor &q = s[0], &k = s[1], &v = s[2], &gamma = s[3], &coef = s[4], &s0 = s[5], &cu = s[6];
    Tensor ws = s[7];
    const Config c{ctx->saved_data["q_scale"].toDouble(), ctx->saved_data["eps"].toDouble(), ctx->saved_data["chunk"].toInt()};
    qpam_scan_args a = scan_args(q, k, v, gamma, coef, s0, cu, Tensor(), Tensor(), c);
    const Tensor dy = grads[0].defined() ? dense_tokens(grads[0].to(q.scalar_type())) : at::zeros_like(q);
    QH_REQUIRE(dy.sizes() == q.sizes(), "dy shape ", shape(dy), " != y shape ", shape(q));
    const Tensor ds = grad_states(grads[1], a);
    Tensor dq = at::empty_like(q), dk = at::empty_like(k), dv = at::empty_like(v), dgamma = at::empty_like(gamma);
    Tensor dcoef = coef.defined() ? at::empty_like(coef) : Tensor();
    Tensor ds0 = s0.defined() && ctx->saved_data["ds0"].toBool() ? at::empty_like(s0) : Tensor();
    const int valid = ws.defined() ? 1 : 0;
    if (!valid) ws = workspace(qpam_scan_workspace_bytes(&a, 1), q);
    set_workspace(a, ws);
    check(qpam_scan_bwd(&a, dy.data_ptr(), dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), fptr(dgamma), fptr(dcoef), fptr(ds), fptr(ds0), valid, stream()),
          "qpam_scan_bwd");
    return {dq, dk, dv, dgamma, dcoef, ds0, Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

void state_ptrs(const Tensor& ys, void** out) {
  const int64_t K = ys.size(0), step = ys.stride(0) * ys.element_size();
  for (int64_t i = 0; i < K; ++i) out[i] = static_cast<char*>(ys.data_ptr()) + i * step;
}

// K = 2..4 states over the same bf16 q, k, v (d = 64), with gradients: the fused K-state kernels, forward and backward (8 x 6 x
// 2048, three states: 500 us with the output kernel once per state and the read-out as a pass of its own).  Without read-out
// weights the per-state outputs themselves are returned, and their gradients' dq, dk, dv added up in one set of buffers
// (qpam_scan_bwd_state).
struct ScanStates : Function<ScanStates> {
  static variable_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& gamma, const OptTensor& coef_,
                               const OptTensor& s0_, const OptTensor& cu_, double q_scale, double eps, int64_t chunk, bool token_major) {
    const Tensor coef = value(coef_), s0 = value(s0_), cu = value(cu_);
    const Config c{q_scale, eps, chunk};
    const int64_t B = q.size(0), H = q.size(1), T = q.size(2), d = q.size(3), K = gamma.size(0);
    Tensor y = !coef.defined() ? at::empty({K, B, H, T, d, 2}, q.options()) : token_major ? at::empty({B, T, H * d, 2}, q.options()) : at::empty_like(q);
    qpam_scan_args a = scan_args(q, k, v, gamma, coef, s0, cu, coef.defined() ? y : Tensor(), Tensor(), c);
    Tensor s_final = final_states(a, q);
    a.s_final = fptr(s_final);
    const bool bwd = needs_grad(q) || needs_grad(k) || needs_grad(v) || needs_grad(gamma) || needs_grad(coef) || needs_grad(s0);
    Tensor ws = workspace(qpam_scan_workspace_bytes(&a, bwd ? 1 : 0), q);
    set_workspace(a, ws);
    if (!coef.defined()) check(qpam_scan_fwd_states(&a, y.data_ptr(), stream()), "qpam_scan_fwd_states");
    else if (token_major) check(qpam_scan_fwd_tokens(&a, stream()), "qpam_scan_fwd_tokens");
    else check(qpam_scan_fwd(&a, stream()), "qpam_scan_fwd");
    ctx->save_for_backward({q, k, v, gamma, coef, s0, cu, bwd ? ws : Tensor()});
    ctx->saved_data["q_scale"] = q_scale;
    ctx->saved_data["eps"] = eps;
    ctx->saved_data["chunk"] = chunk;
    ctx->saved_data["ds0"] = needs_grad(s0);
    ctx->saved_data["tokens"] = token_major;
    ctx->set_materialize_grads(false);
    return {y, s_final};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const Tensor &q = s[0], &k = s[1], &v = s[2], &gamma = s[3], &coef = s[4], &s0 = s[5], &cu = s[6], &ws = s[7];
    const Config c{ctx->saved_data["q_scale"].toDouble(), ctx->saved_data["eps"].toDouble(), ctx->saved_data["chunk"].toInt()};
    const bool tokens = ctx->saved_data["tokens"].toBool();
    const int64_t B = q.size(0), H = q.size(1), T = q.size(2), d = q.size(3), K = gamma.size(0);
    qpam_scan_args a = scan_args(q, k, v, gamma, coef, s0, cu, Tensor(), Tensor(), c);
    set_workspace(a, ws);
    const Tensor ds = grad_states(grads[1], a);
    Tensor dq = at::empty_like(q), dk = at::empty_like(k), dv = at::empty_like(v), dgamma = at::empty_like(gamma), dcoef;
    Tensor ds0 = s0.defined() && ctx->saved_data["ds0"].toBool() ? at::empty_like(s0) : Tensor();
    if (coef.defined()) {
      dcoef = at::empty_like(coef);
      const Tensor dy = grads[0].defined() ? dense(grads[0].to(q.scalar_type())) : at::zeros({q.numel()}, q.options());
      const auto bwd = tokens ? &qpam_scan_bwd_tokens : &qpam_scan_bwd;
      check(bwd(&a, dy.data_ptr(), dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), fptr(dgamma), fptr(dcoef), fptr(ds), fptr(ds0), 1, stream()), "qpam_scan_bwd");
      return {dq, dk, dv, dgamma, dcoef, ds0, Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
    }
    const Tensor dys = grads[0].defined() ? dense(grads[0].to(q.scalar_type())) : at::zeros({K, B, H, T, d, 2}, q.options());
    void* dyk[QPAM_MAX_STATES];
    state_ptrs(dys, dyk);
    const int64_t row = B * H * T, st = (int64_t)a.S * H * d * d * 2;
    for (int64_t i = 0; i < K; ++i)
      check(qpam_scan_bwd_state(&a, (int)i, dyk[i], dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), fptr(dgamma) + i * row,
                                ds.defined() ? fptr(ds) + i * st : nullptr, ds0.defined() ? fptr(ds0) + i * st : nullptr, i > 0 ? 1 : 0, stream()),
            "qpam_scan_bwd_state");
    return {dq, dk, dv, dgamma, dcoef, ds0, Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

Tensor merge_heads(const Tensor& y) {
  return y.transpose(1, 2).reshape({y.size(0), y.size(2), y.size(1) * y.size(3), 2});
}

struct Inputs {
  Tensor q, k, v, gamma, coef, s0, cu;
  double q_scale;
};

Inputs checked(Tensor q, Tensor k, Tensor v, Tensor gamma, const OptTensor& coef_, const OptTensor& s0_, const OptTensor& cu_, int64_t head_dim) {
  // (a call without reverse-mode gradients runs without a node, which would have refused these)
  const auto has_tangent = [](const Tensor& t) { return t.defined() && t._fw_grad(0).defined(); };
  bool tangent = (coef_.has_value() && has_tangent(*coef_)) || (s0_.has_value() && has_tangent(*s0_));
  for (const Tensor* t : {&q, &k, &v, &gamma}) tangent = tangent || has_tangent(*t);
  QH_REQUIRE(!tangent, "the scan has no forward-mode derivative");
  // one dtype for the token tensors: under bf16 autocast the reference's matmuls round their inputs to bf16 anyway, so mixed
  // fp32 / bf16 operands (RoPE promotes q and k to fp32) are taken as bf16; otherwise they are promoted to the widest
  // dtype present.  The C ABI reads all three through q's dtype, so they must agree before the pointers are handed over.
  const at::ScalarType io = autocast_bf16() ? at::kBFloat16 : at::promote_types(at::promote_types(q.scalar_type(), k.scalar_type()), v.scalar_type());
  q = q.to(io); k = k.to(io); v = v.to(io);
  QH_REQUIRE(q.sizes() == k.sizes() && q.sizes() == v.sizes() && q.dim() == 5 && q.size(4) == 2, "q, k, v must share one shape [B,H,T,d,2]; got ", shape(q),
             ", ", shape(k), ", ", shape(v));
  gamma = gamma.to(at::kFloat);
  if (gamma.dim() == 3) gamma = gamma.unsqueeze(0);
  QH_REQUIRE(gamma.dim() == 4 && gamma.size(1) == q.size(0) && gamma.size(2) == q.size(1) && gamma.size(3) == q.size(2), "gamma shape ", shape(gamma),
             " does not match q ", shape(q));
  Tensor coef = value(coef_), s0 = value(s0_), cu = value(cu_);
  if (coef.defined()) {
    coef = coef.to(at::kFloat);
    if (coef.dim() == 4) coef = coef.unsqueeze(0);
    QH_REQUIRE(coef.dim() == 5 && coef.sizes().slice(0, 4) == gamma.sizes() && coef.size(4) == 2, "coef shape ", shape(coef), " != gamma shape + (2,)");
  }
  const int64_t n_seq = cu.defined() ? cu.numel() - 1 : q.size(0), d = q.size(3);
  if (s0.defined()) {
    s0 = s0.to(at::kFloat);
    QH_REQUIRE((s0.sizes() == at::IntArrayRef{gamma.size(0), n_seq, q.size(1), d, d, 2}), "s0 shape ", shape(s0), " != [K,S,H,d,d,2]");
  }
  QH_REQUIRE(!cu.defined() || q.size(0) == 1, "packed mode (cu_seqlens) needs B == 1");
  for (const Tensor* t : {&k, &v, &gamma, &coef, &s0})
    QH_REQUIRE(!t->defined() || t->device() == q.device(), "the scan's operands are on different devices: ", q.device(), " and ", t->device());
  QH_REQUIRE(q.is_cuda(), "PAM kernels need CUDA tensors (there is no CPU path in this package)");
  Inputs in;
  in.q = dense_tokens(q); in.k = dense_tokens(k); in.v = dense_tokens(v);
  in.gamma = gamma.contiguous();
  in.coef = coef.defined() ? dense(coef) : coef;
  in.s0 = s0.defined() ? dense(s0) : s0;
  in.cu = descriptor(cu, q.size(2), q.device());
  in.q_scale = 1.0 / std::sqrt((double)(head_dim > 0 ? head_dim : d));
  return in;
}

OptTensor opt(const Tensor& t) { return t.defined() ? OptTensor(t) : OptTensor(); }

// The inference form: nothing kept for a backward.  With the tensor-core kernels the output kernel writes [B,T,H*d,2] itself.
std::tuple<Tensor, Tensor> forward_only(const Inputs& in, double eps, int64_t chunk, bool token_major) {
  const Config c{in.q_scale, eps, chunk};
  const Tensor& q = in.q;
  const int64_t B = q.size(0), H = q.size(1), T = q.size(2), d = q.size(3), K = in.gamma.size(0);
  const bool direct = token_major && d == 64 && q.scalar_type() == at::kBFloat16 && T > 0 && (K > 1 || !in.coef.defined());
  Tensor y = direct ? at::empty({B, T, H * d, 2}, q.options()) : at::empty_like(q);
  qpam_scan_args a = scan_args(q, in.k, in.v, in.gamma, in.coef, in.s0, in.cu, y, Tensor(), c);
  Tensor s_final = final_states(a, q);
  a.s_final = fptr(s_final);
  Tensor ws = workspace(qpam_scan_workspace_bytes(&a, 0), q);
  set_workspace(a, ws);
  if (direct) check(qpam_scan_fwd_tokens(&a, stream()), "qpam_scan_fwd_tokens");
  else check(qpam_scan_fwd(&a, stream()), "qpam_scan_fwd");
  return {token_major && !direct ? merge_heads(y) : y, s_final};
}

// Returns (y, s_final), or (undefined, undefined) for the forms that are left to the caller: K > 1 tensor-core states
// whose chunk states are to be recomputed in the backward (save_states = false), and more of them than one call takes.
std::tuple<Tensor, Tensor> pam_scan(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& gamma, const OptTensor& coef, const OptTensor& s0,
                                    const OptTensor& cu, int64_t head_dim, double eps, int64_t chunk, bool save_states, bool token_major) {
  const Inputs in = checked(q, k, v, gamma, coef, s0, cu, head_dim);
  const bool grad = at::GradMode::is_enabled() && (needs_grad(in.q) || needs_grad(in.k) || needs_grad(in.v) || needs_grad(in.gamma) || needs_grad(in.coef) ||
                                                   needs_grad(in.s0));
  if (!grad) return forward_only(in, eps, chunk, token_major);
  const int64_t K = in.gamma.size(0);
  if (K > 1 && in.q.scalar_type() == at::kBFloat16 && in.q.size(3) == 64 && in.q.size(2) > 0) {
    if (!save_states || K > QPAM_MAX_STATES) return {Tensor(), Tensor()};
    auto out = ScanStates::apply(in.q, in.k, in.v, in.gamma, opt(in.coef), opt(in.s0), opt(in.cu), in.q_scale, eps, chunk, token_major);
    if (in.coef.defined()) return {out[0], out[1]};
    Tensor y = out[0].sum(0);
    return {token_major ? merge_heads(y) : y, out[1]};
  }
  auto out = Scan::apply(in.q, in.k, in.v, in.gamma, opt(in.coef), opt(in.s0), opt(in.cu), in.q_scale, eps, chunk, save_states);
  return {token_major ? merge_heads(out[0]) : out[0], out[1]};
}

std::tuple<Tensor, Tensor> pam_scan_tokens(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& gamma, const OptTensor& coef, const OptTensor& s0,
                                           const OptTensor& cu, int64_t head_dim, double eps, int64_t chunk) {
  at::NoGradGuard no_grad;
  return forward_only(checked(q, k, v, gamma, coef, s0, cu, head_dim), eps, chunk, true);
}

}  // namespace

Tensor descriptor(const Tensor& cu, int64_t T, at::Device device) {
  if (!cu.defined()) return cu;
  if (!cu.is_cuda()) {
    const Tensor c = cu.to(at::kLong).contiguous();
    const int64_t* p = c.data_ptr<int64_t>();
    bool ok = c.numel() >= 2 && p[0] == 0 && p[c.numel() - 1] <= T;
    for (int64_t i = 1; ok && i < c.numel(); ++i) ok = p[i] >= p[i - 1];
    QH_REQUIRE(ok, "cu_seqlens must start at 0, never decrease and end at or before T=", T, "; got ", c.slice(0, 0, 8));
  }
  return cu.to(device, at::kInt).contiguous();
}

std::tuple<Tensor, Tensor> scan_tokens(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& gamma, const Tensor& coef, const Tensor& s0,
                                       const Tensor& cu, double q_scale) {
  return forward_only(Inputs{q, k, v, gamma, coef, s0, cu, q_scale}, 1e-6, 64, true);
}

bool scan_prefill(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& gamma, const Tensor& coef, const Tensor& s0, const Tensor& cu, double q_scale,
                  const Tensor& pool, const Tensor& slots, int64_t layer, Tensor& y) {
  const int64_t B = q.size(0), H = q.size(1), T = q.size(2), d = q.size(3), K = gamma.size(0);
  if (d != 64 || q.scalar_type() != at::kBFloat16 || T == 0 || (K == 1 && coef.defined())) return false;
  y = at::empty({B, T, H * d, 2}, q.options());
  qpam_scan_args a = scan_args(q, k, v, gamma, coef, s0, cu, y, Tensor(), {q_scale, 1e-6, 64});
  Tensor ws = workspace(qpam_scan_workspace_bytes(&a, 0), q);
  set_workspace(a, ws);
  check(qpam_scan_prefill(&a, pool.data_ptr(), dtype_code(pool.scalar_type()), pool.size(0), (int)pool.size(1), (int)layer,
                          static_cast<const int32_t*>(slots.data_ptr()), stream()),
        "qpam_scan_prefill");
  return true;
}

void bind_scan(pybind11::module_& m) {
  namespace py = pybind11;
  m.def("pam_scan", &pam_scan, py::call_guard<py::gil_scoped_release>());
  m.def("pam_scan_tokens", &pam_scan_tokens, py::call_guard<py::gil_scoped_release>());
}

}  // namespace qhost
