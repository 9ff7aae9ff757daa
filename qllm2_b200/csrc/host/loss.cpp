// fused_linear_cross_entropy on one GPU: the autograd node around the C ABI.
#include "common.h"

namespace qhost {
namespace {

using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::variable_list;

qpam_ce_args ce_args(const Tensor& h, const Tensor& w, const Tensor& targets, const Tensor& mask, int64_t ignore_index, int64_t v_offset) {
  qpam_ce_args a{};
  a.h = h.data_ptr(); a.w = w.data_ptr();
  a.targets = static_cast<int64_t*>(ptr(targets)); a.mask = fptr(mask);
  a.N = h.size(0); a.V = w.size(0); a.v_offset = v_offset;
  a.F = (int32_t)h.size(1); a.io_dtype = dtype_code(h.scalar_type());
  a.ignore_index = ignore_index;
  return a;
}

// h [N,F], w [V,F] of one dtype, contiguous; mask fp32 [N] or undefined.
struct LinearCE : Function<LinearCE> {
  static Tensor forward(AutogradContext* ctx, const Tensor& h, const Tensor& w, const Tensor& targets, const OptTensor& mask_, int64_t ignore_index,
                        int64_t v_offset) {
    const Tensor mask = value(mask_);
    qpam_ce_args a = ce_args(h, w, targets, mask, ignore_index, v_offset);
    Tensor ws = workspace(qpam_ce_workspace_bytes(&a, 0), h);
    a.workspace = ws.data_ptr();
    a.workspace_bytes = (size_t)ws.numel();
    const auto f = h.options().dtype(at::kFloat);
    Tensor loss = at::empty({}, f), lse = at::empty({a.N}, f), denom = at::empty({1}, f);
    check(qpam_ce_loss(&a, fptr(lse), fptr(loss), nullptr, fptr(denom), nullptr, nullptr, nullptr, stream()), "qpam_ce_loss");
    ctx->save_for_backward({h, w, targets, mask, lse, denom});
    ctx->saved_data["ignore"] = ignore_index;
    ctx->saved_data["offset"] = v_offset;
    return loss;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const Tensor &h = s[0], &w = s[1];
    qpam_ce_args a = ce_args(h, w, s[2], s[3], ctx->saved_data["ignore"].toInt(), ctx->saved_data["offset"].toInt());
    Tensor ws = workspace(qpam_ce_workspace_bytes(&a, 1), h);
    a.workspace = ws.data_ptr();
    a.workspace_bytes = (size_t)ws.numel();
    const Tensor scale = grads[0].to(at::kFloat).contiguous();
    Tensor dh = at::empty_like(h), dw = at::empty_like(w);
    check(qpam_ce_bwd(&a, fptr(s[4]), fptr(scale), fptr(s[5]), dh.data_ptr(), dw.data_ptr(), stream()), "qpam_ce_bwd");
    return {dh, dw, Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

void check_rows(const Tensor& h, const Tensor& w, const Tensor& targets, const Tensor& mask) {
  QH_REQUIRE(h.is_cuda(), "PAM kernels need CUDA tensors (there is no CPU path in this package)");
  for (const Tensor* t : {&w, &targets, &mask})
    QH_REQUIRE(!t->defined() || t->device() == h.device(), "the loss's operands are on different devices: ", h.device(), " and ", t->device());
  QH_REQUIRE(h.dim() == 2 && w.dim() == 2 && h.size(1) == w.size(1), "h [N,F] and w [V,F] expected; got ", shape(h), ", ", shape(w));
  QH_REQUIRE(targets.scalar_type() == at::kLong && targets.numel() == h.size(0), "targets must be int64 with one entry per row of h");
  QH_REQUIRE(!mask.defined() || mask.numel() == h.size(0), "mask must have one entry per row of hidden_rows");
}

Tensor linear_ce(const Tensor& hidden, const Tensor& weight, const Tensor& targets, const OptTensor& mask, int64_t ignore_index, int64_t v_offset) {
  Tensor h = hidden.contiguous(), w = weight.contiguous();
  if (w.scalar_type() != h.scalar_type()) w = w.to(h.scalar_type());
  OptTensor m;
  if (mask.has_value()) m = mask->to(at::kFloat).contiguous();
  check_rows(h, w, targets, value(m));
  return LinearCE::apply(h, w, targets.contiguous(), m, ignore_index, v_offset);
}

// (per-token loss [N], [loss_sum, correct, tokens]) without gradients
std::tuple<Tensor, Tensor> linear_ce_rows(const Tensor& hidden, const Tensor& weight, const Tensor& targets_, const OptTensor& mask, int64_t ignore_index) {
  at::NoGradGuard no_grad;
  const Tensor h = hidden.contiguous(), w = weight.to(hidden.scalar_type()).contiguous(), targets = targets_.contiguous();
  const Tensor m = mask.has_value() ? mask->to(at::kFloat).contiguous() : Tensor();
  check_rows(h, w, targets, m);
  qpam_ce_args a = ce_args(h, w, targets, m, ignore_index, 0);
  Tensor ws = workspace(qpam_ce_workspace_bytes(&a, 0), h);
  a.workspace = ws.data_ptr();
  a.workspace_bytes = (size_t)ws.numel();
  const auto f = h.options().dtype(at::kFloat);
  Tensor lse = at::empty({a.N}, f), rows = at::empty({a.N}, f), sums = at::zeros({3}, f);
  if (a.N > 0)
    check(qpam_ce_loss(&a, fptr(lse), nullptr, fptr(rows), nullptr, fptr(sums), fptr(sums) + 1, fptr(sums) + 2, stream()), "qpam_ce_loss");
  return {rows, sums};
}

}  // namespace

void bind_loss(pybind11::module_& m) {
  namespace py = pybind11;
  m.def("linear_ce", &linear_ce, py::call_guard<py::gil_scoped_release>());
  m.def("linear_ce_rows", &linear_ce_rows, py::call_guard<py::gil_scoped_release>());
}

}  // namespace qhost
