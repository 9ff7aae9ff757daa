// Prefill of a packed model: the launch sequence of FusedForward's blocks (library GEMMs and this package's kernels) for a
// batch of prompts, without the interpreter between the ~15 launches of a block.
#include "common.h"

namespace qhost {
namespace {

namespace py = pybind11;

struct Layer {
  Tensor w_gu, w_down, w_front, b_front, w_mag, b_mag, w_o, n1, n2, act_bias, act_beta, cgu_scale, pam_scale, dt_bias, dt_off;
  // columns of dt, pg, phase, score: in the block input's projection (from_mag false) or in that of |x|; -1 = absent
  int64_t col[4];
  bool from_mag[4];
  double gamma_floor;
};

Tensor attr(const py::object& o, const char* name) {
  const py::object v = o.attr(name);
  return v.is_none() ? Tensor() : v.cast<Tensor>();
}

class Packed {
 public:
  Packed(int64_t D, int64_t H, int64_t d, int64_t K, const py::list& layers, Tensor embed_scale, Tensor out_scale, const OptTensor& rope)
      : D_(D), H_(H), d_(d), K_(K), embed_scale_(std::move(embed_scale)), out_scale_(std::move(out_scale)), rope_(value(rope)) {
    for (const auto& item : layers) {
      const py::object o = py::reinterpret_borrow<py::object>(item);
      Layer l;
      l.w_gu = attr(o, "w_gu"); l.w_down = attr(o, "w_down"); l.w_front = attr(o, "w_front"); l.b_front = attr(o, "b_front");
      l.w_mag = attr(o, "w_mag"); l.b_mag = attr(o, "b_mag"); l.w_o = attr(o, "w_o"); l.n1 = attr(o, "n1"); l.n2 = attr(o, "n2");
      l.act_bias = attr(o, "act_bias"); l.act_beta = attr(o, "act_beta"); l.cgu_scale = attr(o, "cgu_scale"); l.pam_scale = attr(o, "pam_scale");
      l.dt_bias = attr(o, "dt_bias"); l.dt_off = attr(o, "dt_off");
      l.gamma_floor = o.attr("gamma_floor").cast<double>();
      const py::dict cols = o.attr("cols");
      const char* names[4] = {"dt", "pg", "phase", "score"};
      for (int i = 0; i < 4; ++i) {
        l.col[i] = -1;
        l.from_mag[i] = false;
        if (cols.contains(names[i])) {
          const py::tuple t = cols[names[i]];
          l.from_mag[i] = t[0].cast<std::string>() == "m";
          l.col[i] = t[1].cast<int64_t>();
        }
      }
      layers_.push_back(l);
    }
  }

  // embed_real, embed_imag [V,D], or the embedded tokens [B,T,D,2]; ids [B,T]; every row (cu undefined) or every piece of the one packed row (cu [S+1]) belongs to slots[i], whose states
  // [n_slots, L, K, H, d, d, 2] it leaves at its end.  resumed [S] (fp32, 0 or 1): pieces that start from their slot's
  // state.  Returns the residual stream after the last block, normalised for the head, [B*T, D, 2].
  Tensor prefill(const OptTensor& embed_real, const OptTensor& embed_imag, const OptTensor& embedded, const Tensor& ids, const Tensor& pool, const Tensor& slots_, const OptTensor& cu_,
                 const OptTensor& positions_, const OptTensor& resumed_) {
    at::NoGradGuard no_grad;
    QH_REQUIRE(ids.dim() == 2 && ids.numel() > 0, "prefill: ids [B,T] expected; got ", shape(ids));
    const int64_t B = ids.size(0), T = ids.size(1), N = B * T, inner = H_ * d_, L = (int64_t)layers_.size();
    const at::ScalarType dt = layers_[0].w_gu.scalar_type();
    // what the kernels index by pointer: one slot (and one resumed flag) a sequence, a pool of this model's states
    const auto is_table = [&](const OptTensor& t) { return t.has_value() && t->dim() == 2 && t->size(1) == D_; };
    QH_REQUIRE(embedded.has_value() ? embedded->sizes() == at::IntArrayRef({B, T, D_, 2}) : is_table(embed_real) && is_table(embed_imag),
               "prefill: embeddings [V,", D_, "] or embedded tokens [B,T,", D_, ",2] expected");
    QH_REQUIRE(!cu_.has_value() || (B == 1 && cu_->dim() == 1 && cu_->numel() >= 2), "prefill: a packed batch is one row of ids with cu [S+1]");
    const int64_t n_seq = cu_.has_value() ? cu_->numel() - 1 : B;
    QH_REQUIRE(slots_.numel() == n_seq && !slots_.is_floating_point() && (!resumed_.has_value() || resumed_->numel() == n_seq), "prefill: one slot a sequence expected, ", n_seq,
               " in all; got ", shape(slots_));
    QH_REQUIRE(pool.is_contiguous() && pool.device() == ids.device() && (pool.sizes().slice(1) == at::IntArrayRef{L, K_, H_, d_, d_, 2}) && pool.dim() == 7,
               "prefill: state pool ", shape(pool), " does not fit this model");
    QH_REQUIRE(!positions_.has_value() || positions_->numel() == N, "prefill: positions must have one entry per token");
    QH_REQUIRE(!rope_.defined() || positions_.has_value() || T <= rope_.size(0), "position beyond max_position of this FusedForward");
    const Tensor cu = descriptor(value(cu_), T, ids.device()), slots = slots_.to(ids.device(), at::kInt).contiguous();
    const Tensor resumed = resumed_.has_value() ? resumed_->to(ids.device(), at::kFloat) : Tensor();
    const Tensor positions = positions_.has_value() ? positions_->reshape({-1}).to(ids.device(), at::kLong).contiguous() : Tensor();
    QH_REQUIRE(ids.is_cuda(), "PAM kernels need CUDA tensors (there is no CPU path in this package)");
    const int code = dtype_code(dt), pool_code = dtype_code(pool.scalar_type());
    const int64_t n_slots = pool.size(0);
    void* st = stream();
    Tensor z = (embedded.has_value() ? *embedded : at::stack({at::embedding(*embed_real, ids), at::embedding(*embed_imag, ids)}, -1)).reshape({N, D_, 2}).to(dt);
    z = dense(z);
    const auto opts = z.options();
    Tensor xn = at::empty_like(z), mag;
    check(qpam_residual_cnorm_fwd(z.data_ptr(), nullptr, nullptr, fptr(embed_scale_), xn.data_ptr(), nullptr, code, N, (int)D_, 1e-6f, st),
          "qpam_residual_cnorm_fwd");
    z = xn;
    xn = at::empty_like(z);
    check(qpam_residual_cnorm_fwd(z.data_ptr(), nullptr, nullptr, fptr(layers_[0].n1), xn.data_ptr(), nullptr, code, N, (int)D_, 1e-6f, st),
          "qpam_residual_cnorm_fwd");
    Tensor q = at::empty({B, H_, T, d_, 2}, opts), k = at::empty_like(q), v = at::empty_like(q);
    Tensor gamma = at::empty({K_, B, H_, T}, opts.dtype(at::kFloat)), coef = K_ > 1 ? at::empty({K_, B, H_, T, 2}, gamma.options()) : Tensor();
    const Tensor slots_long = resumed.defined() ? slots.to(at::kLong) : Tensor();
    for (size_t li = 0; li < layers_.size(); ++li) {
      const Layer& l = layers_[li];
      const int64_t hidden = l.act_bias.numel();
      const Tensor gu = at::linear(xn.view({N, 2 * D_}), l.w_gu);
      Tensor gated = at::empty({N, 2 * hidden}, opts);
      check(qpam_act_gate_packed_fwd(gu.data_ptr(), gu.size(1), code, fptr(l.act_bias), fptr(l.act_beta), gated.data_ptr(), N, (int)hidden, st),
            "qpam_act_gate_packed_fwd");
      const Tensor down = at::linear(gated, l.w_down);
      if (l.w_mag.defined() && !mag.defined()) mag = at::empty({N, D_}, opts);
      check(qpam_residual_cnorm_fwd(z.data_ptr(), down.data_ptr(), fptr(l.cgu_scale), fptr(l.n2), xn.data_ptr(), l.w_mag.defined() ? mag.data_ptr() : nullptr,
                                    code, N, (int)D_, 1e-6f, st),
            "qpam_residual_cnorm_fwd");
      const Tensor raw = at::linear(xn.view({N, 2 * D_}), l.w_front, l.b_front);
      const Tensor rawm = l.w_mag.defined() ? at::linear(mag, l.w_mag, l.b_mag) : Tensor();
      qpam_front_args f{};
      const void* src[4];
      int64_t ld[4];
      for (int i = 0; i < 4; ++i) {
        const Tensor& base = l.from_mag[i] ? rawm : raw;
        src[i] = l.col[i] < 0 ? nullptr : static_cast<char*>(base.data_ptr()) + l.col[i] * base.element_size();
        ld[i] = l.col[i] < 0 ? 0 : base.size(1);
      }
      f.qkv = raw.data_ptr(); f.ld_qkv = raw.size(1);
      f.dt = src[0]; f.ld_dt = ld[0]; f.pg = src[1]; f.ld_pg = ld[1]; f.phase = src[2]; f.ld_phase = ld[2]; f.score = src[3]; f.ld_score = ld[3];
      f.dt_bias = fptr(l.dt_bias); f.state_dt_offset = fptr(l.dt_off);
      f.rope = fptr(rope_); f.rope_len = rope_.defined() ? rope_.size(0) : 0;
      f.positions = static_cast<int64_t*>(ptr(positions)); f.offset = 0;
      f.q = q.data_ptr(); f.k = k.data_ptr(); f.v = v.data_ptr(); f.gamma = fptr(gamma); f.coef = fptr(coef);
      f.gamma_floor = (float)l.gamma_floor; f.q_scale = 1.f;
      f.B = (int)B; f.T = (int)T; f.H = (int)H_; f.d = (int)d_; f.K = (int)K_; f.io_dtype = code;
      check(qpam_pam_front_fwd(&f, st), "qpam_pam_front_fwd");
      Tensor s0;
      if (resumed.defined())     // fresh sequences start from zero whatever their slot held
        s0 = (pool.select(1, (int64_t)li).index_select(0, slots_long).to(at::kFloat) * resumed.view({-1, 1, 1, 1, 1, 1})).transpose(0, 1).contiguous();
      const double q_scale = 1.0 / std::sqrt((double)d_);
      Tensor y;
      if (!scan_prefill(q, k, v, gamma, coef, s0, cu, q_scale, pool, slots, (int64_t)li, y)) {
        Tensor s;
        std::tie(y, s) = scan_tokens(q, k, v, gamma, coef, s0, cu, q_scale);
        check(qpam_pool_store(pool.data_ptr(), pool_code, n_slots, (int)L, (int)li, static_cast<int32_t*>(slots.data_ptr()), fptr(s), (int)s.size(1), (int)H_,
                              (int)d_, (int)K_, st),
              "qpam_pool_store");
      }
      const Tensor o = at::linear(y.view({N, 2 * inner}), l.w_o);
      const Tensor& next = li + 1 < layers_.size() ? layers_[li + 1].n1 : out_scale_;
      check(qpam_residual_cnorm_fwd(z.data_ptr(), o.data_ptr(), fptr(l.pam_scale), fptr(next), xn.data_ptr(), nullptr, code, N, (int)D_, 1e-6f, st),
            "qpam_residual_cnorm_fwd");
    }
    return xn;
  }

 private:
  int64_t D_, H_, d_, K_;
  std::vector<Layer> layers_;
  Tensor embed_scale_, out_scale_, rope_;
};

}  // namespace

void bind_forward(py::module_& m) {
  py::class_<Packed>(m, "Packed")
      .def(py::init<int64_t, int64_t, int64_t, int64_t, const py::list&, Tensor, Tensor, const OptTensor&>())
      .def("prefill", &Packed::prefill, py::call_guard<py::gil_scoped_release>());
}

}  // namespace qhost
