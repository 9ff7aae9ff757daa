// One V11 block as ONE autograd node for bf16-autocast training (fp32 parameters, bf16 residual stream): forward and
// backward as fixed launch sequences of library GEMMs, the scan and the kernels of block_train.cu.  Operator by operator a
// block was ~45 nodes and ~150 launches a step, and at a few hundred tokens all of its time was spent between them.
// The forward rounds where the operators round: each projection is its own GEMM in the operators' shape, every tensor they
// store in bf16 is rounded here too.  (The gate's phase is read off gates of any magnitude, so one flipped bit of a
// projection's input can turn a small gate by tens of degrees: same bits forward means the same gradients.)  For K > 1 states
// these are the operators whose scan keeps every state's output (ops.pam_scan with save_states = False): K outputs rounded to
// bf16, then the read-out.  The operators' default scan forms the read-out in the fused output kernel and rounds once; here
// that form is 3 % faster (8 blocks, 8 x 2048 tokens, three states: 18.5 against 19.1 ms) but moves that step's gradients by
// 0.46 of their norm, so a run could not be continued across the change.  The backward has no such discontinuity and runs
// stacked: one GEMM for [gate | up] and one for [qkv | gates], each way.
#include "common.h"

namespace qhost {
namespace {

using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::variable_list;

// parameters, in the order the Python side passes them (absent ones undefined)
enum {
  N1, GATE_R, GATE_I, UP_R, UP_I, DOWN_R, DOWN_I, ACT_BIAS, ACT_BETA, CGU_SCALE, N2, QKV_R, QKV_I, O_R, O_I, DT_W, DT_B, DT_BIAS, PG_W, PG_B, DT_OFF, PHASE_W,
  PHASE_B, SCORE_W, SCORE_B, PAM_SCALE, N_PARAMS
};

struct Shape {
  int64_t B, T, N, D, H, d, K, inner, hidden;
  // gate sources dt, pg, phase, score: rows, column in their projection, and whether that reads |x|
  int64_t rows[4], col[4];
  bool mag[4];
  int64_t used_a, rows_a, used_m, rows_m;   // columns of the two projections that are used / with padding

  Shape(const Tensor& x, const variable_list& p, int64_t H_, int64_t d_, int64_t K_, bool pg_content, bool routing_content) {
    B = x.size(0); T = x.size(1); D = x.size(2); N = B * T;
    H = H_; d = d_; K = K_; inner = H * d;
    hidden = p[GATE_R].size(0);
    rows[0] = H; rows[1] = p[PG_W].defined() ? H : 0; rows[2] = p[PHASE_W].defined() ? H * K : 0; rows[3] = p[SCORE_W].defined() ? H * K : 0;
    mag[0] = false; mag[1] = !pg_content; mag[2] = mag[3] = !routing_content;
    used_a = 6 * inner;
    used_m = 0;
    for (int i = 0; i < 4; ++i) {
      int64_t& at = mag[i] ? used_m : used_a;
      col[i] = rows[i] ? at : -1;
      at += rows[i];
    }
    rows_a = (used_a + 7) / 8 * 8;
    rows_m = (used_m + 7) / 8 * 8;
  }
  bool pg_with_dt() const { return rows[1] && !mag[1]; }   // one product for both
};

struct Packed {
  Tensor w_gu, w_down, w_front, w_mag, w_o;
  Tensor bias;                               // one row for each gate source, rows 256-byte aligned
};

const int WEIGHT_OF[4] = {DT_W, PG_W, PHASE_W, SCORE_W};
const int BIAS_OF[4] = {DT_B, PG_B, PHASE_B, SCORE_B};

struct PackList {
  qpam_pack_item it[24];
  int n = 0;
  void add(const Tensor& a, const Tensor& b, const Tensor& packed, int64_t row, int64_t out, int64_t in, int kind, int64_t row_len) {
    if (out == 0) return;
    it[n++] = {fptr(a), fptr(b), static_cast<char*>(packed.data_ptr()) + row * row_len * 2, (int)out, (int)in, kind};
  }
};

// The weights' items of both directions: parameters -> packed, or packed gradients -> the parameters' gradients.
void weight_items(PackList& l, const Shape& s, const variable_list& p, const Tensor& gu, const Tensor& down, const Tensor& front, const Tensor& mag,
                  const Tensor& o) {
  const int64_t D2 = 2 * s.D;
  l.add(p[GATE_R], p[GATE_I], gu, 0, s.hidden, s.D, QPAM_PACK_COMPLEX, D2);
  l.add(p[UP_R], p[UP_I], gu, 2 * s.hidden, s.hidden, s.D, QPAM_PACK_COMPLEX, D2);
  l.add(p[DOWN_R], p[DOWN_I], down, 0, s.D, s.hidden, QPAM_PACK_COMPLEX, 2 * s.hidden);
  l.add(p[QKV_R], p[QKV_I], front, 0, 3 * s.inner, s.D, QPAM_PACK_COMPLEX, D2);
  l.add(p[O_R], p[O_I], o, 0, s.D, s.inner, QPAM_PACK_COMPLEX, 2 * s.inner);
  for (int i = 0; i < 4; ++i) {
    if (!s.rows[i]) continue;
    if (s.mag[i]) l.add(p[WEIGHT_OF[i]], Tensor(), mag, s.col[i], s.rows[i], s.D, QPAM_PACK_PLAIN, s.D);
    else l.add(p[WEIGHT_OF[i]], Tensor(), front, s.col[i], s.rows[i], s.D, QPAM_PACK_INTERLEAVE, D2);
  }
}

Packed pack(const Shape& s, const variable_list& p, void* st) {
  const auto o = p[N1].options().dtype(at::kBFloat16);
  Packed w;
  w.w_gu = at::empty({4 * s.hidden, 2 * s.D}, o);
  w.w_down = at::empty({2 * s.D, 2 * s.hidden}, o);
  w.w_front = at::empty({s.rows_a, 2 * s.D}, o);
  w.w_o = at::empty({2 * s.D, 2 * s.inner}, o);
  w.bias = at::empty({4, (s.H * s.K + s.H + 127) / 128 * 128}, o);
  if (s.rows_m) w.w_mag = at::empty({s.rows_m, s.D}, o);
  PackList l;
  weight_items(l, s, p, w.w_gu, w.w_down, w.w_front, w.w_mag, w.w_o);
  const Tensor none;
  for (int i = 0; i < 4; ++i)
    if (s.rows[i]) {
      const bool stacked = i == 1 && s.pg_with_dt();      // beside the decay's bias, as its weight rows are
      l.add(p[BIAS_OF[i]], none, w.bias[stacked ? 0 : i], stacked ? s.H : 0, 1, s.rows[i], QPAM_PACK_PLAIN, 1);
    }
  if (s.rows_a > s.used_a) l.add(none, none, w.w_front, s.used_a, s.rows_a - s.used_a, 2 * s.D, QPAM_PACK_PLAIN, 2 * s.D);
  if (s.rows_m > s.used_m) l.add(none, none, w.w_mag, s.used_m, s.rows_m - s.used_m, s.D, QPAM_PACK_PLAIN, s.D);
  check(qpam_pack_block(l.it, l.n, st), "qpam_pack_block");
  return w;
}

// The gate sources' logits: outputs of their own projections ([1] undefined when it is columns H.. of [0]).
qpam_front_args front_args(const Shape& s, const variable_list& p, const Tensor& qkv, const Tensor* logits, const Tensor& rope, int64_t offset, double floor) {
  qpam_front_args f{};
  const void* src[4];
  int64_t ld[4];
  for (int i = 0; i < 4; ++i) {
    const bool stacked = i == 1 && s.pg_with_dt();
    const Tensor& t = logits[stacked ? 0 : i];
    src[i] = s.rows[i] ? static_cast<char*>(t.data_ptr()) + (stacked ? s.H * 2 : 0) : nullptr;
    ld[i] = s.rows[i] ? t.size(1) : 0;
  }
  f.qkv = qkv.data_ptr(); f.ld_qkv = qkv.size(1);
  f.dt = src[0]; f.ld_dt = ld[0]; f.pg = src[1]; f.ld_pg = ld[1]; f.phase = src[2]; f.ld_phase = ld[2]; f.score = src[3]; f.ld_score = ld[3];
  f.dt_bias = fptr(p[DT_BIAS]); f.state_dt_offset = fptr(p[DT_OFF]);
  f.rope = fptr(rope); f.rope_len = rope.defined() ? rope.size(0) : 0; f.offset = offset;
  f.gamma_floor = (float)floor; f.q_scale = 1.f;
  f.B = (int)s.B; f.T = (int)s.T; f.H = (int)s.H; f.d = (int)s.d; f.K = (int)s.K; f.io_dtype = QPAM_BF16;
  return f;
}

qpam_scan_args scan_args(const Shape& s, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& gamma) {
  qpam_scan_args a{};
  a.q = q.data_ptr(); a.k = k.data_ptr(); a.v = v.data_ptr(); a.gamma = fptr(gamma);
  a.B = (int)s.B; a.H = (int)s.H; a.T = (int)s.T; a.d = (int)s.d; a.K = (int)s.K; a.S = (int)s.B;
  a.chunk = 64; a.io_dtype = QPAM_BF16;
  a.q_scale = (float)(1.0 / std::sqrt((double)s.d)); a.gamma_eps = 1e-6f;
  return a;
}
void state_ptrs(const Tensor& ys, void** out) {
  const int64_t step = ys.stride(0) * ys.element_size();
  for (int64_t i = 0; i < ys.size(0); ++i) out[i] = static_cast<char*>(ys.data_ptr()) + i * step;
}
int parts_of(int64_t n, int64_t per) { return (int)std::max<int64_t>(1, std::min<int64_t>(at::cuda::getCurrentDeviceProperties()->multiProcessorCount * per, n)); }

struct Block : Function<Block> {
  // params: those that are present, bit i of `present` for parameter i (the node's inputs have to be defined tensors)
  static variable_list forward(AutogradContext* ctx, const Tensor& x_, at::TensorList params, const OptTensor& rope_, int64_t present, int64_t H, int64_t d,
                               int64_t K, bool pg_content, bool routing_content, double gamma_floor, int64_t offset) {
    c10::impl::ExcludeDispatchKeyGuard no_autocast(c10::DispatchKey::AutocastCUDA);
    variable_list p(N_PARAMS);
    for (int i = 0, at = 0; i < N_PARAMS; ++i)
      if (present >> i & 1) p[i] = params[at++];
    const Tensor x = x_, rope = value(rope_);
    const Shape s(x, p, H, d, K, pg_content, routing_content);
    void* st = stream();
    bool bwd = x_.requires_grad();
    for (const Tensor& t : p) bwd = bwd || needs_grad(t);
    const auto o = x.options();
    const auto f32o = o.dtype(at::kFloat);
    const int64_t N = s.N, D = s.D;
    const float eps = 1e-6f;
    const Packed w = pack(s, p, st);
    // channel mix
    Tensor xn = at::empty_like(x);
    check(qpam_norm_train_fwd(x.data_ptr(), nullptr, nullptr, fptr(p[N1]), nullptr, xn.data_ptr(), nullptr, N, (int)D, eps, st), "qpam_norm_train_fwd");
    const Tensor gate = at::linear(xn.view({N, 2 * D}), w.w_gu.narrow(0, 0, 2 * s.hidden)), up = at::linear(xn.view({N, 2 * D}), w.w_gu.narrow(0, 2 * s.hidden, 2 * s.hidden));
    Tensor gated = at::empty({N, 2 * s.hidden}, o);
    check(qpam_act_gate_train_fwd(gate.data_ptr(), up.data_ptr(), fptr(p[ACT_BIAS]), fptr(p[ACT_BETA]), gated.data_ptr(), N, (int)s.hidden, st), "qpam_act_gate_train_fwd");
    const Tensor mixed = at::linear(gated, w.w_down);
    Tensor x1 = at::empty_like(x), xn2 = at::empty_like(x), mag = s.rows_m ? at::empty({N, D}, o) : Tensor();
    check(qpam_norm_train_fwd(x.data_ptr(), mixed.data_ptr(), fptr(p[CGU_SCALE]), fptr(p[N2]), x1.data_ptr(), xn2.data_ptr(), ptr(mag), N, (int)D, eps, st),
          "qpam_norm_train_fwd");
    // sequence mix
    const Tensor rows = xn2.view({N, 2 * D});
    const Tensor qkv = at::linear(rows, w.w_front.narrow(0, 0, 6 * s.inner));
    Tensor logits[4];
    for (int i = 0; i < 4; ++i) {
      if (!s.rows[i] || (i == 1 && s.pg_with_dt())) continue;
      const int64_t n = s.rows[i] + (i == 0 && s.pg_with_dt() ? s.rows[1] : 0);
      logits[i] = at::linear(s.mag[i] ? mag : rows, (s.mag[i] ? w.w_mag : w.w_front).narrow(0, s.col[i], n), w.bias[i].narrow(0, 0, n));
    }
    Tensor q = at::empty({s.B, H, s.T, d, 2}, o), k = at::empty_like(q), v = at::empty_like(q);
    Tensor gamma = at::empty({K, s.B, H, s.T}, f32o), coef = K > 1 ? at::empty({K, s.B, H, s.T, 2}, f32o) : Tensor();
    qpam_front_args f = front_args(s, p, qkv, logits, rope, offset, gamma_floor);
    f.q = q.data_ptr(); f.k = k.data_ptr(); f.v = v.data_ptr(); f.gamma = fptr(gamma); f.coef = fptr(coef);
    check(qpam_pam_front_fwd(&f, st), "qpam_pam_front_fwd");
    Tensor y = at::empty({N, 2 * s.inner}, o), s_final = at::empty({K, s.B, H, d, d, 2}, f32o);
    qpam_scan_args a = scan_args(s, q, k, v, gamma);
    a.s_final = fptr(s_final);
    if (K > 1 && !bwd) a.coef = fptr(coef);
    Tensor ws = workspace(qpam_scan_workspace_bytes(&a, bwd ? 1 : 0), q);
    a.workspace = ws.data_ptr();
    a.workspace_bytes = (size_t)ws.numel();
    if (K == 1 || !bwd) {
      a.y = y.data_ptr();
      check(qpam_scan_fwd_tokens(&a, st), "qpam_scan_fwd_tokens");
    } else {
      // every state's output rounded to bf16 before the read-out (see the top of this file)
      const Tensor ys = at::empty({K, s.B, H, s.T, d, 2}, o);
      check(qpam_scan_fwd_states(&a, ys.data_ptr(), st), "qpam_scan_fwd_states");
      void* yk[QPAM_MAX_STATES];
      state_ptrs(ys, yk);
      check(qpam_state_combine_tokens_fwd(yk, fptr(coef), y.data_ptr(), QPAM_BF16, (int)K, (int)s.B, (int)H, (int)s.T, (int)d, st), "qpam_state_combine_tokens_fwd");
    }
    const Tensor out = at::linear(y, w.w_o);
    Tensor x2 = at::empty_like(x);
    check(qpam_scaled_residual_fwd(x1.data_ptr(), QPAM_BF16, out.data_ptr(), QPAM_BF16, fptr(p[PAM_SCALE]), x2.data_ptr(), x.numel(), st), "qpam_scaled_residual_fwd");
    if (bwd) {
      variable_list keep = {x, xn, gate, up, gated, mixed, x1, xn2, mag, qkv, logits[0], logits[1], logits[2], logits[3], q, k, v, gamma, coef, ws, y, out, w.w_gu, w.w_down, w.w_front, w.w_mag, w.w_o, rope};
      keep.insert(keep.end(), p.begin(), p.end());
      ctx->save_for_backward(std::move(keep));
      ctx->saved_data["H"] = H;
      ctx->saved_data["d"] = d;
      ctx->saved_data["K"] = K;
      ctx->saved_data["pc"] = pg_content;
      ctx->saved_data["rc"] = routing_content;
      ctx->saved_data["floor"] = gamma_floor;
      ctx->saved_data["offset"] = offset;
    }
    ctx->set_materialize_grads(false);
    return {x2, s_final};
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    c10::impl::ExcludeDispatchKeyGuard no_autocast(c10::DispatchKey::AutocastCUDA);
    const auto sv = ctx->get_saved_variables();
    enum { X, XN, GATE, UP, GATED, MIXED, X1, XN2, MAG, QKV, LOGITS, LOGITS_END = LOGITS + 3, Q, KK, V, GAMMA, COEF, WS, Y, OUT, W_GU, W_DOWN, W_FRONT, W_MAG, W_O, ROPE, FIRST_PARAM };
    const variable_list p(sv.begin() + FIRST_PARAM, sv.end());
    const int64_t H = ctx->saved_data["H"].toInt(), d = ctx->saved_data["d"].toInt(), K = ctx->saved_data["K"].toInt();
    const Tensor& x = sv[X];
    const Shape s(x, p, H, d, K, ctx->saved_data["pc"].toBool(), ctx->saved_data["rc"].toBool());
    void* st = stream();
    const auto o = x.options();
    const auto f32o = o.dtype(at::kFloat);
    const int64_t N = s.N, D = s.D;
    const float eps = 1e-6f;
    const Tensor dx2 = grads[0].defined() ? dense(grads[0].to(at::kBFloat16)) : at::zeros_like(x);
    variable_list g(N_PARAMS);
    for (int i = 0; i < N_PARAMS; ++i)
      if (p[i].defined()) g[i] = at::empty_like(p[i]);
    std::vector<qpam_colsum_item> sums;
    variable_list keep;                      // partial sums, alive until k_colsum has been enqueued
    auto partial = [&](int64_t P, int64_t C) {
      keep.push_back(at::empty({P, C}, f32o));
      return fptr(keep.back());
    };
    auto sum = [&](const float* part, int64_t P, int64_t ld, int64_t C, const Tensor& out) { sums.push_back({part, fptr(out), (int)P, (int)C, (int)ld}); };

    // ---- residual and output projection of the sequence mix
    Tensor dout = at::empty({N, 2 * D}, o);
    const int Pr = parts_of(x.numel() / 4096 + 1, 8);
    float* part = partial(Pr, 1);
    check(qpam_scaled_residual_bwd(dx2.data_ptr(), QPAM_BF16, sv[OUT].data_ptr(), QPAM_BF16, fptr(p[PAM_SCALE]), dout.data_ptr(), part, Pr, x.numel(), st),
          "qpam_scaled_residual_bwd");
    sum(part, Pr, 1, 1, g[PAM_SCALE]);
    const Tensor dy = at::mm(dout, sv[W_O]);
    const Tensor dw_o = at::mm(dout.t(), sv[Y]);
    // ---- scan
    Tensor dq = at::empty_like(sv[Q]), dk = at::empty_like(sv[Q]), dv = at::empty_like(sv[Q]), dgamma = at::empty_like(sv[GAMMA]);
    Tensor dcoef;
    qpam_scan_args a = scan_args(s, sv[Q], sv[KK], sv[V], sv[GAMMA]);
    a.workspace = sv[WS].data_ptr();
    a.workspace_bytes = (size_t)sv[WS].numel();
    const Tensor ds = grads[1].defined() ? dense(grads[1].to(at::kFloat)) : Tensor();
    if (K == 1) {
      const Tensor dyh = dy.view({s.B, s.T, H, d, 2}).transpose(1, 2).contiguous();
      check(qpam_scan_bwd(&a, dyh.data_ptr(), dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), fptr(dgamma), nullptr, fptr(ds), nullptr, 1, st), "qpam_scan_bwd");
    } else {
      dcoef = at::empty_like(sv[COEF]);
      a.coef = fptr(sv[COEF]);
      check(qpam_scan_bwd_tokens(&a, dy.data_ptr(), dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), fptr(dgamma), fptr(dcoef), fptr(ds), nullptr, 1, st),
            "qpam_scan_bwd_tokens");
    }
    // ---- front
    Tensor d_raw = at::empty({N, s.rows_a}, o), d_rawm = s.rows_m ? at::empty({N, s.rows_m}, o) : Tensor();
    const int NS = (int)(3 * K + 1);
    const int Pf = parts_of((N + 3) / 4, 4);
    qpam_front_bwd_args fb{};
    fb.f = front_args(s, p, sv[QKV], &sv[LOGITS], sv[ROPE], ctx->saved_data["offset"].toInt(), ctx->saved_data["floor"].toDouble());
    fb.f.q = dq.data_ptr(); fb.f.k = dk.data_ptr(); fb.f.v = dv.data_ptr(); fb.f.gamma = fptr(dgamma); fb.f.coef = fptr(dcoef);
    fb.d_raw = d_raw.data_ptr(); fb.ld_raw = s.rows_a; fb.d_rawm = ptr(d_rawm); fb.ld_rawm = s.rows_m;
    fb.P = Pf; fb.part = partial(Pf, H * NS); fb.used_raw = (int)s.used_a; fb.used_rawm = (int)s.used_m;
    for (int i = 0; i < 4; ++i) {
      fb.col[i] = (int)s.col[i];
      fb.from_mag[i] = s.mag[i];
    }
    check(qpam_pam_front_bwd(&fb, st), "qpam_pam_front_bwd");
    Tensor fsum = at::empty({H * NS}, f32o);
    sum(fb.part, Pf, H * NS, H * NS, fsum);
    const Tensor dxn2 = at::mm(d_raw, sv[W_FRONT]);
    const Tensor dw_front = at::mm(d_raw.t(), sv[XN2].view({N, 2 * D}));
    Tensor dmag, dw_mag;
    if (s.rows_m) {
      dmag = at::mm(d_rawm, sv[W_MAG]);
      dw_mag = at::mm(d_rawm.t(), sv[MAG]);
    }
    // ---- second norm, residual, channel mix
    Tensor dx1 = at::empty_like(x), dmixed = at::empty({N, 2 * D}, o);
    const int Pn = parts_of((N + 3) / 4, 4);
    part = partial(Pn, D + 1);
    check(qpam_cnorm_res_bwd(sv[X1].data_ptr(), fptr(p[N2]), dxn2.data_ptr(), ptr(dmag), dx2.data_ptr(), sv[MIXED].data_ptr(), fptr(p[CGU_SCALE]), dx1.data_ptr(),
                             dmixed.data_ptr(), part, Pn, N, (int)D, eps, st),
          "qpam_cnorm_res_bwd");
    sum(part, Pn, D + 1, D, g[N2]);
    sum(part + D, Pn, D + 1, 1, g[CGU_SCALE]);
    const Tensor dgated = at::mm(dmixed, sv[W_DOWN]);
    const Tensor dw_down = at::mm(dmixed.t(), sv[GATED]);
    Tensor dgu = at::empty({N, 4 * s.hidden}, o);
    const int Pa = qpam_act_gate_bwd_parts(N, (int)s.hidden);
    const bool swish = p[ACT_BETA].defined();
    const int64_t ldp = swish ? 2 * s.hidden : s.hidden;
    part = partial(Pa, ldp);
    check(qpam_act_gate_bwd(sv[GATE].data_ptr(), sv[UP].data_ptr(), dgated.data_ptr(), fptr(p[ACT_BIAS]), fptr(p[ACT_BETA]), dgu.data_ptr(), part, Pa, N, (int)s.hidden, st),
          "qpam_act_gate_bwd");
    sum(part, Pa, ldp, s.hidden, g[ACT_BIAS]);
    if (swish) sum(part + s.hidden, Pa, ldp, s.hidden, g[ACT_BETA]);
    const Tensor dxn = at::mm(dgu, sv[W_GU]);
    const Tensor dw_gu = at::mm(dgu.t(), sv[XN].view({N, 2 * D}));
    Tensor dx = at::empty_like(x);
    part = partial(Pn, D + 1);
    check(qpam_cnorm_res_bwd(x.data_ptr(), fptr(p[N1]), dxn.data_ptr(), nullptr, dx1.data_ptr(), nullptr, nullptr, dx.data_ptr(), nullptr, part, Pn, N, (int)D, eps, st),
          "qpam_cnorm_res_bwd");
    sum(part, Pn, D + 1, D, g[N1]);
    // ---- parameters
    check(qpam_colsum(sums.data(), (int)sums.size(), st), "qpam_colsum");
    check(qpam_front_params(fptr(fsum), (int)H, (int)K, fptr(g[DT_BIAS]), fptr(g[DT_B]), fptr(g[DT_OFF]), fptr(g[PG_B]), fptr(g[PHASE_B]), fptr(g[SCORE_B]), st),
          "qpam_front_params");
    PackList l;
    weight_items(l, s, g, dw_gu, dw_down, dw_front, dw_mag, dw_o);
    check(qpam_unpack_block(l.it, l.n, st), "qpam_unpack_block");
    variable_list r = {dx};
    for (const Tensor& t : g)
      if (t.defined()) r.push_back(t);
    r.resize(r.size() + 9);                   // rope and the plain arguments
    return r;
  }
};

// Rows and columns of parameter i (1-D parameters: their length by one).
std::pair<int64_t, int64_t> param_shape(int i, const Shape& s) {
  switch (i) {
    case N1: case N2: return {s.D, 1};
    case GATE_R: case GATE_I: case UP_R: case UP_I: return {s.hidden, s.D};
    case DOWN_R: case DOWN_I: return {s.D, s.hidden};
    case ACT_BIAS: case ACT_BETA: return {s.hidden, 1};
    case CGU_SCALE: case PAM_SCALE: return {1, 1};
    case QKV_R: case QKV_I: return {3 * s.inner, s.D};
    case O_R: case O_I: return {s.D, s.inner};
    case DT_W: return {s.H, 2 * s.D};
    case DT_B: case DT_BIAS: case PG_B: return {s.H, 1};
    case DT_OFF: return {s.K, 1};
    case PG_W: return {s.H, s.mag[1] ? s.D : 2 * s.D};
    case PHASE_W: case SCORE_W: return {s.H * s.K, s.mag[2] ? s.D : 2 * s.D};
    default: return {s.H * s.K, 1};           // PHASE_B, SCORE_B
  }
}
constexpr int64_t bits(std::initializer_list<int> l) {
  int64_t b = 0;
  for (int i : l) b |= (int64_t)1 << i;
  return b;
}

// The operators this node stands for check their operands one by one; the kernels behind it take pointers and the sizes of x,
// H, d and K, so all of it is checked here, before the first launch.
std::tuple<Tensor, Tensor> block(const Tensor& x, const std::vector<OptTensor>& params, const OptTensor& rope_, int64_t H, int64_t d, int64_t K, bool pg_content,
                                 bool routing_content, double gamma_floor, int64_t offset) {
  QH_REQUIRE((int64_t)params.size() == N_PARAMS, "block: ", (int)N_PARAMS, " parameters expected");
  QH_REQUIRE(x.scalar_type() == at::kBFloat16 && x.dim() == 4 && x.size(3) == 2 && x.size(0) > 0 && x.size(1) > 0,
             "block: bfloat16 x [B,T,D,2] expected; got ", shape(x));
  QH_REQUIRE(d == 64 && H >= 1 && H <= 64 && K >= 1 && K <= QPAM_MAX_STATES, "block: d=", d, ", H=", H, ", K=", K, " are not covered");
  QH_REQUIRE(x.size(2) % 4 == 0 && x.size(2) <= 768, "block: the channel count must be a multiple of 4 up to 768; got ", x.size(2));
  variable_list p(N_PARAMS), present_params;
  int64_t present = 0;
  for (int i = 0; i < N_PARAMS; ++i) {
    if (!params[i].has_value()) continue;
    QH_REQUIRE(params[i]->device() == x.device() && params[i]->scalar_type() == at::kFloat, "block: parameters must be float32 on x's device");
    p[i] = dense(*params[i]);
    present_params.push_back(p[i]);
    present |= (int64_t)1 << i;
  }
  const int64_t gsp = bits({PG_W, PG_B}), routing = bits({DT_OFF, PHASE_W, PHASE_B}), score = bits({SCORE_W, SCORE_B}), optional = gsp | routing | score | bits({ACT_BETA});
  const int64_t all = ((int64_t)1 << N_PARAMS) - 1;
  const auto whole = [&](int64_t group) { return (present & group) == 0 || (present & group) == group; };
  QH_REQUIRE((present | optional) == all && whole(gsp) && whole(score) && (present & routing) == (K > 1 ? routing : 0) && (K > 1 || !(present & score)),
             "block: parameters are missing or do not go together");
  const Shape s(x, p, H, d, K, pg_content, routing_content);
  QH_REQUIRE(s.hidden > 0 && s.hidden % 4 == 0, "block: the hidden width must be a multiple of 4; got ", s.hidden);
  for (int i = 0; i < N_PARAMS; ++i) {
    if (!p[i].defined()) continue;
    const auto [rows, cols] = param_shape(i, s);
    QH_REQUIRE(p[i].numel() == rows * cols && (cols == 1 || (p[i].dim() == 2 && p[i].size(0) == rows)), "block: parameter ", i, " is ", shape(p[i]), ", [", rows, ", ",
               cols, "] expected for x ", shape(x));
  }
  OptTensor rope;
  if (rope_.has_value()) {
    QH_REQUIRE(rope_->device() == x.device() && rope_->dim() == 3 && rope_->size(1) == d && rope_->size(2) == 2 && offset + x.size(1) <= rope_->size(0),
               "block: the rotary table must be [P, ", d, ", 2] with P >= offset + T = ", offset + x.size(1), "; got ", shape(*rope_));
    rope = dense(rope_->detach().to(at::kFloat));
  }
  QH_REQUIRE(x.is_cuda(), "PAM kernels need CUDA tensors (there is no CPU path in this package)");
  auto out = Block::apply(dense(x), at::TensorList(present_params), rope, present, H, d, K, pg_content, routing_content, gamma_floor, offset);
  return {out[0], out[1]};
}

}  // namespace

void bind_block(pybind11::module_& m) {
  namespace py = pybind11;
  m.def("block", &block, py::call_guard<py::gil_scoped_release>());
}

}  // namespace qhost
