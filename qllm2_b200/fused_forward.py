"""Inference-only forward of a V11LM through packed weights and the fused block kernels.

A V11 block at inference is four projections with element-wise work between them.  The module
path (`V11Block.forward`, mirroring v11/model.py) spends most of a decode step launching ~80 small
operators per layer; here a layer is

    GEMM gate|up -> k_act_gate_packed -> GEMM down -> k_residual_cnorm
    -> GEMM qkv|gates (-> GEMM gates on |x|) -> k_pam_front -> scan or decode step -> GEMM o
    -> k_residual_cnorm (which also produces the next layer's pre-norm)

with every weight packed once: complex projections as one real block matrix acting on interleaved
(re, im) columns, the small gate/routing Linears appended as extra output columns of the qkv
projection (their planar-input weights permuted to the interleaved column order).  The GEMMs are
library calls (cuBLAS through `F.linear`); everything between them is this package's kernels.
Weights are snapshots: build a new `FusedForward` after changing the model's parameters.
"""
from __future__ import annotations

from types import SimpleNamespace
from typing import Optional

import torch
import torch.nn.functional as F
from torch.nn.modules.module import _has_any_global_hook

from . import _lib, ops
from ._lib import check, dtype_code, ptr, stream_ptr
from .fused_elementwise import _dense
from .model import ModSwish, V11LM, _stock_operators, build_rope_cache


def _f32(t: torch.Tensor) -> torch.Tensor:
    return _dense(t.detach().float())


def _is_table(m) -> bool:
    """Whether an embedding is its weight's rows and nothing else (no subclass, hook or renormalisation), laid out as the kernels
    read it; anything else is called as the module it is."""
    w = m.weight if type(m) is torch.nn.Embedding else None
    return (w is not None and m.max_norm is None and "forward" not in m.__dict__ and not m._forward_hooks and not m._forward_pre_hooks and
            not _has_any_global_hook() and w.is_contiguous() and w.data_ptr() % 16 == 0)


class PoolDecodeMix:
    """Sequence mixing at decode, as `FusedForward.hidden` takes it: one recurrent step in place on the pool slots of the live
    sequences.  slots [n]: integers of any type, those that name no slot are idle rows."""

    def __init__(self, pool, slots, head_dim):
        self.pool, self.slots, self.q_scale = pool, slots, head_dim ** -0.5

    def __call__(self, layer, q, k, v, gamma, coef):
        n, H, _, d, _ = q.shape
        K = gamma.shape[0]
        y = ops.pam_decode_step(self.pool, self.slots, q.view(n, H, d, 2), k.view(n, H, d, 2), v.view(n, H, d, 2),
                                gamma.view(K, n, H), None if coef is None else coef.view(K, n, H, 2), layer=layer)
        return y.view(n, -1)


class FusedForward:
    def __init__(self, model: V11LM, max_position: int = 8192):
        cfg = model.config
        why = self.unsupported_reason(model)
        if why:
            raise _lib.QPamError(f"FusedForward: {why}")
        p = next(model.parameters())
        self.model, self.cfg = model, cfg
        self.device, self.dtype = p.device, p.dtype
        self.D, self.H, self.d, self.K = cfg.dim, cfg.n_heads, cfg.head_dim, cfg.n_states
        self.inner = cfg.n_heads * cfg.head_dim
        self.rope = build_rope_cache(max_position, cfg.head_dim).to(self.device) if cfg.use_rope else None
        self.embed_scale = _f32(model.embed_norm.scale)
        self.out_scale = _f32(model.output_norm.scale)
        self.head_norm_scale = _f32(model.lm_head_norm.scale)
        hp = model.lm_head_proj
        self.w_head_proj = hp.block_weight().detach().to(self.dtype).contiguous()
        self.b_head_proj = (None if hp.bias_real is None else
                            torch.stack([hp.bias_real, hp.bias_imag], -1).reshape(-1).detach().to(self.dtype))
        self.w_vocab = torch.cat([model.embed.embed_real.weight, model.embed.embed_imag.weight], -1).detach().to(self.dtype).contiguous()
        self.layers = [self.pack_block(blk, self.dtype) for blk in model.blocks]
        self._step_layers = None
        self._native = _lib.host().Packed(self.D, self.H, self.d, self.K, self.layers, self.embed_scale, self.out_scale, self.rope)

    @staticmethod
    def unsupported_reason(model: V11LM) -> Optional[str]:
        cfg = model.config
        d = cfg.head_dim
        if not cfg.fused_qkv or cfg.qk_norm:
            return "needs fused_qkv without qk_norm"
        if cfg.use_learned_pos:
            return "learned position embeddings are not packed"
        if d < 4 or d > 128 or d & (d - 1) or cfg.n_heads > 64:
            return "head_dim must be a power of two in [4,128] and n_heads <= 64"
        if cfg.dim % 4 or (cfg.dim * cfg.expand) % 4:
            return "dim and dim*expand must be multiples of 4"
        if not _stock_operators(model):
            return "operators of the model were replaced or have hooks: they are called as modules"
        p = next(model.parameters())
        if not p.is_cuda or p.dtype not in (torch.float32, torch.bfloat16):
            return "needs a CUDA model in float32 or bfloat16"
        return None

    # ---------------------------------------------------------------------------------- packing
    @staticmethod
    def pack_block(blk, dtype) -> SimpleNamespace:
        """Packed weights of one V11Block (any device): `w_gu` [4*hidden, 2D] = gate | up block matrices,
        `w_down`, `w_front` = qkv block matrix followed by the gate / routing Linears that read the layer
        input (columns permuted from [re | im] planes to interleaved order; `cols[name]` = ("a", column)),
        `w_mag` = the Linears that read |x| (`cols[name]` = ("m", column)), `w_o`, and fp32 parameters."""
        cgu, pam = blk.cgu, blk.pam
        D, H, K, T = pam.dim, pam.num_heads, pam.n_states, dtype
        inner, device = pam.inner_dim, blk.norm1.scale.device
        L = SimpleNamespace()
        L.n1, L.n2 = _f32(blk.norm1.scale), _f32(blk.norm2.scale)
        L.hidden = cgu.gate_proj.out_dim
        L.w_gu = torch.cat([cgu.gate_proj.block_weight(), cgu.up_proj.block_weight()], 0).detach().to(T).contiguous()
        L.act_bias = _f32(cgu.act.bias)
        L.act_beta = _f32(cgu.act.beta) if isinstance(cgu.act, ModSwish) else None
        L.w_down = cgu.down_proj.block_weight().detach().to(T).contiguous()
        L.cgu_scale, L.pam_scale = _f32(blk.cgu_scale).view(1), _f32(blk.pam_scale).view(1)
        L.w_o = pam.o_proj.block_weight().detach().to(T).contiguous()
        L.dt_bias = _f32(pam.dt_bias)
        L.dt_off = _f32(pam.state_dt_offset) if K > 1 else None
        L.gamma_floor = float(pam.gamma_floor or 0.0)

        def interleaved_cols(lin):      # a Linear over [x_re | x_im] -> the same Linear over interleaved (re, im) columns
            w = lin.weight.detach()
            return w.view(w.shape[0], 2, D).transpose(1, 2).reshape(w.shape[0], 2 * D)

        rows_a, bias_a, rows_m, bias_m = [pam.qkv_proj.block_weight().detach()], [torch.zeros(6 * inner, device=device)], [], []
        L.cols = {}

        def add(name, lin, content_aware):
            if content_aware:
                L.cols[name] = ("a", sum(r.shape[0] for r in rows_a))
                rows_a.append(interleaved_cols(lin))
                bias_a.append(lin.bias.detach())
            else:
                L.cols[name] = ("m", sum(r.shape[0] for r in rows_m))
                rows_m.append(lin.weight.detach())
                bias_m.append(lin.bias.detach())

        add("dt", pam.dt_proj, True)
        if pam.use_gsp:
            add("pg", pam.protect_gate, pam.gate_content_aware)
        if K > 1:
            add("phase", pam.phase_proj, pam.routing_content_aware)
            if pam.state_compete:
                add("score", pam.score_proj, pam.routing_content_aware)
        n_a = sum(r.shape[0] for r in rows_a)
        pad = (-n_a) % 8            # rows of the projection output stay 16-byte aligned
        if pad:
            rows_a.append(torch.zeros(pad, 2 * D, device=device))
            bias_a.append(torch.zeros(pad, device=device))
        L.w_front = torch.cat([r.float() for r in rows_a], 0).to(T).contiguous()
        L.b_front = torch.cat([b.float() for b in bias_a], 0).to(T).contiguous()
        if rows_m and (-sum(r.shape[0] for r in rows_m)) % 8:
            pad = (-sum(r.shape[0] for r in rows_m)) % 8     # aligned output rows here too: a ragged width costs the GEMM its tensor-core kernels
            rows_m.append(torch.zeros(pad, D, device=device))
            bias_m.append(torch.zeros(pad, device=device))
        L.w_mag = torch.cat([r.float() for r in rows_m], 0).to(T).contiguous() if rows_m else None
        L.b_mag = torch.cat([b.float() for b in bias_m], 0).to(T).contiguous() if rows_m else None
        return L

    # ---------------------------------------------------------------------------------- kernels
    def _res_norm(self, z, delta, res_scale, norm_scale, want_mag=False):
        N = z.shape[0]
        xn = torch.empty_like(z)
        mag = torch.empty(N, self.D, dtype=z.dtype, device=z.device) if want_mag else None
        check(_lib.lib().qpam_residual_cnorm_fwd(ptr(z), ptr(delta), ptr(res_scale), ptr(norm_scale), ptr(xn), ptr(mag),
                                                 dtype_code(z.dtype), N, self.D, 1e-6, stream_ptr()), "qpam_residual_cnorm_fwd")
        return xn, mag

    def _front_args(self, a, L, raw, rawm, positions, offset, q_scale):
        """The operands of the gate / head-split kernels: raw, rawm are the outputs of w_front and w_mag (rawm None: not formed)."""
        es = raw.element_size()

        def col(name):
            src, off = L.cols.get(name, ("", 0))
            base = raw if src == "a" else rawm if src == "m" else None
            return (None, 0) if base is None else (base.data_ptr() + off * es, base.shape[1])

        a.qkv, a.ld_qkv = raw.data_ptr(), raw.shape[1]
        a.dt, a.ld_dt = col("dt")
        a.pg, a.ld_pg = col("pg")
        a.phase, a.ld_phase = col("phase")
        a.score, a.ld_score = col("score")
        a.dt_bias, a.state_dt_offset = ptr(L.dt_bias), ptr(L.dt_off)
        a.rope, a.rope_len = ptr(self.rope), 0 if self.rope is None else self.rope.shape[0]
        a.positions, a.offset = ptr(positions), int(offset)
        a.gamma_floor, a.q_scale = L.gamma_floor, float(q_scale)
        a.H, a.d, a.K, a.io_dtype = self.H, self.d, self.K, dtype_code(raw.dtype)

    def _front(self, L, raw, rawm, B, T, positions, offset, q_scale):
        H, d, K = self.H, self.d, self.K
        dev, dt = raw.device, raw.dtype
        q, k, v = (torch.empty(B, H, T, d, 2, dtype=dt, device=dev) for _ in range(3))
        gamma = torch.empty(K, B, H, T, dtype=torch.float32, device=dev)
        coef = torch.empty(K, B, H, T, 2, dtype=torch.float32, device=dev) if K > 1 else None
        a = _lib.FrontArgs()
        self._front_args(a, L, raw, rawm, positions, offset, q_scale)
        a.q, a.k, a.v, a.gamma, a.coef = ptr(q), ptr(k), ptr(v), ptr(gamma), ptr(coef)
        a.B, a.T = B, T
        check(_lib.lib().qpam_pam_front_fwd(a, stream_ptr()), "qpam_pam_front_fwd")
        return q, k, v, gamma, coef

    def _decodes_in_place(self, mix, T) -> bool:
        """Whether one launch forms q, k, v and the gates of a token and does the recurrent step on the pool of `mix`.  Only for
        `PoolDecodeMix` itself: any other object, a subclass too, may do something else when it is called."""
        if T != 1 or type(mix) is not PoolDecodeMix:
            return False
        pool = mix.pool
        return (pool.device == self.device and self.dtype == pool.dtype == torch.bfloat16 and self.d == 64 and self.D % 8 == 0 and
                pool.is_contiguous() and pool.data_ptr() % 16 == 0 and tuple(pool.shape[1:]) == (len(self.layers), self.K, self.H, 64, 64, 2))

    def _decode(self, li, L, raw, mag, positions, offset, mix, slots):
        n = raw.shape[0]
        a = _lib.DecodeFrontArgs()
        self._front_args(a.f, L, raw, None, positions, offset, mix.q_scale)
        a.mag_row[:] = [L.cols[name][1] if L.cols.get(name, "?")[0] == "m" else -1 for name in ("dt", "pg", "phase", "score")]
        a.mag, a.w_mag, a.b_mag, a.D = ptr(mag), ptr(L.w_mag), ptr(L.b_mag), self.D
        y = torch.empty(n, self.inner * 2, dtype=raw.dtype, device=raw.device)
        check(_lib.lib().qpam_decode_front(mix.pool.data_ptr(), mix.pool.shape[0], mix.pool.shape[1], li, ptr(slots), a, ptr(y), n, stream_ptr()),
              "qpam_decode_front")
        return y

    # ---------------------------------------------------------------------------------- forward
    @torch.no_grad()
    def hidden(self, ids: torch.Tensor, mix, positions: Optional[torch.Tensor] = None, offset: int = 0):
        """Run the blocks over ids [B, T]; `mix(layer, q, k, v, gamma, coef) -> y [B*T, inner*2]` is the
        sequence-mixing step (a scan at prefill, the recurrent step at decode; `PoolDecodeMix` is the latter, and may be
        done in one launch with what it takes instead of being called).  Returns the final residual stream normalised by
        output_norm, [B*T, D, 2]."""
        m, D = self.model, self.D
        B, T = ids.shape
        N = B * T
        if self.rope is not None and positions is None and offset + T > self.rope.shape[0]:
            raise _lib.QPamError("position beyond max_position of this FusedForward")
        if positions is not None:
            positions = positions.reshape(-1).to(torch.int64).contiguous()
        z = torch.stack([m.embed.embed_real(ids), m.embed.embed_imag(ids)], dim=-1).reshape(N, D, 2).to(self.dtype)
        z, _ = self._res_norm(z, None, None, self.embed_scale)          # embed_norm
        xn, _ = self._res_norm(z, None, None, self.layers[0].n1)
        lib = _lib.lib()
        slots = None                                                    # of a step that is done in one launch with what it takes
        if self._decodes_in_place(mix, T):
            slots = mix.slots.to(device=self.device, dtype=torch.int32).contiguous()
            if slots.numel() != N:
                raise _lib.QPamError("slot_ids must have one entry per sequence")
        for li, L in enumerate(self.layers):
            gu = F.linear(xn.view(N, 2 * D), L.w_gu)                      # [N, 4*hidden]
            gated = torch.empty(N, L.hidden, 2, dtype=z.dtype, device=z.device)
            check(lib.qpam_act_gate_packed_fwd(ptr(gu), gu.shape[1], dtype_code(gu.dtype), ptr(L.act_bias), ptr(L.act_beta),
                                               ptr(gated), N, L.hidden, stream_ptr()), "qpam_act_gate_packed_fwd")
            dn = F.linear(gated.view(N, 2 * L.hidden), L.w_down)
            xn2, mag = self._res_norm(z, dn, L.cgu_scale, L.n2, want_mag=L.w_mag is not None)
            raw = F.linear(xn2.view(N, 2 * D), L.w_front, L.b_front)
            if slots is not None:
                y = self._decode(li, L, raw, mag, positions, offset, mix, slots)      # [N, inner*2]
            else:
                rawm = F.linear(mag, L.w_mag, L.b_mag) if L.w_mag is not None else None
                q, k, v, gamma, coef = self._front(L, raw, rawm, B, T, positions, offset, mix.q_scale)
                y = mix(li, q, k, v, gamma, coef)
            o = F.linear(y, L.w_o)
            nxt = self.layers[li + 1].n1 if li + 1 < len(self.layers) else self.out_scale
            xn, _ = self._res_norm(z, o, L.pam_scale, nxt)
        return xn                                                          # output_norm(z)

    @torch.no_grad()
    def head_hidden(self, xn: torch.Tensor) -> torch.Tensor:
        """lm_head_norm(lm_head_proj(.)) of rows [n, D, 2] already normalised by output_norm."""
        n = xn.shape[0]
        h = F.linear(xn.reshape(n, 2 * self.D), self.w_head_proj, self.b_head_proj).view(n, self.D, 2)
        h, _ = self._res_norm(h, None, None, self.head_norm_scale)
        return h

    @torch.no_grad()
    def prefill(self, ids, pool, slots, cu=None, positions=None, resumed=None):
        """Absorb prompts: ids [B, T] (cu None: a prompt per row; otherwise the pieces of one packed row, cu int32 [S+1]) into the
        states of `slots` int32 [S] of `pool` [n_slots, L, K, H, d, d, 2].  resumed float32 [S]: 1 for pieces that continue from
        their slot's state.  Returns what `hidden` does.  (csrc/host/forward.cpp: the same launches as `hidden` around a scan,
        ~15 per block; issuing them from Python took longer than the GPU needs for a few hundred tokens.)"""
        er, ei = self.model.embed.embed_real, self.model.embed.embed_imag
        if _is_table(er) and _is_table(ei):
            return self._native.prefill(er.weight, ei.weight, None, ids, pool, slots, cu, positions, resumed)
        return self._native.prefill(None, None, torch.stack([er(ids), ei(ids)], dim=-1), ids, pool, slots, cu, positions, resumed)

    # ---------------------------------------------------------------------------------- decode step for few rows
    def step_supported(self, n: int) -> bool:
        """Whether `step` covers a batch of n rows: few enough that the weights' bytes, not the arithmetic, set the
        time (there the step reads half of them in a third of the launches), bf16 weights, head dim 64."""
        er, ei = self.model.embed.embed_real, self.model.embed.embed_imag
        return (self.dtype == torch.bfloat16 and _is_table(er) and _is_table(ei) and er.weight.dtype == ei.weight.dtype == torch.bfloat16 and
                bool(_lib.lib().qpam_step_supported(n, self.D, self.H, self.d, self.K, self.layers[0].hidden, self.w_vocab.shape[0])))

    def _pack_step_layers(self):
        H, inner = self.H, self.inner
        arr = (_lib.StepLayer * len(self.layers))()
        for s, L in zip(arr, self.layers):
            for name in ("w_gu", "w_down", "w_front", "b_front", "w_mag", "b_mag", "w_o", "n1", "n2", "act_bias", "act_beta", "cgu_scale",
                         "pam_scale", "dt_bias"):
                setattr(s, name, ptr(getattr(L, name)))
            s.dt_off = ptr(L.dt_off)
            s.gamma_floor = L.gamma_floor
            rows_a = L.w_front.shape[0] - 6 * inner
            for name in ("dt", "pg", "phase", "score"):
                src, off = L.cols.get(name, ("", -1))
                setattr(s, "col_" + name, off - 6 * inner if src == "a" else rows_a + off if src == "m" else -1)
        return arr

    @torch.no_grad()
    def step(self, ids, positions, slots, pool, logits: bool = False):
        """One decode step of the whole model (qpam_step_fwd): ids, positions int64 [n], slots int32 [n], `pool`
        [n_slots, L, K, H, d, d, 2] updated in place.  Returns the arg-max ids [n], or bf16 logits [n, V]."""
        if self._step_layers is None:
            self._step_layers = self._pack_step_layers()
        n, V, L0 = ids.numel(), self.w_vocab.shape[0], self.layers[0]
        dev, emb = self.device, self.model.embed
        a = _lib.StepArgs()
        a.layers = self._step_layers
        er, ei = emb.embed_real.weight, emb.embed_imag.weight
        a.embed_real, a.embed_imag, a.w_head, a.b_head, a.w_vocab = ptr(er), ptr(ei), ptr(self.w_head_proj), ptr(self.b_head_proj), ptr(self.w_vocab)
        a.embed_scale, a.out_scale, a.head_norm_scale, a.rope = ptr(self.embed_scale), ptr(self.out_scale), ptr(self.head_norm_scale), ptr(self.rope)
        ids, positions, slots = ids.reshape(-1).contiguous(), positions.reshape(-1).to(torch.int64).contiguous(), slots.contiguous()
        a.ids, a.positions, a.slot_ids, a.pool = ptr(ids), ptr(positions), ptr(slots), ptr(pool)
        if slots.dtype != torch.int32 or slots.numel() != n or positions.numel() != n or ids.dtype != torch.int64:
            raise _lib.QPamError("step: ids / positions int64 [n] and slots int32 [n] expected")
        if pool.dim() != 7 or not pool.is_contiguous() or tuple(pool.shape[1:]) != (len(self.layers), self.K, self.H, self.d, self.d, 2):
            raise _lib.QPamError(f"step: state pool {tuple(pool.shape)} does not fit this model")
        a.n, a.n_layers, a.D, a.H, a.d, a.K, a.hidden, a.V = n, len(self.layers), self.D, self.H, self.d, self.K, L0.hidden, V
        a.rows_a, a.rows_m = L0.w_front.shape[0] - 6 * self.inner, 0 if L0.w_mag is None else L0.w_mag.shape[0]
        a.n_slots, a.rope_len, a.state_dtype, a.q_scale = pool.shape[0], 0 if self.rope is None else self.rope.shape[0], dtype_code(pool.dtype), self.d ** -0.5
        if logits:
            ld = (V + 7) // 8 * 8
            out = torch.empty(n, ld, dtype=torch.bfloat16, device=dev)
            a.logits, a.ld_logits = ptr(out), ld
        else:
            out = torch.empty(n, dtype=torch.int64, device=dev)
            a.next_ids = ptr(out)
        ws = torch.empty(_lib.lib().qpam_step_workspace_bytes(a), dtype=torch.uint8, device=dev)
        a.workspace, a.workspace_bytes = ptr(ws), ws.numel()
        check(_lib.lib().qpam_step_fwd(a, stream_ptr()), "qpam_step_fwd")
        return out[:, :V] if logits else out

    @torch.no_grad()
    def logits(self, lm: torch.Tensor) -> torch.Tensor:
        """Tied-head logits [n, V] (float32) of rows lm [n, D, 2]: Re(lm . conj(E)) as one real GEMM
        (v11/model.py:1136-1139); only the sampling path needs them."""
        Hm = torch.cat([lm[..., 0], lm[..., 1]], dim=-1)
        if Hm.dtype == torch.bfloat16 and self.w_vocab.dtype == torch.bfloat16:
            return ops.head_logits(Hm, self.w_vocab).float()       # the cross-entropy's tensor-core GEMM, bf16 tiles out
        return F.linear(Hm, self.w_vocab).float()

    @torch.no_grad()
    def greedy_next(self, lm: torch.Tensor) -> torch.Tensor:
        """argmax over the tied head for rows lm [n, D, 2] (no logits are formed)."""
        Hm = torch.cat([lm[..., 0], lm[..., 1]], dim=-1).contiguous()
        ids, _ = ops.head_argmax(Hm, self.w_vocab)
        return ids
