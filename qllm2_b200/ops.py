"""torch-facing wrappers of the C ABI: the scan through its native nodes (csrc/host), the rest over raw device pointers.

torch is used here for what it is good at on this path -- owning device memory, the current
stream and autograd bookkeeping.  All arithmetic happens in libqllm2_pam_b200.so.
"""
from __future__ import annotations

import ctypes as C
from typing import Optional

import torch

from . import _lib
from ._lib import CEArgs, ScanArgs, check, dtype_code, ptr, stream_ptr

GAMMA_EPS = 1e-6


def _require_cuda(*ts):
    for t in ts:
        if t is not None and not t.is_cuda:
            raise _lib.QPamError("PAM kernels need CUDA tensors (there is no CPU path in this package)")


def _workspace(nbytes: int, device) -> torch.Tensor:
    return torch.empty(max(int(nbytes), 256), dtype=torch.uint8, device=device)


# --------------------------------------------------------------------------------------- tracing
class _Recorded(torch.autograd.Function):
    """A native call as one operator of a torch.jit trace.  A trace records torch operators; the launches of a native call are
    not among them, and replayed it would hand out its outputs' memory as allocated."""

    @staticmethod
    def forward(ctx, call, *tensors):
        ctx.call = call
        ctx.save_for_backward(*tensors)
        ctx.set_materialize_grads(False)
        return call(*tensors)

    @staticmethod
    def backward(ctx, *grads):
        leaves = [None if t is None else t.detach().requires_grad_(need) for t, need in zip(ctx.saved_tensors, ctx.needs_input_grad[1:])]
        with torch.enable_grad():
            outs = ctx.call(*leaves)
        pairs = [(o, g) for o, g in zip(outs if isinstance(outs, tuple) else (outs,), grads) if g is not None]
        wanted = [t for t in leaves if t is not None and t.requires_grad]
        got = iter(torch.autograd.grad([o for o, _ in pairs], wanted, [g for _, g in pairs], allow_unused=True))
        return (None, *(next(got) if t is not None and t.requires_grad else None for t in leaves))


def recorded(call, *tensors):
    """call(*tensors) as one operator of the trace that is being taken."""
    return _Recorded.apply(call, *tensors)


#: torch.jit.is_tracing without its Python frames: asked at every call
is_tracing = torch._C._is_tracing


# --------------------------------------------------------------------------------------- scan
def _scan_args(q, k, v, gamma, coef, s0, cu_seqlens, y, s_final, q_scale, eps, chunk):
    B, H, T, d = q.shape[0], q.shape[1], q.shape[2], q.shape[3]
    K = gamma.shape[0]
    S = B if cu_seqlens is None else cu_seqlens.numel() - 1
    a = ScanArgs()
    a.q, a.k, a.v = ptr(q), ptr(k), ptr(v)
    a.gamma, a.coef, a.s0, a.cu_seqlens = ptr(gamma), ptr(coef), ptr(s0), ptr(cu_seqlens)
    a.y, a.s_final = ptr(y), ptr(s_final)
    a.B, a.H, a.T, a.d, a.K, a.S = B, H, T, d, K, S
    a.chunk, a.io_dtype = int(chunk), dtype_code(q.dtype)
    a.q_scale, a.gamma_eps = float(q_scale), float(eps)
    return a


def pam_scan(q, k, v, gamma, *, coef=None, s0=None, cu_seqlens=None, head_dim: Optional[int] = None,
             eps: float = GAMMA_EPS, chunk: int = 64, save_states: bool = True, token_major: bool = False):
    """Chunked dual-form PAM scan on the GPU.  (token_major=True returns y as [B, T, H*d, 2], the head merge
    of v11/model.py:835-836, straight from the last kernel where that kernel can write it.)

    q, k, v  [B,H,T,d,2] (float32 or bfloat16; q unscaled -- it is multiplied by head_dim**-0.5
             inside, as V11PAMLayer._forward_chunked_head does, v11/model.py:381-382)
    gamma    [B,H,T] or [K,B,H,T] decay in (0,1];  coef optional [K,B,H,T,2] read-out weights
    s0       optional [K,S,H,d,d,2] initial state;  cu_seqlens optional int32 [S+1] (then B == 1)
    Returns (y [B,H,T,d,2] in q's dtype, s_final float32 [K,S,H,d,d,2]).

    Checks, autograd node and launches are native (csrc/host/scan.cpp).  K = 2..4 states in bf16 at d = 64:
    y = sum_k c_k y^(k), where y^(k) is the single-state scan with decay gamma^(k) on the same q, k, v (the fused K-state form
    of the reference, v11/model.py:657-781, is algebraically this sum), through the fused K-state kernels, forward and backward.
    Without read-out weights (coef) and with gradients: one output kernel per state, whose dq, dk, dv the backward accumulates
    in place.  save_states=False with gradients, or more states than four: one single-state scan per state.
    """
    if not is_tracing():
        y, s = _lib.host().pam_scan(q, k, v, gamma, coef, s0, cu_seqlens, head_dim or 0, eps, chunk, save_states, token_major)
    else:
        if torch.is_autocast_enabled("cuda") and torch.get_autocast_dtype("cuda") == torch.bfloat16:
            q, k, v = q.bfloat16(), k.bfloat16(), v.bfloat16()       # what autocast decides belongs to the trace, not to its replay
        each = (gamma.dim() == 4 and gamma.shape[0] > 1 and (not save_states or gamma.shape[0] > _lib.MAX_STATES) and q.dtype == torch.bfloat16 and
                q.shape[3] == 64 and torch.is_grad_enabled() and any(t is not None and t.requires_grad for t in (q, k, v, gamma, coef, s0)))
        y, s = (None, None) if each else recorded(
            lambda q, k, v, gamma, coef, s0, cu: _lib.host().pam_scan(q, k, v, gamma, coef, s0, cu, head_dim or 0, eps, chunk, save_states, token_major),
            q, k, v, gamma, coef, s0, cu_seqlens)
    if y is not None:
        return y, s
    # K tensor-core states recomputed in the backward, or more of them than the fused kernels take: one scan per state, autograd
    # sums the gradients
    gamma = gamma.float()
    ys, finals = zip(*(pam_scan(q, k, v, gamma[kk:kk + 1], s0=None if s0 is None else s0[kk:kk + 1], cu_seqlens=cu_seqlens, head_dim=head_dim,
                                eps=eps, chunk=chunk, save_states=save_states) for kk in range(gamma.shape[0])))
    if coef is None:
        y = ys[0]
        for yk in ys[1:]:
            y = y + yk
        return (_merge_heads(y) if token_major else y), torch.cat(finals, dim=0)
    from .fused_elementwise import state_combine
    return state_combine(coef.float(), ys, token_major=token_major), torch.cat(finals, dim=0)


def _merge_heads(y):
    B, H, T, d = y.shape[:4]
    return y.transpose(1, 2).reshape(B, T, H * d, 2)


@torch.no_grad()
def pam_scan_states(k, v, gamma, s0=None, cu_seqlens=None, *, eps: float = GAMMA_EPS, chunk: int = 64):
    """Final state(s) of the scan only -- S after the last token, float32 [K,S,H,d,d,2] -- without forming Y:
    the chunk-local sums and the inter-chunk carry run, the output kernel does not (about a third of a forward
    scan).  k, v [B,H,T,d,2]; gamma [B,H,T] or [K,B,H,T]; s0 / cu_seqlens as in `pam_scan`."""
    L = _lib.lib()
    _require_cuda(k, v, gamma)
    if gamma.dim() == 3:
        gamma = gamma.unsqueeze(0)
    if k.dtype != v.dtype:
        dt = torch.promote_types(k.dtype, v.dtype)
        k, v = k.to(dt), v.to(dt)
    k, v = k.contiguous(), v.contiguous()
    gamma = gamma.float().contiguous()
    B, H, T, d = k.shape[:4]
    K = gamma.shape[0]
    if k.shape != v.shape or k.dim() != 5 or k.shape[-1] != 2 or tuple(gamma.shape) != (K, B, H, T):
        raise _lib.QPamError(f"pam_scan_states: k/v must be one [B,H,T,d,2] shape and gamma [K,B,H,T]; got {tuple(k.shape)}, "
                             f"{tuple(v.shape)}, {tuple(gamma.shape)}")
    if cu_seqlens is not None:
        if B != 1:
            raise _lib.QPamError("packed mode (cu_seqlens) needs B == 1")
        cu_seqlens = cu_seqlens.to(device=k.device, dtype=torch.int32).contiguous()
    S = B if cu_seqlens is None else cu_seqlens.numel() - 1
    if s0 is not None:
        if s0.numel() != K * S * H * d * d * 2:
            raise _lib.QPamError(f"s0 must be [K,S,H,d,d,2] = {(K, S, H, d, d, 2)}, got {tuple(s0.shape)}")
        s0 = s0.float().contiguous()
    s_final = torch.empty(K, S, H, d, d, 2, dtype=torch.float32, device=k.device)
    a = _scan_args(k, k, v, gamma, None, s0, cu_seqlens, None, s_final, d ** -0.5, eps, chunk)   # q is not read
    ws = _workspace(L.qpam_scan_workspace_bytes(C.byref(a), 0), k.device)
    a.workspace, a.workspace_bytes = ws.data_ptr(), ws.numel()
    check(L.qpam_scan_fwd(C.byref(a), stream_ptr()), "qpam_scan_fwd")
    return s_final


@torch.no_grad()
def pam_scan_tokens(q, k, v, gamma, coef=None, s0=None, cu_seqlens=None, *, head_dim=None, eps: float = 1e-6,
                    chunk: int = 64):
    """Inference form of `pam_scan`: same arguments, but Y comes back token-major, [B, T, H*d, 2] -- the layout
    the output projection reads (the head merge of v11/model.py:835-836) -- and nothing is kept for a backward
    pass (K phase-routed states in bf16 at d = 64 then run the fused K-state output kernel)."""
    if not is_tracing():
        return _lib.host().pam_scan_tokens(q, k, v, gamma, coef, s0, cu_seqlens, head_dim or 0, eps, chunk)
    return recorded(lambda q, k, v, gamma, coef, s0, cu: _lib.host().pam_scan_tokens(q, k, v, gamma, coef, s0, cu, head_dim or 0, eps, chunk),
                    q, k, v, gamma, coef, s0, cu_seqlens)


# --------------------------------------------------------------------------------------- decode
def pam_decode_step(state_pool, slot_ids, q_scaled, k, v, gamma, coef=None, *, layer: int = 0):
    """One recurrent step, in place on ``state_pool`` [n_slots, L, K, H, d, d, 2].

    q_scaled, k, v [n,H,d,2]; gamma [K,n,H] (or [n,H]); coef optional [K,n,H,2];
    slot_ids int32 [n].  Returns y [n,H,d,2].  (v11/model.py:927-965)
    """
    L = _lib.lib()
    _require_cuda(state_pool, q_scaled, k, v, gamma, coef)
    n_slots, n_layers, K, H, d = state_pool.shape[:5]
    if gamma.dim() == 2:
        gamma = gamma.unsqueeze(0)
    if coef is not None and coef.dim() == 3:
        coef = coef.unsqueeze(0)
    gamma = gamma.float().contiguous()
    coef = None if coef is None else coef.float().contiguous()
    k, v = k.to(q_scaled.dtype), v.to(q_scaled.dtype)
    q_scaled, k, v = q_scaled.contiguous(), k.contiguous(), v.contiguous()
    slot_ids = slot_ids.to(device=state_pool.device, dtype=torch.int32).contiguous()
    n = q_scaled.shape[0]
    if not (q_scaled.shape == k.shape == v.shape == (n, H, d, 2)):
        raise _lib.QPamError(f"q, k, v must be [n,H,d,2] = {(n, H, d, 2)}; got {tuple(q_scaled.shape)}, {tuple(k.shape)}, {tuple(v.shape)}")
    if slot_ids.numel() != n:
        raise _lib.QPamError("slot_ids must have one entry per sequence")
    if coef is not None and coef.shape != (K, n, H, 2):
        raise _lib.QPamError(f"coef shape {tuple(coef.shape)} != {(K, n, H, 2)}")
    if gamma.shape != (K, n, H):
        raise _lib.QPamError(f"gamma shape {tuple(gamma.shape)} != {(K, n, H)}")
    if not state_pool.is_contiguous():
        raise _lib.QPamError("state_pool must be contiguous")
    y = torch.empty_like(q_scaled)
    check(L.qpam_decode_step(state_pool.data_ptr(), dtype_code(state_pool.dtype), n_slots, n_layers, layer,
                             ptr(slot_ids), ptr(q_scaled), ptr(k), ptr(v), ptr(gamma), ptr(coef), ptr(y),
                             n, H, d, K, dtype_code(q_scaled.dtype), stream_ptr()), "qpam_decode_step")
    return y


def pam_pool_store(state_pool, slot_ids, states, *, layer: int = 0):
    """Write prefill states [K,S,H,d,d,2] (float32) into pool slots ``slot_ids`` [S]."""
    L = _lib.lib()
    _require_cuda(state_pool, states)
    n_slots, n_layers, K, H, d = state_pool.shape[:5]
    states = states.float().contiguous()
    S = states.shape[1]
    if states.shape != (K, S, H, d, d, 2) or slot_ids.numel() != S:
        raise _lib.QPamError(f"states must be [K,S,H,d,d,2] with one slot id per sequence; got {tuple(states.shape)}")
    slot_ids = slot_ids.to(device=state_pool.device, dtype=torch.int32).contiguous()
    check(L.qpam_pool_store(state_pool.data_ptr(), dtype_code(state_pool.dtype), n_slots, n_layers, layer,
                            ptr(slot_ids), ptr(states), S, H, d, K, stream_ptr()), "qpam_pool_store")


# --------------------------------------------------------------------------------------- CE
def _ce_args(h, w, targets, mask, ignore_index, v_offset=0):
    a = CEArgs()
    a.h, a.w, a.targets, a.mask = ptr(h), ptr(w), ptr(targets), ptr(mask)
    a.N, a.V, a.v_offset = h.shape[0], w.shape[0], int(v_offset)
    a.F, a.io_dtype = h.shape[1], dtype_code(h.dtype)
    a.ignore_index = int(ignore_index)
    return a


def ce_row_stats(h, w, targets, *, ignore_index=-100, v_offset=0):
    """Per-row shard statistics (max, sumexp, target logit, argmax) without forming logits."""
    L = _lib.lib()
    _require_cuda(h, w)
    h, w = h.contiguous(), w.contiguous()
    if h.dtype != w.dtype:
        w = w.to(h.dtype)
    if h.dim() != 2 or w.dim() != 2 or h.shape[1] != w.shape[1]:
        raise _lib.QPamError(f"h [N,F] and w [V,F] expected; got {tuple(h.shape)}, {tuple(w.shape)}")
    if targets is not None and (targets.dtype != torch.int64 or targets.numel() != h.shape[0]):
        raise _lib.QPamError("targets must be int64 with one entry per row of h")
    targets = None if targets is None else targets.contiguous()
    N = h.shape[0]
    f32 = dict(dtype=torch.float32, device=h.device)
    row_max, row_sum, row_tgt = torch.empty(N, **f32), torch.empty(N, **f32), torch.empty(N, **f32)
    row_arg = torch.empty(N, dtype=torch.int64, device=h.device)
    a = _ce_args(h, w, targets, None, ignore_index, v_offset)
    ws = _workspace(L.qpam_ce_workspace_bytes(C.byref(a), 0), h.device)
    a.workspace, a.workspace_bytes = ws.data_ptr(), ws.numel()
    check(L.qpam_ce_partial(C.byref(a), ptr(row_max), ptr(row_sum), ptr(row_tgt if targets is not None else None),
                            ptr(row_arg), stream_ptr()), "qpam_ce_partial")
    return row_max, row_sum, row_tgt, row_arg


def ce_finalize(h, w, targets, mask, stats, *, ignore_index=-100):
    """Combined stats -> dict(lse, per_token, loss_sum, denom, correct, tokens) (device tensors)."""
    L = _lib.lib()
    row_max, row_sum, row_tgt, row_arg = stats
    N = h.shape[0]
    f32 = dict(dtype=torch.float32, device=h.device)
    out = dict(lse=torch.empty(N, **f32), per_token=torch.empty(N, **f32), loss_sum=torch.zeros(1, **f32),
               denom=torch.ones(1, **f32), correct=torch.zeros(1, **f32), tokens=torch.zeros(1, **f32))
    a = _ce_args(h, w, targets, mask, ignore_index)
    ws = _workspace(256, h.device)
    a.workspace, a.workspace_bytes = ws.data_ptr(), ws.numel()
    check(L.qpam_ce_finalize(C.byref(a), ptr(row_max), ptr(row_sum), ptr(row_tgt), ptr(row_arg), ptr(out["lse"]),
                             ptr(out["per_token"]), ptr(out["loss_sum"]), ptr(out["denom"]), ptr(out["correct"]),
                             ptr(out["tokens"]), stream_ptr()), "qpam_ce_finalize")
    return out


def ce_backward(h, w, targets, mask, lse, grad_scale, denom, *, ignore_index=-100, v_offset=0, dh_ready_stream=None):
    """dH [N,F], dW [V,F] (dtype of h / w) for  grad_scale * loss_sum / denom.  `dh_ready_stream` (a
    torch.cuda.Stream) is made to wait until dH is complete while dW is still being formed on the current stream."""
    L = _lib.lib()
    dh = torch.empty_like(h)
    dw = torch.empty_like(w)
    a = _ce_args(h, w, targets, mask, ignore_index, v_offset)
    ws = _workspace(L.qpam_ce_workspace_bytes(C.byref(a), 1), h.device)
    a.workspace, a.workspace_bytes = ws.data_ptr(), ws.numel()
    side = None if dh_ready_stream is None else dh_ready_stream.cuda_stream
    check(L.qpam_ce_bwd_overlap(C.byref(a), ptr(lse), ptr(grad_scale), ptr(denom), ptr(dh), ptr(dw), stream_ptr(), side),
          "qpam_ce_bwd")
    return dh, dw


def head_logits(h, w):
    """Sampling decode head: bf16 logits [N, V] = h @ w^T (a view of rows padded to a multiple of 8 columns) on the
    tensor-core GEMM of the cross-entropy; h [N,F] and w [V,F] bfloat16 with 16-byte aligned rows
    (v11/model.py:1218-1221 forms the same product before its sampling block)."""
    L = _lib.lib()
    _require_cuda(h, w)
    h, w = h.contiguous(), w.contiguous()
    if h.dtype != torch.bfloat16 or w.dtype != torch.bfloat16 or h.dim() != 2 or w.dim() != 2 or h.shape[1] != w.shape[1]:
        raise _lib.QPamError(f"head_logits: bfloat16 h [N,F] and w [V,F] expected; got {tuple(h.shape)} {h.dtype}, {tuple(w.shape)} {w.dtype}")
    N, V = h.shape[0], w.shape[0]
    ld = (V + 7) // 8 * 8
    out = torch.empty(N, ld, dtype=torch.bfloat16, device=h.device)
    a = _ce_args(h, w, None, None, -100, 0)
    check(L.qpam_head_logits(C.byref(a), ptr(out), ld, stream_ptr()), "qpam_head_logits")
    return out[:, :V]


def head_argmax(h, w):
    """Greedy decode head: (ids int64 [N], best logit float32 [N]) of argmax_v (h @ w^T)."""
    row_max, _, _, row_arg = ce_row_stats(h, w, None)
    return row_arg, row_max


def sample_logits(logits, uniforms=None, *, temperature: float = 1.0, top_k: int = 0, top_p: float = 0.0,
                  repetition_penalty: float = 1.0, history=None, hist_len=None, slot_ids=None, append: bool = False,
                  return_stats: bool = False):
    """Draw one token per row of `logits` [n, V] on the device (one kernel; v11/model.py:1221-1244): temperature,
    repetition penalty over `history` (int64 [rows, cols] token ids; `hist_len` int32 [rows] valid entries per
    row, `slot_ids` int32 [n] maps logits rows to history rows), top-k, top-p, then the inverse-CDF draw of
    `uniforms` [n] (default: torch.rand on the logits' device, i.e. torch's generator).  `append=True` also writes
    the drawn id behind the row's history and advances `hist_len`.  Masses are float32, e^((x - max) / temperature): a
    token more than about 103 temperatures below the maximum has none.  Returns ids int64 [n] (and, with
    `return_stats`, float32 [n,4] = (max, kept mass, kept count, mass after top-k))."""
    L = _lib.lib()
    _require_cuda(logits)
    if logits.dim() != 2 or logits.dtype not in (torch.float32, torch.bfloat16):
        raise _lib.QPamError(f"sample_logits: logits must be [n, V] float32 or bfloat16, got {tuple(logits.shape)} {logits.dtype}")
    if logits.stride(1) != 1:
        logits = logits.contiguous()
    n, V = logits.shape
    dev = logits.device
    if uniforms is None:
        uniforms = torch.rand(n, device=dev, dtype=torch.float32)
    if uniforms.dtype != torch.float32 or uniforms.numel() != n or not uniforms.is_cuda:
        raise _lib.QPamError("sample_logits: uniforms must be a float32 CUDA tensor with one entry per row")
    rows = cols = ld = 0
    if history is not None:
        if history.dim() != 2 or history.dtype != torch.int64 or not history.is_cuda or history.stride(1) != 1:
            raise _lib.QPamError("sample_logits: history must be a 2-D int64 CUDA tensor with unit column stride")
        rows, cols, ld = history.shape[0], history.shape[1], history.stride(0)
        if slot_ids is None and rows < n:
            raise _lib.QPamError(f"sample_logits: history has {rows} rows for {n} rows of logits")
    if hist_len is not None and (history is None or hist_len.dtype != torch.int32 or hist_len.numel() != rows or not hist_len.is_cuda):
        raise _lib.QPamError("sample_logits: hist_len must be int32 [history rows] on the device")
    if slot_ids is not None and (slot_ids.dtype != torch.int32 or slot_ids.numel() != n or not slot_ids.is_cuda):
        raise _lib.QPamError("sample_logits: slot_ids must be int32 [n] on the device")
    if append and (history is None or hist_len is None):
        raise _lib.QPamError("sample_logits: append needs history and hist_len")
    if append and not hist_len.is_contiguous():
        raise _lib.QPamError("sample_logits: append advances hist_len in place, so it must be contiguous")
    uniforms = uniforms.contiguous()
    slot_ids = None if slot_ids is None else slot_ids.contiguous()
    hist_len = None if hist_len is None else hist_len.contiguous()
    ids = torch.empty(n, dtype=torch.int64, device=dev)
    stats = torch.empty(n, 4, dtype=torch.float32, device=dev) if return_stats else None
    need = L.qpam_sample_workspace_bytes(n, V)
    ws = _workspace(need, dev) if need else None
    check(L.qpam_sample_logits(logits.data_ptr(), dtype_code(logits.dtype), n, V, logits.stride(0), float(temperature), int(top_k),
                               float(top_p), float(repetition_penalty), ptr(slot_ids), ptr(history), rows, cols, ld,
                               ptr(hist_len), int(bool(append)), uniforms.data_ptr(), ids.data_ptr(), ptr(stats),
                               ptr(ws), need, stream_ptr()), "qpam_sample_logits")
    return (ids, stats) if return_stats else ids
