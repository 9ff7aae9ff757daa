"""The block as one native node against the block operator by operator (torch autograd in between), each against the fp32 block:
output, input gradient and every parameter's gradient, for each source of the gates and both activations.  The node's forward has
the bits of the operators with every state's output rounded to bf16 before the read-out (the form of their scan that keeps no
chunk states; with one state there is only one form)."""
import functools

import pytest
import torch

from qllm2_b200 import model as M
from qllm2_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"
CONFIGS = {
    "k1_magnitude": dict(n_states=1),
    "k3_content": dict(n_states=3, gate_content_aware=True),
    "k2_compete": dict(n_states=2, routing_content_aware=True, state_compete=True, phase_init="spread", gamma_floor=0.3),
    "k4_magnitude_scores": dict(n_states=4, gate_content_aware=True, state_compete=True, activation="modrelu"),
    "k1_plain": dict(n_states=1, use_gsp=False, use_rope=False),
}


@pytest.mark.parametrize("name", CONFIGS)
@pytest.mark.parametrize("B,T,dim,heads", [(2, 130, 64, 2), (1, 5, 388, 3), (3, 257, 768, 2), (2, 1531, 128, 12)])
def test_native_block_matches_operators(name, B, T, dim, heads, monkeypatch):
    torch.manual_seed(11)
    cfg = M.V11Config(vocab_size=64, dim=dim, n_heads=heads, head_dim=64, n_layers=1, dropout=0.0, gradient_checkpointing=False, max_seq_len=2048, **CONFIGS[name])
    blk = M.V11Block(cfg).to(DEV).train()
    with torch.no_grad():
        for k, p in blk.named_parameters():
            if k.endswith(("weight_real", "weight_imag")):
                p.normal_(0, (2 * p.shape[1]) ** -0.5)
            elif p.dim() == 2:
                p.normal_(0, 0.2 * p.shape[1] ** -0.5)
            elif k.endswith(("bias", "scale", "beta")) and p.dim() == 1:
                p.add_(torch.randn_like(p) * 0.1)
    x = torch.randn(B, T, dim, 2, device=DEV).bfloat16()
    dy = torch.randn(B, T, dim, 2, device=DEV).bfloat16()
    ds = None
    res = {}
    scan = ops.pam_scan
    for mode in ("native", "per_state", "operators", "fp32"):
        xi = (x.float() if mode == "fp32" else x).clone().requires_grad_(True)
        blk.zero_grad()
        hook = blk.norm1.register_forward_hook(lambda *a: None) if mode != "native" else None         # keeps the operators
        monkeypatch.setattr(ops, "pam_scan", functools.partial(scan, save_states=False) if mode == "per_state" else scan)
        with torch.autocast("cuda", dtype=torch.bfloat16, enabled=mode != "fp32"):
            assert blk._native_ok(xi, None) == (mode == "native")
            out, state = blk(xi)
        if ds is None:
            ds = torch.randn_like(state)
        torch.autograd.backward([out, state], [dy.to(out.dtype), ds.to(state.dtype)])
        if hook:
            hook.remove()
        res[mode] = [out.detach().float(), state.detach().float(), xi.grad.float()] + [p.grad for p in blk.parameters()]
    names = ["out", "state", "x"] + [k for k, _ in blk.named_parameters()]
    for i in (0, 1):                                                # the forward rounds where these operators do
        assert torch.equal(res["native"][i], res["per_state"][i])
    for n, a, b, ref in zip(names, res["native"], res["operators"], res["fp32"]):
        assert a is not None and torch.isfinite(a).all(), n
        err, err_ops = float((a - ref).norm() / ref.norm()), float((b - ref).norm() / ref.norm())
        # (scalars and biases are sums over all tokens that cancel to a few per cent of their terms)
        assert err <= max(2e-2 if ref.numel() > 16 else 1e-1, 1.5 * err_ops), (n, err, err_ops)
