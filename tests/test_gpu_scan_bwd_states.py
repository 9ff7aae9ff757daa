"""Backward of the K-state scan in one kernel (bf16, d = 64) against the fp32 kernels on the same numbers: chunk edges, ragged
packed sequences, initial states, a state that forgets within a chunk, both layouts of the output gradient."""
import pytest
import torch

from qllm2_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("K,B,T,lengths,strong,tokens", [
    (2, 2, 1, None, False, True), (3, 1, 127, None, False, False), (4, 2, 128, None, True, True), (3, 2, 129, None, False, True),
    (2, 1, 700, (1, 0, 130, 128, 300, 141), False, False), (4, 1, 385, (257, 128), True, False), (3, 5, 640, None, True, True),
])
def test_bwd_of_all_states(K, B, T, lengths, strong, tokens):
    g = torch.Generator(device=DEV).manual_seed(K * 1000 + T)
    H, d = 3, 64
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)
    q, k, v = [(rnd(B, H, T, d, 2) * 0.09).bfloat16() for _ in range(3)]
    gamma = torch.sigmoid(rnd(K, B, H, T) + torch.tensor([1.0, 3.0, 5.0, 4.0], device=DEV)[:K, None, None, None])
    if strong:
        gamma[0] = gamma[0] * 0.3                     # e^-80 is passed well inside a chunk
    coef = rnd(K, B, H, T, 2)
    cu = None if lengths is None else torch.tensor([0, *lengths], device=DEV).cumsum(0).int()
    S = B if cu is None else len(lengths)
    s0 = rnd(K, S, H, d, d, 2) * 0.1
    dy, ds = rnd(B, H, T, d, 2).bfloat16(), rnd(K, S, H, d, d, 2) * 0.1
    res = []
    for dtype in (torch.bfloat16, torch.float32):
        leaves = [t.to(dtype).requires_grad_() for t in (q, k, v)] + [t.clone().requires_grad_() for t in (gamma, coef, s0)]
        tm = tokens and dtype is torch.bfloat16
        y, s = ops.pam_scan(*leaves[:4], coef=leaves[4], s0=leaves[5], cu_seqlens=cu, token_major=tm)
        dyt = dy.to(dtype)
        if tm:
            dyt = dyt.transpose(1, 2).reshape(y.shape)
        res.append(torch.autograd.grad([y, s], leaves, [dyt, ds]))
    for name, a, b in zip(("dq", "dk", "dv", "dgamma", "dcoef", "ds0"), *res):
        assert torch.isfinite(a).all(), name
        err = float((a.float() - b).norm() / b.norm())
        assert err < 1e-2, (name, err)
