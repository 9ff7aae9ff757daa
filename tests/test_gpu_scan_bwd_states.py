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


@pytest.mark.parametrize("dtype,K,T", [(torch.bfloat16, 1, 1), (torch.bfloat16, 1, 93), (torch.bfloat16, 1, 128), (torch.bfloat16, 3, 128),
                                       (torch.bfloat16, 2, 17), (torch.float32, 1, 64), (torch.float32, 2, 5)])
@pytest.mark.parametrize("state_grad", [False, True])
def test_one_chunk_alone_equals_packed(dtype, K, T, state_grad):
    """A batch of one-chunk sequences runs without carries; the same sequence described by cu_seqlens takes every launch."""
    g = torch.Generator(device=DEV).manual_seed(T + K)
    H, d = 3, 64
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)
    data = [(rnd(1, H, T, d, 2) * 0.09).to(dtype) for _ in range(3)] + [torch.sigmoid(rnd(K, 1, H, T) + 2)] + ([rnd(K, 1, H, T, 2)] if K > 1 else [])
    dy, ds = rnd(1, H, T, d, 2).to(dtype), rnd(K, 1, H, d, d, 2)
    res = []
    for cu in (None, torch.tensor([0, T], device=DEV, dtype=torch.int32)):
        leaves = [t.clone().requires_grad_() for t in data]
        y, s = ops.pam_scan(*leaves[:4], coef=leaves[4] if K > 1 else None, cu_seqlens=cu)
        res.append([y, s, *torch.autograd.grad([y, s] if state_grad else [y], leaves, [dy, ds] if state_grad else [dy])])
    for a, b in zip(*res):
        assert torch.isfinite(a).all() and torch.equal(a, b)
