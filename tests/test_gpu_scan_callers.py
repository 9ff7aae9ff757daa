"""Ways to call the scan and the loss that a native node in their place has to serve as the operators did."""
import pytest
import torch
import torch.autograd.forward_ad as fwAD

from qllm2_b200 import _lib, ops
from qllm2_b200 import model as M
from qllm2_b200.fused_ce import fused_linear_cross_entropy, linear_ce_stats

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _data(K, T=140, S=1):
    g = torch.Generator(device=DEV).manual_seed(K)
    q, k, v = [(torch.randn(1, 2, T, 64, 2, device=DEV, generator=g) * 0.1).bfloat16() for _ in range(3)]
    gamma = torch.sigmoid(torch.randn(K, 1, 2, T, device=DEV, generator=g) + 2)
    return q, k, v, gamma, torch.randn(K, S, 2, 64, 64, 2, device=DEV, generator=g)


@pytest.mark.parametrize("save_states", [True, False])
@pytest.mark.parametrize("token_major", [True, False])
def test_more_states_than_the_fused_kernels_take(save_states, token_major):
    """Five states without read-out weights: the sum of five scans, outputs, states and gradients."""
    q, k, v, gamma, s0 = _data(5, S=2)
    cu = torch.tensor([0, 60, 140], dtype=torch.int32)
    leaves = [t.clone().requires_grad_() for t in (q, k, v, gamma, s0)]
    y, s = ops.pam_scan(*leaves[:4], s0=leaves[4], cu_seqlens=cu, save_states=save_states, token_major=token_major)
    assert s.shape == (5, 2, 2, 64, 64, 2)
    dy = torch.randn(y.shape, device=DEV, generator=torch.Generator(device=DEV).manual_seed(9)).bfloat16()
    got = [y, s, *torch.autograd.grad([y, s], leaves, [dy, s0])]
    refs = [t.clone().requires_grad_() for t in (q, k, v, gamma, s0)]
    one = [ops.pam_scan(*refs[:3], refs[3][i:i + 1], s0=refs[4][i:i + 1], cu_seqlens=cu, token_major=token_major) for i in range(5)]
    y_ref, s_ref = sum(o[0].float() for o in one), torch.cat([o[1] for o in one])
    want = [y_ref, s_ref, *torch.autograd.grad([y_ref, s_ref], refs, [dy.float(), s0])]
    for a, b in zip(got, want):       # (bf16 sums of five terms in another order: a few roundings of 2^-9)
        assert float((a.float() - b.float()).norm() / b.float().norm()) < 1e-2


def test_read_out_of_more_states_is_refused():
    q, k, v, gamma, _ = _data(5)
    with pytest.raises(_lib.QPamError):
        ops.pam_scan(q.requires_grad_(), k, v, gamma, coef=torch.ones(5, 1, 2, 140, 2, device=DEV))
    with pytest.raises(_lib.QPamError):
        ops.pam_scan(q.detach(), k, v, gamma)


@pytest.mark.parametrize("which", range(6))
@pytest.mark.parametrize("call", ["scan", "token_major", "tokens"])
def test_forward_mode_is_refused(which, call):
    """Never silently without the tangent, whichever input carries one."""
    q, k, v, gamma, s0 = _data(3)
    args = [q, k, v, gamma, torch.ones(3, 1, 2, 140, 2, device=DEV), s0]
    fn = {"scan": ops.pam_scan, "tokens": ops.pam_scan_tokens}.get(call, lambda *a, **kw: ops.pam_scan(*a, token_major=True, **kw))
    with fwAD.dual_level():
        args[which] = fwAD.make_dual(args[which], torch.ones_like(args[which]))
        with pytest.raises(RuntimeError, match="forward-mode"):
            fn(*args[:4], coef=args[4], s0=args[5])


@pytest.mark.parametrize("K,grad,call", [(1, False, "scan"), (1, True, "scan"), (3, True, "scan"), (3, True, "token_major"), (3, False, "tokens"), (3, True, "recompute")])
def test_traced_scan_runs_its_kernels(K, grad, call):
    """A replayed trace on other inputs equals the call itself, gradients included."""
    q, k, v, gamma, _ = _data(K)
    coef = torch.randn(K, 1, 2, 140, 2, device=DEV, generator=torch.Generator(device=DEV).manual_seed(2)) if K > 1 else None
    kw = {"token_major": dict(token_major=True), "recompute": dict(save_states=False)}.get(call, {})
    fn = lambda q, k, v, gamma: (ops.pam_scan_tokens if call == "tokens" else ops.pam_scan)(q, k, v, gamma, coef=coef, **kw)
    inputs = [t.clone().requires_grad_(grad) for t in (q, k, v, gamma)]
    traced = torch.jit.trace(fn, inputs, check_trace=False)
    res = []
    for f in (traced, fn):
        leaves = [(t.detach() * 0.5).requires_grad_(grad) for t in inputs]
        y, s = f(*leaves)
        res.append([y, s, *(torch.autograd.grad([y, s], leaves, [torch.ones_like(y), torch.ones_like(s)]) if grad else ())])
    for a, b in zip(*res):
        assert torch.equal(a, b)


def test_traced_loss_and_block():
    g = torch.Generator(device=DEV).manual_seed(3)
    h, w = torch.randn(48, 64, device=DEV, generator=g).requires_grad_(), torch.randn(100, 64, device=DEV, generator=g).requires_grad_()
    t = torch.randint(0, 100, (48,), device=DEV, generator=g)
    traced = torch.jit.trace(fused_linear_cross_entropy, (h, w, t), check_trace=False)
    res = []
    for f in (traced, fused_linear_cross_entropy):
        leaves = [(x.detach() * 0.5).requires_grad_() for x in (h, w)]
        loss = f(*leaves, t)
        res.append([loss, *torch.autograd.grad(loss, leaves)])
    for a, b in zip(*res):
        assert torch.equal(a, b)
    torch.manual_seed(0)
    blk = M.V11Block(M.V11Config(vocab_size=64, dim=64, n_heads=1, head_dim=64, n_layers=1, dropout=0.0, max_seq_len=64)).to(DEV).requires_grad_(False)
    x = torch.randn(1, 40, 64, 2, device=DEV, generator=g).bfloat16()
    with torch.autocast("cuda", dtype=torch.bfloat16):
        traced = torch.jit.trace(lambda x: blk(x)[0], (x,), check_trace=False)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        want = blk(x * 0.5)[0]
        assert torch.equal(traced(x * 0.5), want)


def _off(t, elements=1):
    """The same values, `elements` behind an aligned address."""
    v = torch.empty(t.numel() + 8, dtype=t.dtype, device=t.device)[elements:elements + t.numel()].view(t.shape)
    return v.copy_(t)


@pytest.mark.parametrize("K,dtype", [(1, torch.bfloat16), (3, torch.bfloat16), (1, torch.float32), (2, torch.float32)])
@pytest.mark.parametrize("token_major", [False, True])
def test_operands_off_their_alignment(K, dtype, token_major):
    """Every operand one element behind an aligned address: the results of the aligned ones."""
    q, k, v, gamma, s0 = _data(K)
    data = [t.to(dtype) for t in (q, k, v)] + [gamma, s0] + ([torch.randn(K, 1, 2, 140, 2, device=DEV)] if K > 1 else [])
    res = []
    for place in (torch.clone, _off):
        leaves = [place(t).requires_grad_() for t in data]
        y, s = ops.pam_scan(*leaves[:4], s0=leaves[4], coef=leaves[5] if K > 1 else None, token_major=token_major)
        g = [place(torch.linspace(-1, 1, t.numel(), device=DEV).view(t.shape).to(t.dtype)) for t in (y, s)]
        res.append([y, s, *torch.autograd.grad([y, s], leaves, g)])
    for a, b in zip(*res):
        if dtype is torch.float32:
            assert torch.equal(a, b)
        else:                     # (an output gradient off its alignment takes the scalar kernels backward: bf16 rounding apart)
            assert float((a.detach().float() - b.detach().float()).norm() / a.detach().float().norm()) < 1e-2


def test_operands_on_other_devices_are_refused():
    """Host memory never reaches a kernel as a pointer."""
    q, k, v, gamma, s0 = _data(3)
    coef = torch.ones(3, 1, 2, 140, 2, device=DEV)
    for i in range(1, 6):
        a = [q, k, v, gamma, coef, s0]
        a[i] = a[i].cpu()
        with pytest.raises(_lib.QPamError, match="devices"):
            ops.pam_scan(*a[:4], coef=a[4], s0=a[5])
    h, w = torch.randn(8, 64, device=DEV), torch.randn(30, 64, device=DEV)
    t, m = torch.randint(0, 30, (8,), device=DEV), torch.ones(8, device=DEV)
    for a in ((h, w.cpu(), t, m), (h, w, t.cpu(), m), (h, w, t, m.cpu())):
        for fn in (fused_linear_cross_entropy, linear_ce_stats):
            with pytest.raises(_lib.QPamError, match="devices"):
                fn(*a[:3], mask=a[3])
    with pytest.raises(_lib.QPamError, match="one entry per row"):
        linear_ce_stats(h, w, t, mask=m[:5])
    pool, one = torch.zeros(2, 1, 1, 2, 64, 64, 2, device=DEV), torch.zeros(1, 2, 64, 2, device=DEV)
    with pytest.raises(_lib.QPamError):
        ops.pam_decode_step(pool, torch.tensor([0]), one, one.cpu(), one, torch.ones(1, 1, 2, device=DEV))
    with pytest.raises(_lib.QPamError):
        ops.pam_pool_store(pool, torch.tensor([0]), torch.zeros(1, 1, 2, 64, 64, 2))


@pytest.mark.parametrize("K", [1, 3])
def test_errors_of_a_backward_pass_are_qpam_errors(K):
    """Here a workspace that comes back too small from a saved-tensor hook, which the call refuses before any launch."""
    q, k, v, gamma, _ = _data(K)
    q.requires_grad_()
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: t[:256].clone() if t.dtype == torch.uint8 else t):
        y, _ = ops.pam_scan(q, k, v, gamma, coef=torch.ones(K, 1, 2, 140, 2, device=DEV) if K > 1 else None)
    with pytest.raises(_lib.QPamError, match="workspace"):
        y.float().sum().backward()
