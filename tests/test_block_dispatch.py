"""When a block may run as one native node: not with an operator replaced, wrapped, hooked or built otherwise than the node assumes."""
import pytest
import torch
import torch.nn as nn

from qllm2_b200 import _lib
from qllm2_b200 import model as M
from qllm2_b200.fused_forward import FusedForward
from qllm2_b200.serving import ContinuousBatcher


def _block(**kw):
    torch.manual_seed(3)
    kw = {**dict(n_states=3, gate_content_aware=True, state_compete=True, dim=64, n_heads=1), **kw}
    return M.V11Block(M.V11Config(vocab_size=64, head_dim=64, n_layers=1, dropout=0.0, gradient_checkpointing=False, max_seq_len=64, **kw))


class _Adapter(M.ComplexLinear):
    """A projection with a term of its own, as low-rank adapters add it."""

    def forward(self, x):
        return super().forward(x) * 2


class _OtherBlock(M.V11Block):
    @staticmethod
    def _residual(x, delta, scale):
        return x + 2 * delta * scale


def _wrap_forward(m):
    inner = m.forward
    m.forward = lambda *a, **k: inner(*a, **k) * 2


def _swap(owner, name, new):
    new.load_state_dict(getattr(owner, name).state_dict())
    setattr(owner, name, new)


CHANGES = {
    "subclass of a projection": lambda b: _swap(b.cgu, "up_proj", _Adapter(64, 192, bias=False)),
    "projection with a bias": lambda b: setattr(b.pam, "o_proj", M.ComplexLinear(64, 64, bias=True)),
    "Linear without a bias": lambda b: setattr(b.pam, "phase_proj", nn.Linear(64, 3, bias=False)),
    "other activation": lambda b: setattr(b.cgu, "act", nn.Identity()),
    "other epsilon": lambda b: setattr(b.norm2, "eps", 1e-5),
    "forward replaced on an instance": lambda b: _wrap_forward(b.pam.o_proj),
    "sequence mixing replaced": lambda b: setattr(b, "pam", nn.Identity()),
    "dropout replaced": lambda b: setattr(b, "cgu_dropout", nn.Identity()),
    "hook": lambda b: b.pam.dt_proj.register_forward_hook(lambda *a: None),
    "bf16 parameter": lambda b: b.pam.dt_proj.bfloat16(),
}


def test_stock_blocks_are_recognised():
    for kw in (dict(), dict(n_states=1, use_gsp=False), dict(activation="modrelu", state_compete=False)):
        assert M._stock(_block(**kw), torch.float32)


@pytest.mark.parametrize("change", CHANGES)
def test_changed_blocks_keep_their_operators(change):
    blk = _block()
    CHANGES[change](blk)
    assert not M._stock(blk, torch.float32)
    assert M._stock(blk) == (change == "bf16 parameter")         # inference takes weights of any type


def _net():
    torch.manual_seed(3)
    return M.V11LM(M.V11Config(vocab_size=64, dim=64, n_heads=1, head_dim=64, n_layers=2, dropout=0.0, gradient_checkpointing=False, max_seq_len=64))


NET_CHANGES = {
    "adapter": lambda n: _swap(n.blocks[1].cgu, "up_proj", _Adapter(64, 192, bias=False)),
    "block subclass": lambda n: setattr(n.blocks[0], "__class__", _OtherBlock),
    "hook": lambda n: n.blocks[1].pam.dt_proj.register_forward_hook(lambda *a: None),
    "head epsilon": lambda n: setattr(n.lm_head_norm, "eps", 1e-5),
    "head hook": lambda n: n.lm_head_proj.register_forward_hook(lambda *a: None),
}


@pytest.mark.parametrize("change", NET_CHANGES)
def test_changed_models_are_not_packed(change):
    net = _net()
    assert M._stock_operators(net) and "CUDA" in FusedForward.unsupported_reason(net)
    NET_CHANGES[change](net)
    assert "called as modules" in FusedForward.unsupported_reason(net)


def _x(D=64, T=40):
    return torch.zeros(1, T, D, 2, dtype=torch.bfloat16)


MISFITS = {     # what is changed about the block, and the input it then gets
    "other channel count": (lambda b: None, _x(D=68)),
    "wider down projection": (lambda b: setattr(b.cgu, "down_proj", M.ComplexLinear(256, 64, bias=False)), _x()),
    "fewer heads in the input projection": (lambda b: setattr(b.pam, "qkv_proj", M.ComplexLinear(64, 64, bias=False)), _x()),
    "short activation bias": (lambda b: setattr(b.cgu.act, "bias", nn.Parameter(torch.zeros(100))), _x()),
    "narrow routing": (lambda b: setattr(b.pam, "phase_proj", nn.Linear(32, 3)), _x()),
    "scalar of two": (lambda b: setattr(b, "pam_scale", nn.Parameter(torch.ones(2))), _x()),
    "short rotary table": (lambda b: setattr(b.pam, "rope_table", lambda x, o: b.pam.rope_cache[:39]), _x()),
    "other rotary width": (lambda b: setattr(b.pam, "rope_cache", torch.zeros(64, 32, 2)), _x()),
    "no input": (lambda b: None, _x(T=0)),
}


@pytest.mark.parametrize("case", MISFITS)
def test_native_node_checks_every_shape(case):
    """The node's kernels get pointers and sizes: operands that do not fit are refused before anything is launched."""
    change, x = MISFITS[case]
    blk = _block()
    change(blk)
    with pytest.raises(_lib.QPamError, match="block: "):
        blk._native(x, 0)


def test_native_node_has_no_cpu_path():
    with pytest.raises(_lib.QPamError, match="need CUDA tensors"):
        _block()._native(_x(), 0)


@pytest.mark.gpu
def test_parameters_of_any_layout():
    """Parameters as views into one flat buffer, each starting off a 16-byte boundary, and transposed ones: the same results."""
    ref, blk = _block().cuda(), _block().cuda()
    buf = torch.zeros(sum(p.numel() + 9 for p in blk.parameters()), device="cuda")
    at = 1
    for i, p in enumerate(blk.parameters()):
        if p.dim() == 2 and i % 2:
            p.data = p.data.t().contiguous().t()
        else:
            flat = buf[at:at + p.numel()].view(p.shape)
            flat.copy_(p.data)
            p.data = flat
            at = (at + p.numel() + 4) // 4 * 4 + 1
    assert any(not p.is_contiguous() for p in blk.parameters()) and any(p.data_ptr() % 16 for p in blk.parameters())
    g = torch.Generator(device="cuda").manual_seed(1)
    xs = torch.randn(1 + 2 * 50 * 64 * 2, device="cuda", generator=g).bfloat16()
    x = [t.requires_grad_() for t in (xs[1:].view(2, 50, 64, 2).clone(), xs[1:].view(2, 50, 64, 2).detach())]
    dys = torch.randn(1 + 2 * 50 * 64 * 2, device="cuda", generator=g).bfloat16()[1:].view(2, 50, 64, 2)
    assert x[0].data_ptr() % 16 == 0 and x[1].data_ptr() % 16 and dys.data_ptr() % 16
    res = []
    for b, xi, dy in ((ref, x[0], dys.clone()), (blk, x[1], dys)):
        with torch.autocast("cuda", dtype=torch.bfloat16):
            assert b._native_ok(xi, None)
            y, s = b._native(xi, 0)
        y.backward(dy)
        res.append([y, s, xi.grad] + [p.grad for p in b.parameters()])
    for a, c in zip(*res):
        assert torch.equal(a, c)


@pytest.mark.gpu
@pytest.mark.parametrize("case", ["adapter", "block subclass", "global hook"])
def test_native_node_does_not_bypass(case):
    blk = (_OtherBlock(M.V11Config(vocab_size=64, dim=64, n_heads=1, head_dim=64, n_layers=1, dropout=0.0, max_seq_len=64)) if case == "block subclass" else _block()).cuda()
    x = torch.randn(1, 40, 64, 2, device="cuda").bfloat16()
    seen, hook = [], None
    with torch.autocast("cuda", dtype=torch.bfloat16):
        if case != "block subclass":
            assert blk._native_ok(x, None)
        if case == "adapter":
            blk.cgu.up_proj = _Adapter(64, 192, bias=False).cuda()
        if case == "global hook":
            hook = nn.modules.module.register_module_forward_hook(lambda m, *a: seen.append(type(m)))
        try:
            assert not blk._native_ok(x, None)
            y, _ = blk(x)
        finally:
            if hook is not None:
                hook.remove()
        if case == "global hook":
            assert M.ComplexLinear in seen and M.ComplexNorm in seen
            return
        blk.norm1.register_forward_hook(lambda *a: None)           # the operators, in any case
        want, _ = blk(x)
    assert torch.equal(y, want)


@pytest.mark.gpu
def test_adapters_take_part_in_generation_and_serving():
    """A projection with a term of its own: its tokens are those of the module-by-module loop, not of the packed weights."""
    net = _net().cuda().eval()
    with torch.no_grad():
        for p in net.parameters():
            p.add_(torch.randn(p.shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(p.numel())) * 0.2)
    ids = torch.randint(0, 64, (2, 9), device="cuda", generator=torch.Generator(device="cuda").manual_seed(5))
    plain = net.generate(ids, 12, temperature=0)
    NET_CHANGES["adapter"](net)
    net.cuda()
    got = net.generate(ids, 12, temperature=0)
    assert torch.equal(got, net.generate(ids, 12, temperature=0, fused=False)) and not torch.equal(got, plain)
    eng = ContinuousBatcher(net, n_slots=2, max_position=64)
    rids = [eng.submit(row, 12) for row in ids.tolist()]
    done = eng.run()
    assert [done[r] for r in rids] == got[:, 9:].tolist()
