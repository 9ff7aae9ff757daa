"""When a block may run as one native node: not with an operator replaced, wrapped, hooked or built otherwise than the node assumes."""
import pytest
import torch
import torch.nn as nn

from qllm2_b200 import model as M


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
        assert M._stock(_block(**kw))


@pytest.mark.parametrize("change", CHANGES)
def test_changed_blocks_keep_their_operators(change):
    blk = _block()
    CHANGES[change](blk)
    assert not M._stock(blk)


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
