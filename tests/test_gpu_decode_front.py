"""The decode step that forms q, k, v and the gates where it uses them (qpam_decode_front) against the separate kernels, for every
source that a gate can have, idle rows among the live ones."""
import pytest
import torch

from qllm2_b200 import _lib, model as M
from qllm2_b200.fused_forward import FusedForward
from qllm2_b200.serving import _PoolDecodeMix

pytestmark = pytest.mark.gpu
DEV = "cuda"

CONFIGS = {
    "k3_content": dict(dim=64, n_heads=2, n_states=3, gate_content_aware=True, routing_content_aware=True),      # no gate reads |x|
    "k3_chat": dict(dim=768, n_heads=12, n_states=3, gate_content_aware=True),
    "k1_magnitude": dict(dim=96, n_heads=1, n_states=1, gate_content_aware=False),
    "k2_compete": dict(dim=168, n_heads=3, n_states=2, state_compete=True, phase_init="spread", gamma_floor=0.5),
    "k4_plain": dict(dim=264, n_heads=2, n_states=4, state_compete=True, use_gsp=False, use_rope=False),
}


class _Separate:
    """The same mix without a pool to work in place on."""

    def __init__(self, mix):
        self.mix, self.q_scale = mix, mix.q_scale

    def __call__(self, *args):
        return self.mix(*args)


@pytest.mark.parametrize("n", [1, 33])
@pytest.mark.parametrize("name", CONFIGS)
def test_decode_front_against_separate_kernels(name, n):
    torch.manual_seed(3)
    cfg = M.V11Config(vocab_size=101, head_dim=64, n_layers=2, dropout=0.0, gradient_checkpointing=False, max_seq_len=64, **CONFIGS[name])
    net = M.V11LM(cfg).to(DEV)
    g = torch.Generator(device=DEV).manual_seed(1)
    with torch.no_grad():
        for k, p in net.named_parameters():
            if k.endswith(("weight_real", "weight_imag")):
                p.normal_(0, (2 * p.shape[1]) ** -0.5, generator=g)
            elif p.dim() == 2 or k.endswith("bias"):
                p.add_(torch.randn(p.shape, device=DEV, generator=g) * 0.1)
    ff = FusedForward(net.bfloat16().eval(), 64)
    pool = (torch.randn(n + 3, 2, cfg.n_states, cfg.n_heads, 64, 64, 2, device=DEV, generator=g) * 0.1).bfloat16()
    ids = torch.randint(0, 101, (n, 1), device=DEV, generator=g)
    pos = torch.randint(0, 70, (n, 1), device=DEV, generator=g)              # the last positions are past the table: clamped alike
    slots = torch.randperm(n + 3, device=DEV, generator=g)[:n].int()
    if n > 1:
        slots[1], slots[2] = -1, n + 3
    p1, p2 = pool.clone(), pool.clone()
    want = ff.hidden(ids, _Separate(_PoolDecodeMix(p1, slots, 64)), positions=pos)
    n0 = _lib.launch_count()
    got = ff.hidden(ids, _PoolDecodeMix(p2, slots, 64), positions=pos)
    assert _lib.launch_count() - n0 == 2 + 2 * 4      # embedding and first norm, then per layer gated unit, two norms and the step
    assert _lib.device_status() == 0
    if ff.layers[0].w_mag is None:
        assert torch.equal(got, want) and torch.equal(p1, p2)
    else:      # a gate of |x| is a sum of bf16 products in another order: it may round to the neighbouring bf16 number (2^-8)
        assert (got.float() - want.float()).norm() / want.float().norm() < 1e-2
        assert (p2.float() - p1.float()).norm() / p1.float().norm() < 4e-3
    untouched = torch.ones(n + 3, dtype=torch.bool, device=DEV)
    untouched[slots[(slots >= 0) & (slots < n + 3)].long()] = False
    assert torch.equal(p2[untouched], pool[untouched])


def _small():
    torch.manual_seed(5)
    cfg = M.V11Config(vocab_size=101, head_dim=64, n_layers=2, dropout=0.0, gradient_checkpointing=False, max_seq_len=64, **CONFIGS["k3_content"])
    ff = FusedForward(M.V11LM(cfg).to(DEV).bfloat16().eval(), 64)
    pool = torch.randn(5, 2, 3, 2, 64, 64, 2, device=DEV, generator=torch.Generator(device=DEV).manual_seed(2)).bfloat16()
    return ff, pool, torch.tensor([[3], [8], [1]], device=DEV), torch.tensor([2, 0, 4], device=DEV, dtype=torch.int32)


class _Scaled(_PoolDecodeMix):
    def __call__(self, *args):
        return super().__call__(*args) * 256


class _Own:
    """Anything with a pool, slots and a q_scale; its mixing is its own."""

    def __init__(self, pool, slots):
        self.pool, self.slots, self.q_scale, self.calls = pool, slots, 0.125, []

    def __call__(self, layer, q, k, v, gamma, coef):
        self.calls.append((layer, tuple(q.shape)))
        return v[:, :, 0].reshape(v.shape[0], -1)


def test_a_callers_mix_is_called():
    ff, pool, ids, slots = _small()
    plain = ff.hidden(ids, _PoolDecodeMix(pool.clone(), slots, 64))
    scaled = ff.hidden(ids, _Scaled(pool.clone(), slots, 64))
    assert torch.equal(scaled, ff.hidden(ids, _Separate(_Scaled(pool.clone(), slots, 64)))) and not torch.equal(scaled, plain)
    own, before = _Own(pool, slots), pool.clone()
    got = ff.hidden(ids, own)
    assert own.calls == [(0, (3, 2, 1, 64, 2)), (1, (3, 2, 1, 64, 2))] and torch.equal(pool, before)
    assert torch.equal(got, ff.hidden(ids, _Separate(own)))


def test_slot_ids_and_pools_as_the_separate_step_takes_them():
    ff, pool, ids, slots = _small()
    want_pool = pool.clone()
    want = ff.hidden(ids, _Separate(_PoolDecodeMix(want_pool, slots, 64)))
    for other in (slots.long(), slots.cpu(), slots.short(), torch.stack([slots, slots], 1)[:, 0]):
        p = pool.clone()
        assert torch.equal(ff.hidden(ids, _PoolDecodeMix(p, other, 64)), want) and torch.equal(p, want_pool)
    for mix in (_PoolDecodeMix(pool, slots[:2], 64), _PoolDecodeMix(pool.cpu(), slots, 64), _PoolDecodeMix(pool.transpose(0, 1), slots, 64)):
        with pytest.raises(_lib.QPamError):
            ff.hidden(ids, mix)
