"""The decode step for few rows (qpam_step_fwd) against the block-by-block packed forward it replaces there, at the edges of
its dispatch: rows around the one-kernel limit (4) and the groups of four and eight, split and unsplit projections, every gate source."""
import pytest
import torch

from qllm2_b200 import model as M
from qllm2_b200.fused_forward import FusedForward
from qllm2_b200.serving import _PoolDecodeMix

pytestmark = pytest.mark.gpu
DEV = "cuda"

CONFIGS = {
    "k3_content": dict(dim=64, n_heads=2, n_states=3, gate_content_aware=True),
    "k1_magnitude": dict(dim=96, n_heads=1, n_states=1, gate_content_aware=False),
    "k2_compete": dict(dim=160, n_heads=3, n_states=2, routing_content_aware=True, state_compete=True, phase_init="spread", gamma_floor=0.5),
    "k4_plain": dict(dim=768, n_heads=12, n_states=4, use_gsp=False, use_rope=False, activation="modrelu"),
}


def _setup(name, n, state_dtype):
    torch.manual_seed(7)
    cfg = M.V11Config(vocab_size=1003, head_dim=64, n_layers=2, dropout=0.0, gradient_checkpointing=False, max_seq_len=64, **CONFIGS[name])
    net = M.V11LM(cfg).to(DEV)
    g = torch.Generator(device=DEV).manual_seed(1)
    with torch.no_grad():
        for k, p in net.named_parameters():
            if k.endswith(("weight_real", "weight_imag")):
                p.normal_(0, (2 * p.shape[1]) ** -0.5, generator=g)
            elif p.dim() == 2 or k.endswith("bias"):
                p.add_(torch.randn(p.shape, device=DEV, generator=g) * 0.1)
    net = net.bfloat16().eval()
    pool = (torch.randn(n + 3, 2, cfg.n_states, cfg.n_heads, 64, 64, 2, device=DEV, generator=g) * 0.1).to(state_dtype)
    ids = torch.randint(0, 1003, (n, 1), device=DEV, generator=g)
    pos = torch.randint(0, 64, (n, 1), device=DEV, generator=g)
    slots = torch.randperm(n + 3, device=DEV, generator=g)[:n].int()
    return cfg, FusedForward(net, 64), pool, ids, pos, slots


@pytest.mark.parametrize("name,n", [(c, n) for c in CONFIGS for n in (1, 4, 5, 16)] + [("k3_content", n) for n in (2, 3, 8, 9)])
def test_step_matches_the_packed_forward(name, n):
    state_dtype = torch.float32 if n in (3, 5) else torch.bfloat16
    cfg, ff, pool, ids, pos, slots = _setup(name, n, state_dtype)
    assert ff.step_supported(n)
    p1, p2 = pool.clone(), pool.clone()
    xn = ff.hidden(ids, _PoolDecodeMix(p1, slots, 64), positions=pos)
    want = ff.logits(ff.head_hidden(xn))
    got = ff.step(ids, pos, slots, p2, logits=True).float()
    assert (got - want).norm() / want.norm() < 2e-2
    assert (p2.float() - p1.float()).norm() / p1.float().norm() < 1e-2
    untouched = torch.ones(n + 3, dtype=torch.bool, device=DEV)
    untouched[slots.long()] = False
    assert torch.equal(p2[untouched], pool[untouched])
    # greedy: the same arithmetic, arg-max of the unrounded logits
    p3 = pool.clone()
    pick = ff.step(ids, pos, slots, p3)
    assert torch.equal(p3, p2)
    assert torch.equal(got.gather(1, pick[:, None])[:, 0], got.max(1).values)


def test_padded_rows_leave_the_pool_alone():
    cfg, ff, pool, ids, pos, slots = _setup("k3_content", 5, torch.bfloat16)
    full = pool.clone()
    want = ff.step(ids, pos, slots, full, logits=True)
    slots[2] = -1
    part = pool.clone()
    got = ff.step(ids, pos, slots, part, logits=True)
    rest = [0, 1, 3, 4]
    assert torch.equal(got[rest], want[rest]) and torch.isfinite(got.float()).all()
    changed = (part != pool).flatten(1).any(1).nonzero().flatten().tolist()
    assert sorted(changed) == sorted(slots[rest].tolist())
