"""Idle rows of a decode batch (slot -1) and rows of NaN: defined outputs and token ids of the vocabulary, since a captured step
feeds its ids to the next one on the device."""
import pytest
import torch

from qllm2_b200 import model as M
from qllm2_b200 import ops
from qllm2_b200.serving import ContinuousBatcher

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("state", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("io", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("d", [16, 32, 64])
def test_decode_step_of_idle_rows_is_zero(d, io, state):
    n, H, K = 5, 3, 2
    g = torch.Generator(device=DEV).manual_seed(d)
    pool = torch.randn(4, 2, K, H, d, d, 2, device=DEV, generator=g).to(state)
    q, k, v = [torch.randn(n, H, d, 2, device=DEV, generator=g).to(io) for _ in range(3)]
    gamma, coef = torch.rand(K, n, H, device=DEV, generator=g), torch.randn(K, n, H, 2, device=DEV, generator=g)
    want = pool.clone()
    full = ops.pam_decode_step(want, torch.tensor([2, 0, 3, 1, 1])[:4], *(t[:4] for t in (q, k, v)), gamma[:, :4].contiguous(), coef[:, :4].contiguous(), layer=1)
    junk = [torch.full((n, H, d, 2), float("nan"), dtype=io, device=DEV) for _ in range(8)]       # what a fresh output may hold
    del junk
    idle = torch.tensor([2, -1, 3, 4, 1])                # -1 and one past the pool
    got_pool = pool.clone()
    y = ops.pam_decode_step(got_pool, idle, q, k, v, gamma, coef, layer=1)
    assert not y[[1, 3]].any() and torch.equal(y[[0, 2]], full[[0, 2]])
    assert torch.equal(got_pool[[2, 3]], want[[2, 3]]) and torch.equal(got_pool[0], pool[0])


def test_captured_steps_feed_ids_of_the_vocabulary():
    """Twenty slots, one live sequence: more steps than one between the host's reads, nineteen idle rows."""
    torch.manual_seed(1)
    cfg = M.V11Config(vocab_size=101, dim=64, n_heads=1, head_dim=64, n_layers=2, n_states=2, dropout=0.0, gradient_checkpointing=False, max_seq_len=128)
    net = M.V11LM(cfg).to(DEV).bfloat16().eval()
    out = []
    for graph in (False, True):
        eng = ContinuousBatcher(net, n_slots=20, cuda_graph=graph, max_position=128)
        rid = eng.submit([3, 7, 11], 40)
        out.append(eng.run()[rid])
        if graph:
            assert int(eng._g_ids.min()) >= 0 and int(eng._g_ids.max()) < 101 and torch.isfinite(eng.pool.float()).all()
    assert out[0] == out[1]


@pytest.mark.parametrize("dtype,N,F,V", [(torch.float32, 9, 32, 101), (torch.bfloat16, 9, 64, 1003), (torch.bfloat16, 300, 64, 1003)])
def test_arg_max_of_rows_without_a_number(dtype, N, F, V):
    """A row of NaN has no arg-max; its id is one of the vocabulary all the same, and the other rows' are what they were."""
    g = torch.Generator(device=DEV).manual_seed(V)
    h, w = torch.randn(N, F, device=DEV, generator=g).to(dtype), torch.randn(V, F, device=DEV, generator=g).to(dtype)
    want, _ = ops.head_argmax(h, w)
    bad = h.clone()
    bad[::4] = float("nan")
    ids, _ = ops.head_argmax(bad, w)
    assert int(ids.min()) >= 0 and int(ids.max()) < V
    keep = torch.ones(N, dtype=torch.bool, device=DEV)
    keep[::4] = False
    assert torch.equal(ids[keep], want[keep])
