"""The packed prefill checks what its kernels index by pointer, and takes slots and descriptors of any integer type."""
import pytest
import torch

from qllm2_b200 import _lib
from qllm2_b200 import model as M
from qllm2_b200.fused_forward import FusedForward

D, H, d, K, L = 64, 2, 64, 2, 2


def _net():
    torch.manual_seed(5)
    return M.V11LM(M.V11Config(vocab_size=67, dim=D, n_heads=H, head_dim=d, n_layers=L, n_states=K, dropout=0.0, max_seq_len=64, gradient_checkpointing=False))


def _call(**kw):
    net = _net()
    scale = torch.ones(D)
    layers = [FusedForward.pack_block(b, torch.float32) for b in net.blocks]
    packed = _lib.host().Packed(D, H, d, K, layers, scale, scale, torch.zeros(64, d, 2))
    a = dict(ids=torch.zeros(1, 9, dtype=torch.long), pool=torch.zeros(4, L, K, H, d, d, 2), slots=torch.tensor([1, 0]), cu=torch.tensor([0, 4, 9]), positions=None,
             resumed=None, embed=torch.zeros(67, D))
    a.update(kw)
    packed.prefill(a["embed"], torch.zeros(67, D), a.get("embedded"), a["ids"], a["pool"], a["slots"], a["cu"], a["positions"], a["resumed"])


@pytest.mark.parametrize("kw", [
    dict(pool=torch.zeros(4, L, K + 1, H, d, d, 2)), dict(pool=torch.zeros(4, L, K, H - 1, d, d, 2)), dict(pool=torch.zeros(4, L, K, H, 32, 32, 2)),
    dict(pool=torch.zeros(4, L + 1, K, H, d, d, 2)), dict(pool=torch.zeros(4, d, d, 2)), dict(slots=torch.tensor([1])), dict(slots=torch.tensor([1, 0, 2])),
    dict(slots=torch.tensor([1.0, 0.0])), dict(ids=torch.zeros(2, 9, dtype=torch.long)), dict(ids=torch.zeros(0, 9, dtype=torch.long)), dict(positions=torch.arange(8)),
    dict(resumed=torch.ones(3)), dict(embed=torch.zeros(67, D + 4)), dict(embed=None), dict(embedded=torch.zeros(1, 8, D, 2)), dict(cu=None), dict(ids=torch.zeros(1, 80, dtype=torch.long), cu=None, slots=torch.tensor([1]))],
    ids=lambda kw: "-".join("%s%s" % (k, "" if v is None else list(v.shape)) for k, v in kw.items()))
def test_operands_that_do_not_fit_are_refused(kw):
    with pytest.raises(_lib.QPamError, match="prefill:|max_position"):
        _call(**kw)


def test_bad_host_descriptor_is_refused():
    with pytest.raises(_lib.QPamError, match="cu_seqlens"):
        _call(cu=torch.tensor([0, 10, 9]))


def test_no_cpu_path():
    with pytest.raises(_lib.QPamError, match="need CUDA tensors"):
        _call()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_integer_types_of_slots_and_descriptors(dtype):
    net = _net().to("cuda", dtype).eval()
    ff = FusedForward(net, 64)
    ids = torch.randint(0, 67, (1, 23), device="cuda")
    res = []
    for it in (torch.int32, torch.int64):
        pool = torch.zeros(4, L, K, H, d, d, 2, device="cuda", dtype=dtype)
        slots, cu = torch.tensor([2, 0, 3], device="cuda", dtype=it), torch.tensor([0, 5, 6, 23], device="cuda", dtype=it)
        pos = torch.tensor([*range(5), 0, *range(17)], device="cuda", dtype=it)
        res.append((ff.prefill(ids, pool, slots, cu, pos), pool))
    assert torch.equal(res[0][0], res[1][0]) and torch.equal(res[0][1], res[1][1])
    assert res[0][1][[0, 2, 3]].abs().amax() > 0 and not res[0][1][1].any()


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["hook", "subclass", "strided"])
def test_embeddings_that_are_more_than_a_table(kind):
    """Prefill and decode step call them as the modules they are."""
    net = _net().to("cuda", torch.bfloat16).eval()
    ids = torch.randint(0, 67, (2, 11), device="cuda")
    slots = torch.tensor([1, 0], dtype=torch.int32, device="cuda")

    class Doubled(torch.nn.Embedding):
        def forward(self, ids):
            return super().forward(ids) * 2

    table = net.embed.embed_real.weight.data
    if kind == "strided":
        net.embed.embed_real.weight.data = table.t().contiguous().t()
    elif kind == "hook":
        net.embed.embed_real.register_forward_hook(lambda m, i, o: o * 2)
    else:
        net.embed.embed_real = Doubled(67, D, _weight=table)
    ff = FusedForward(net, 64)
    assert not ff.step_supported(2)
    pools = [torch.zeros(2, L, K, H, d, d, 2, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
    got = ff.prefill(ids, pools[0], slots)
    ref = _net().to("cuda", torch.bfloat16).eval()
    if kind != "strided":
        ref.embed.embed_real.weight.data.mul_(2)
    want = FusedForward(ref, 64)
    assert want.step_supported(2)
    assert torch.equal(got, want.prefill(ids, pools[1], slots)) and torch.equal(pools[0], pools[1])
