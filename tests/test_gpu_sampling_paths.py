"""The sampler's dispatch at its edges: list and bin paths around the list's top-k limit, rows that start off a 16-byte
boundary, rows shorter than the block, and rows whose ties overflow the list."""
import threading

import pytest
import torch

from qllm2_b200 import _lib, ops
from tests.test_gpu_sampling import _check_rows

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("n", [3, 150])
@pytest.mark.parametrize("dtype,V,lead", [(torch.bfloat16, 50261, 0), (torch.bfloat16, 4099, 3), (torch.float32, 1027, 1), (torch.float32, 9, 0)])
@pytest.mark.parametrize("top_k,top_p", [(384, 0.9), (385, 0.9), (1500, 0.0), (0, 0.6)])
def test_paths(n, dtype, V, lead, top_k, top_p):
    g = torch.Generator().manual_seed(V + top_k + n)
    store = (torch.randn(n, V + 11, generator=g) * 2.0).to(dtype).to(DEV)
    logits = store[:, lead:lead + V]
    hist = torch.randint(0, V, (n, 33), generator=g)
    u = torch.rand(n, generator=g)
    cfg = dict(temperature=0.8, top_k=top_k, top_p=top_p, repetition_penalty=1.2345)
    ids, stats = ops.sample_logits(logits, u.to(DEV), history=hist.to(DEV), return_stats=True, **cfg)
    _check_rows(logits, hist.numpy(), None, u.numpy(), ids.cpu().numpy(), stats.cpu().numpy(), cfg, count_exact=dtype == torch.float32)


@pytest.mark.parametrize("top_k,top_p", [(50, 0.9), (900, 0.5), (0, 0.5)])
def test_ties_beyond_the_list(top_k, top_p):
    """Every token at one of two values: all of the upper ones tie with the threshold and stay."""
    n, V = 4, 20000
    g = torch.Generator().manual_seed(3)
    logits = (torch.rand(n, V, generator=g) < 0.5).float().to(DEV)
    u = torch.rand(n, generator=g)
    cfg = dict(temperature=1.0, top_k=top_k, top_p=top_p, repetition_penalty=1.0)
    ids, stats = ops.sample_logits(logits, u.to(DEV), return_stats=True, **cfg)
    _check_rows(logits, None, None, u.numpy(), ids.cpu().numpy(), stats.cpu().numpy(), cfg)
    assert stats[:, 2].tolist() == (logits == 1).sum(1).tolist()


def test_strided_vectors():
    """Uniforms, slots and lengths as columns of wider tensors mean what their values say."""
    n, V = 5, 997
    g = torch.Generator().manual_seed(8)
    logits = (torch.randn(n, V, generator=g) * 3).to(DEV)
    wide = lambda t: torch.stack([t, torch.zeros_like(t)], dim=1).to(DEV)[:, 0]
    u, slots = torch.rand(n, generator=g), torch.tensor([4, 0, 2, 1, 3], dtype=torch.int32)
    lens, hist = torch.tensor([3, 7, 1, 5, 9], dtype=torch.int32), torch.randint(0, V, (n, 12), generator=g)
    cfg = dict(history=hist.to(DEV), top_p=0.9, repetition_penalty=1.5)
    want = ops.sample_logits(logits, u.to(DEV), slot_ids=slots.to(DEV), hist_len=lens.to(DEV), **cfg)
    got = ops.sample_logits(logits, wide(u), slot_ids=wide(slots), hist_len=wide(lens), **cfg)
    assert torch.equal(got, want)
    with pytest.raises(_lib.QPamError):
        ops.sample_logits(logits, u.to(DEV), hist_len=wide(lens), append=True, **cfg)


def test_threads_with_vocabularies_of_different_size():
    """The penalty's bitmap is sized by the vocabulary: threads with different ones do not shrink each other's shared memory."""
    errors, want = [], {}

    def draw(V):
        g = torch.Generator().manual_seed(V)
        logits, hist = torch.randn(2, V, generator=g).to(DEV), torch.randint(0, V, (2, 9), generator=g).to(DEV)
        u = torch.rand(2, generator=g).to(DEV)
        return lambda: ops.sample_logits(logits, u, history=hist, top_k=20, repetition_penalty=1.2)

    calls = {V: draw(V) for V in (1000, 200_000, 1_200_000)}
    for V, f in calls.items():
        want[V] = f().tolist()

    def work(V):
        try:
            for _ in range(200):
                got = calls[V]()
            assert got.tolist() == want[V]
        except Exception as e:      # reported in the test's own thread
            errors.append((V, e))

    ts = [threading.Thread(target=work, args=(V,)) for V in calls]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors
