"""Every entry point whose kernels overlap (programmatic dependent launch) gives the bits it gives when each launch waits for the one
before it: in calls whose inputs are still being written when they are issued, back to back, on two streams at once, and as
replays of a captured graph.  (While launches are profiled an event lies between any two of them, so none overlap.)"""
import pytest
import torch

from qllm2_b200 import _lib, ops
from qllm2_b200 import model as M
from qllm2_b200.fused_ce import fused_linear_cross_entropy, linear_ce_stats
from qllm2_b200.fused_forward import FusedForward
from qllm2_b200.serving import _PoolDecodeMix

pytestmark = pytest.mark.gpu
DEV = "cuda"
CALLS = 3


def _outputs(got):
    return [t.detach() for t in got if torch.is_tensor(t)]


def _check(base, call):
    """call(inputs) -> tensors, with inputs of `base` (dict of tensors) that launches right before it write."""
    def inputs(i):
        return {n: t.clone() if n in FIXED or not t.is_floating_point() else t * (1.0 - 0.125 * i) for n, t in base.items()}

    def isolated(i):
        x = inputs(i)
        torch.cuda.synchronize()
        _lib.profile_begin()
        try:
            out = _outputs(call(x))
        finally:
            kernels = _lib.profile_end()
        torch.cuda.synchronize()
        assert kernels
        return [t.clone() for t in out]

    def same(got, want, what):
        for i, (a, b) in enumerate(zip(got, want)):
            assert len(a) == len(b)
            for j, (x, y) in enumerate(zip(a, b)):
                assert torch.equal(x, y), (what, i, j)

    want = [isolated(i) for i in range(CALLS)]
    same([_outputs(call(inputs(i))) for i in range(CALLS)], want, "back to back")
    here, streams = torch.cuda.current_stream(), [torch.cuda.Stream(), torch.cuda.Stream()]
    got = [[], []]
    for st in streams:
        st.wait_stream(here)
    for i in range(CALLS):
        for st, g in zip(streams, got):
            with torch.cuda.stream(st):
                g.append(_outputs(call(inputs(i))))
    for st in streams:
        here.wait_stream(st)
    torch.cuda.synchronize()
    for g in got:
        same(g, want, "two streams")
    static = inputs(0)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = _outputs(call(static))
    replayed = []
    for i in range(CALLS):
        for n, t in inputs(i).items():
            static[n].copy_(t)
        graph.replay()
        replayed.append([t.clone() for t in out])
    same(replayed, want, "replayed")
    assert _lib.device_status() == 0


FIXED = ("gamma", "cu", "slots")


def _scan_inputs(B, H, T, K, coef=False, s0=0, seed=0):
    g = torch.Generator(device=DEV).manual_seed(T + seed)
    x = {n: (torch.randn(B, H, T, 64, 2, device=DEV, generator=g) * 0.09).bfloat16() for n in ("q", "k", "v")}
    x["gamma"] = torch.sigmoid(torch.randn(K, B, H, T, device=DEV, generator=g) + 2.0)
    if coef:
        x["coef"] = torch.randn(K, B, H, T, 2, device=DEV, generator=g)
    if s0:
        x["s0"] = torch.randn(K, s0, H, 64, 64, 2, device=DEV, generator=g)
    return x


def _lengths(lengths):
    cu = torch.zeros(len(lengths) + 1, dtype=torch.int32)
    cu[1:] = torch.tensor(lengths).cumsum(0)
    return cu.to(DEV)


PACKED = [1, 130, 640, 3, 128, 517]


@pytest.mark.parametrize("lengths,H,K,s0", [
    (PACKED, 4, 1, False),
    (PACKED, 4, 3, False),
    (PACKED, 4, 3, True),
    (PACKED, 4, 1, True),
    ([1030, 1100, 1024, 1300] * 6, 16, 1, False),       # the chunk sums carry: wide, eight chunks and more a sequence
    ([1030, 6000, 1024, 1300] * 6, 16, 1, False),       # taken for wide by the host, too narrow by the device's count
])
def test_packed_prefill(lengths, H, K, s0):
    x = _scan_inputs(1, H, sum(lengths), K, coef=K > 1, s0=len(lengths) if s0 else 0)
    x["cu"] = _lengths(lengths)
    _check(x, lambda x: ops.pam_scan_tokens(x["q"], x["k"], x["v"], x["gamma"], coef=x.get("coef"), s0=x.get("s0"), cu_seqlens=x["cu"]))


@pytest.mark.parametrize("B,H,T,K,coef,s0,cu,save", [
    (2, 4, 300, 1, False, False, False, False),         # chunk states formed again in the backward
    (2, 4, 300, 1, False, True, False, True),
    (1, 4, 93, 1, False, True, False, True),            # one chunk with a state before it
    (1, 4, sum(PACKED), 1, False, True, True, True),
    (1, 4, sum(PACKED), 3, True, True, True, True),
    (2, 4, 300, 3, True, False, False, False),          # one scan per state
    (2, 4, 300, 3, False, False, False, True),          # one output kernel per state
    (4, 6, 700, 2, False, True, False, True),
    (1, 4, 93, 3, False, False, False, True),
])
def test_scan_with_gradients(B, H, T, K, coef, s0, cu, save):
    x = _scan_inputs(B, H, T, K, coef=coef, s0=(len(PACKED) if cu else B) if s0 else 0)
    if cu:
        x["cu"] = _lengths(PACKED)
    dy = torch.randn(B, H, T, 64, 2, device=DEV, generator=torch.Generator(device=DEV).manual_seed(5)).bfloat16()
    ds = torch.randn(K, len(PACKED) if cu else B, H, 64, 64, 2, device=DEV, generator=torch.Generator(device=DEV).manual_seed(6)) if s0 else None

    def call(x):
        leaves = {n: t.detach().requires_grad_(n != "cu") for n, t in x.items()}
        y, last = ops.pam_scan(leaves["q"], leaves["k"], leaves["v"], leaves["gamma"], coef=leaves.get("coef"), s0=leaves.get("s0"),
                               cu_seqlens=leaves.get("cu"), save_states=save)
        outs, grads = ([y], [dy]) if ds is None else ([y, last], [dy, ds])
        return [y, last, *torch.autograd.grad(outs, [t for n, t in leaves.items() if n != "cu"], grads)]
    _check(x, call)


@pytest.mark.parametrize("N,F,V", [(1, 64, 300), (509, 192, 5003), (8192 + 300, 64, 520), (300, 64, 50261)])
def test_loss(N, F, V):
    g = torch.Generator(device=DEV).manual_seed(N)
    x = dict(h=torch.randn(N, F, device=DEV, generator=g).bfloat16(), w=(torch.randn(V, F, device=DEV, generator=g) * 0.3).bfloat16(),
             t=torch.randint(0, V, (N,), device=DEV, generator=g))

    def call(x):
        h, w = x["h"].detach().requires_grad_(True), x["w"].detach().requires_grad_(True)
        loss = fused_linear_cross_entropy(h, w, x["t"])
        return [loss, *torch.autograd.grad(loss, [h, w]), *ops.head_argmax(x["h"], x["w"]), ops.head_logits(x["h"], x["w"])]
    _check(x, call)


def _net(K, layers=2, dim=64, heads=2, **kw):
    torch.manual_seed(7)
    cfg = M.V11Config(vocab_size=1003, head_dim=64, n_layers=layers, dim=dim, n_heads=heads, n_states=K, dropout=0.0, gradient_checkpointing=False,
                      gate_content_aware=True, max_seq_len=512, **kw)
    net = M.V11LM(cfg).to(DEV)
    g = torch.Generator(device=DEV).manual_seed(1)
    with torch.no_grad():
        for k, p in net.named_parameters():
            if k.endswith(("weight_real", "weight_imag")):
                p.normal_(0, (2 * p.shape[1]) ** -0.5, generator=g)
            elif p.dim() == 2 or k.endswith("bias"):
                p.add_(torch.randn(p.shape, device=DEV, generator=g) * 0.1)
    return net


@pytest.mark.parametrize("state", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n,K,few", [(24, 3, False), (200, 1, False), (8, 3, True), (13, 1, True), (2, 3, True), (4, 1, True)])
def test_decode_steps(n, K, few, state):
    """Three steps, each feeding the next its tokens on the device: the packed blocks, the chain of a few rows, the one kernel."""
    ff = FusedForward(_net(K).bfloat16().eval(), 64)
    assert ff.step_supported(n) or not few
    g = torch.Generator(device=DEV).manual_seed(n)
    x = dict(pool=(torch.randn(n + 3, 2, K, 2, 64, 64, 2, device=DEV, generator=g) * 0.1).to(state),
             ids=torch.randint(0, 1003, (n, 1), device=DEV, generator=g), pos=torch.randint(0, 60, (n, 1), device=DEV, generator=g),
             slots=torch.randperm(n + 3, device=DEV, generator=g)[:n].int())

    def call(x):
        ids, out = x["ids"], []
        pool = x["pool"].clone()
        for t in range(3):
            if few:
                ids = ff.step(ids, x["pos"] + t, x["slots"], pool).view(n, 1)
            else:
                xn = ff.hidden(ids, _PoolDecodeMix(pool, x["slots"], 64), positions=x["pos"] + t)
                ids = ff.greedy_next(ff.head_hidden(xn)).view(n, 1)
                out.append(xn)
            out.append(ids)
        return [*out, pool]
    _check(x, call)


@pytest.mark.parametrize("K", [1, 3])
def test_prefill_of_a_model(K):
    """The packed forward of prompts into the slots of a state pool (rows of several kilobytes and short ones)."""
    ff = FusedForward(_net(K).bfloat16().eval(), 1024)
    lengths = [5, 300, 129, 77]
    g = torch.Generator(device=DEV).manual_seed(K)
    x = dict(ids=torch.randint(0, 1003, (1, sum(lengths)), device=DEV, generator=g), cu=_lengths(lengths),
             pos=torch.cat([torch.arange(n) for n in lengths])[None].to(DEV), slots=torch.tensor([3, 0, 4, 1], dtype=torch.int32, device=DEV),
             pool=torch.randn(5, 2, K, 2, 64, 64, 2, device=DEV, generator=g).bfloat16())

    def call(x):
        pool = x["pool"].clone()
        return [ff.prefill(x["ids"], pool, x["slots"], cu=x["cu"], positions=x["pos"]), pool]
    _check(x, call)


@pytest.mark.parametrize("K", [1, 3])
def test_training_block(K):
    """The native block, forward and backward: its scan's kernels among library products and ordinary launches."""
    blk = _net(K, layers=1).blocks[0].train()
    g = torch.Generator(device=DEV).manual_seed(K)
    x = dict(x=torch.randn(2, 300, 64, 2, device=DEV, generator=g).bfloat16(), dy=torch.randn(2, 300, 64, 2, device=DEV, generator=g).bfloat16())
    params = list(blk.parameters())

    def call(x):
        xi = x["x"].detach().requires_grad_(True)
        with torch.autocast("cuda", dtype=torch.bfloat16):
            assert blk._native_ok(xi, None)
            out, state = blk(xi)
        return [out, state, *torch.autograd.grad(out, [xi, *params], x["dy"], allow_unused=True)]
    _check(x, call)


def test_statistics_of_a_head():
    g = torch.Generator(device=DEV).manual_seed(2)
    h, w = torch.randn(777, 64, device=DEV, generator=g).bfloat16(), torch.randn(5003, 64, device=DEV, generator=g).bfloat16()
    t = torch.randint(0, 5003, (777,), device=DEV, generator=g)
    torch.cuda.synchronize()
    want = linear_ce_stats(h, w, t)
    for _ in range(3):
        assert linear_ce_stats(h * 1.0, w * 1.0, t) == want


@pytest.mark.parametrize("lengths,H,K,s0", [
    ([130, 1, 384, 257, 64, 300] * 6, 12, 1, False),      # walked, the list's kernel before them
    ([130, 1, 384, 257, 64, 300] * 6, 12, 3, False),
    ([130, 1, 384, 257, 64, 300] * 6, 12, 2, True),
    ([130, 1, 6000, 257, 64, 300] + [50, 100] * 15, 12, 1, True),      # one of them split: sums, carry and outputs behind the list
    ([130, 1, 6000, 257, 64, 300] + [50, 100] * 15, 12, 3, False),
    ([100, 1, 128, 64], 4, 1, False),                     # finished by the chunk sums
    ([100, 1, 128, 64], 4, 3, False),
])
def test_packed_prefill_that_walks(lengths, H, K, s0):
    x = _scan_inputs(1, H, sum(lengths), K, coef=K > 1, s0=len(lengths) if s0 else 0)
    x["cu"] = _lengths(lengths)
    _check(x, lambda x: ops.pam_scan_tokens(x["q"], x["k"], x["v"], x["gamma"], coef=x.get("coef"), s0=x.get("s0"), cu_seqlens=x["cu"]))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n,top_k,top_p", [(1, 50, 0.9), (64, 0, 0.9), (200, 0, 0.0)])
def test_sampler(n, top_k, top_p, dtype):
    g = torch.Generator(device=DEV).manual_seed(n)
    x = dict(logits=(torch.randn(n, 5008, device=DEV, generator=g) * 3).to(dtype), u=torch.rand(n, device=DEV, generator=g),
             history=torch.randint(0, 5003, (n, 40), device=DEV, generator=g), hist_len=torch.randint(0, 41, (n,), device=DEV, generator=g).int())

    def call(x):
        got = ops.sample_logits(x["logits"][:, :5003], x["u"], temperature=0.8, top_k=top_k, top_p=top_p, repetition_penalty=1.1, history=x["history"],
                                hist_len=x["hist_len"], return_stats=True)
        return [t for t in got] if isinstance(got, (tuple, list)) else [*got.values()] if isinstance(got, dict) else [got]
    _check(x, call)
