"""The work that this framework is used for, as cases that can be timed and compared.

Six kinds of work, each over the range of sizes it is met with:

  scan     one PAM scan of a training step, forward and backward, through ``ops.pam_scan``
  prefill  the packed ragged scan that absorbs a batch of prompts, through ``ops.pam_scan_tokens``
  ce       the tied head with its cross-entropy, forward and backward, through ``fused_linear_cross_entropy``
  sample   one draw for every row of logits, through ``ops.sample_logits``
  train    forward, loss and backward of a whole model, through ``V11LM`` under bf16 autocast
  serve    prompts to tokens through ``ContinuousBatcher`` (one packed prefill, then captured decode steps)

``listed()`` names the sizes that stand for each of them, ``draw()`` gives further sizes of the same ranges.
"""
from __future__ import annotations

import math
import random

import torch

from qllm2_b200 import model as M
from qllm2_b200 import ops
from qllm2_b200.fused_ce import fused_linear_cross_entropy
from qllm2_b200.serving import ContinuousBatcher

DTYPES = {"bf16": torch.bfloat16, "fp32": torch.float32}
SIZES = {"bf16": 2, "fp32": 4}
#: decay logits of the states: the learned offsets of a K-state layer spread them from fast to slow
STATE_LOGITS = {1: [3.0], 2: [1.0, 5.0], 3: [1.0, 3.0, 5.0]}


def listed():
    return [
        # a fine-tuning step on one short example: a single ragged chunk, so launches and host work are all there is
        dict(name="scan short example", kind="scan", dtype="bf16", B=1, H=6, T=93, d=64, K=1),
        # the layer of the 8-block training configuration: 8 sequences of 2048 tokens, six heads
        dict(name="scan training layer", kind="scan", dtype="bf16", B=8, H=6, T=2048, d=64, K=1),
        # the same layer with three phase-routed states and their read-out weights, as the chat models train it
        dict(name="scan three states", kind="scan", dtype="bf16", B=8, H=6, T=2048, d=64, K=3),
        # complex64 parity runs of a small layer
        dict(name="scan complex64", kind="scan", dtype="fp32", B=2, H=4, T=512, d=32, K=1),
        # long documents, 512 to 16384 tokens each, absorbed in one packed batch (one state, 16 heads)
        dict(name="prefill long documents", kind="prefill", sequences=32, shortest=512, longest=16384, H=16, K=1),
        # chat prompts admitted together by a serving engine (three states, 12 heads)
        dict(name="prefill chat prompts", kind="prefill", sequences=48, shortest=32, longest=1024, H=12, K=3),
        # the head and loss of a training batch: 8192 rows against the whole vocabulary
        dict(name="loss training batch", kind="ce", N=8192, D=384, V=50261, masked=False),
        # the head and loss of one chat example: a few hundred rows, the prompt's masked out or ignored
        dict(name="loss one example", kind="ce", N=509, D=384, V=50257, masked=True),
        # one token for each of 256 live sequences, with every filter of the chat settings
        dict(name="sample 256 sequences", kind="sample", dtype="bf16", rows=256, V=50261, top_k=50, top_p=0.9, penalty=1.1),
        # a step of the 8-block three-state model on 8 x 2048 tokens
        dict(name="train step", kind="train", B=8, T=2048, blocks=8, K=3),
        # one user's chat turn
        dict(name="serve one user", kind="serve", users=1, shortest=211, longest=211, new=24, K=3),
        # a full engine: 256 short prompts, all decoding together
        dict(name="serve 256 users", kind="serve", users=256, shortest=16, longest=128, new=16, K=3),
    ]


def _log_between(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    kind = rng.choice(["scan", "scan", "prefill", "ce", "sample", "train", "serve"])
    if kind == "scan":
        dtype = rng.choice(["bf16", "bf16", "fp32"])
        T = _log_between(rng, 17, 2048)
        if dtype == "bf16":
            return dict(kind=kind, dtype=dtype, B=_log_between(rng, 1, 8), H=rng.choice([6, 12]) if T <= 1024 else 6, T=T, d=64, K=rng.choice([1, 2, 3]))
        return dict(kind=kind, dtype=dtype, B=rng.randint(1, 4), H=rng.choice([2, 4, 6]), T=T, d=rng.choice([32, 64]), K=1)
    if kind == "prefill":
        K = rng.choice([1, 3])
        shortest = _log_between(rng, 16, 512)
        longest = _log_between(rng, 2 * shortest, 16384 if K == 1 else 4096)
        most = min(32, 280000 // longest) if K == 1 else min(48, 60000 // longest)
        return dict(kind=kind, sequences=rng.randint(1, most), shortest=shortest, longest=longest, H=rng.choice([6, 12, 16]), K=K)
    if kind == "ce":
        D = rng.choice([384, 768])
        return dict(kind=kind, N=_log_between(rng, 60, 8192 if D == 384 else 4096), D=D, V=rng.choice([50257, 50261]), masked=rng.random() < 0.5)
    if kind == "sample":
        top_k, top_p = rng.choice([(50, 0.0), (50, 0.9), (0, 0.9), (rng.randint(5, 200), 0.95), (0, 0.0)])
        return dict(kind=kind, dtype=rng.choice(["bf16", "fp32"]), rows=_log_between(rng, 1, 256), V=rng.choice([50257, 50261]), top_k=top_k,
                    top_p=top_p, penalty=rng.choice([1.0, 1.1, 1.3]))
    if kind == "train":
        T = _log_between(rng, 65, 2048)
        return dict(kind=kind, B=_log_between(rng, 1, 8), T=T, blocks=rng.randint(2, 8), K=rng.choice([1, 3]))
    users = _log_between(rng, 1, 256)
    shortest = rng.randint(8, 64)
    return dict(kind=kind, users=users, shortest=shortest, longest=max(shortest + 1, min(1024, _log_between(rng, 64, 18000) // users)), new=rng.randint(4, 16),
                K=rng.choice([1, 3]))


# ------------------------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _lengths(case, count):
    """The lengths of a case's sequences: part of the case, so the work of every batch of it is the same."""
    rng = random.Random("%d %d %d" % (count, case["shortest"], case["longest"]))
    return [rng.randint(case["shortest"], case["longest"]) for _ in range(count)]


def _tokens(g, B, H, T, d, dtype):
    """Complex-normal token tensor, std 1/sqrt(2d) for each component (normalised rows, as a trained projection gives)."""
    return (torch.randn(B, H, T, d, 2, device="cuda", generator=g) * (2 * d) ** -0.5).to(dtype)


def _decays(g, K, B, H, T):
    logits = torch.tensor(STATE_LOGITS[K], device="cuda").view(K, 1, 1, 1)
    return torch.sigmoid(torch.randn(K, B, H, T, device="cuda", generator=g) + logits)


def _config(K, **kw):
    return M.V11Config(n_states=K, gate_content_aware=True, dropout=0.0, gradient_checkpointing=False, **kw)


def _model(cfg, seed, dtype, confident):
    """A model with weights of trained size.  `confident`: the head maps a hidden state to its own embedding, so that the
    arg-max has the clear margin it has in a trained model (random heads leave near-ties everywhere)."""
    with torch.device("meta"):
        net = M.V11LM(cfg)
    net = net.to(dtype).to_empty(device="cuda")
    g = _gen(seed)
    with torch.no_grad():
        for name, p in net.named_parameters():
            last = name.rsplit(".", 1)[-1]
            if last in ("weight_real", "weight_imag"):                 # complex projections keep the variance; the two that
                std = (2 * p.shape[1]) ** -0.5                         # write to the residual stream add a third of it
                p.normal_(0, std * (0.3 if "down_proj" in name or "o_proj" in name else 1.0), generator=g)
            elif last == "state_dt_offset":
                p.copy_(torch.linspace(-cfg.state_dt_spread, cfg.state_dt_spread, cfg.n_states))
            elif last == "dt_bias":
                p.fill_(cfg.base_dt_bias)
            elif last in ("scale", "beta", "cgu_scale"):
                p.fill_(1.0)
            elif last == "pam_scale":
                p.fill_(0.1)
            elif "protect_gate.bias" in name:
                p.fill_(cfg.protect_gate_bias)
            elif p.dim() == 2:                                          # embeddings and the small gate projections
                p.normal_(0, 0.02, generator=g)
            else:
                p.zero_()
        if confident:
            torch.nn.init.eye_(net.lm_head_proj.weight_real)
            net.lm_head_proj.weight_imag.zero_()
    rope = M.build_rope_cache(cfg.max_seq_len, cfg.head_dim).to("cuda")
    for blk in net.blocks:
        blk.pam.rope_cache = rope
    return net


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    if kind == "scan":
        B, H, T, d, K = (case[k] for k in "BHTdK")
        dt = DTYPES[case["dtype"]]
        leaves = [_tokens(g, B, H, T, d, dt) for _ in range(3)]
        leaves.append(_decays(g, K, B, H, T))
        if K > 1:
            leaves.append(torch.randn(K, B, H, T, 2, device="cuda", generator=g))
        dy = (torch.randn(B, H, T, d, 2, device="cuda", generator=g) * 0.5 ** 0.5).to(dt)
        return dict(kind=kind, leaves=[t.requires_grad_(True) for t in leaves], dy=dy)
    if kind == "prefill":
        H, K = case["H"], case["K"]
        lengths = torch.tensor(_lengths(case, case["sequences"]))
        T = int(lengths.sum())
        cu = torch.zeros(len(lengths) + 1, dtype=torch.int32)
        cu[1:] = lengths.cumsum(0)
        q, k, v = (_tokens(g, 1, H, T, 64, torch.bfloat16) for _ in range(3))
        return dict(kind=kind, q=q, k=k, v=v, gamma=_decays(g, K, 1, H, T), cu=cu.to("cuda"),
                    coef=torch.randn(K, 1, H, T, 2, device="cuda", generator=g) if K > 1 else None)
    if kind == "ce":
        N, F, V = case["N"], 2 * case["D"], case["V"]
        h = torch.randn(N, F, device="cuda", generator=g).bfloat16().requires_grad_(True)
        w = (torch.randn(V, F, device="cuda", generator=g) * 0.02).bfloat16().requires_grad_(True)
        targets = torch.randint(0, V, (N,), device="cuda", generator=g)
        mask = None
        if case["masked"]:
            targets[torch.rand(N, device="cuda", generator=g) < 0.1] = -100
            mask = (torch.rand(N, device="cuda", generator=g) < 0.7).float()
        return dict(kind=kind, h=h, w=w, targets=targets, mask=mask)
    if kind == "sample":
        n, V = case["rows"], case["V"]
        ld = (V + 7) // 8 * 8                                           # rows as `ops.head_logits` lays them out
        logits = (torch.randn(n, ld, device="cuda", generator=g) * 2.0).to(DTYPES[case["dtype"]])[:, :V]
        return dict(kind=kind, logits=logits, uniforms=torch.rand(n, device="cuda", generator=g),
                    history=torch.randint(0, V, (n, 513), device="cuda", generator=g),
                    hist_len=torch.randint(16, 513, (n,), device="cuda", generator=g).int(),
                    settings=dict(temperature=0.8, top_k=case["top_k"], top_p=case["top_p"], repetition_penalty=case["penalty"]))
    if kind == "train":
        B, T = case["B"], case["T"]
        net = _model(_config(case["K"], vocab_size=50261, dim=384, n_heads=6, n_layers=case["blocks"], chunk_size=64), seed, torch.float32, False).train()
        parts = [net.embed] + list(net.blocks) + [torch.nn.ModuleList([net.embed_norm, net.output_norm, net.lm_head_proj, net.lm_head_norm])]
        buckets = []
        for part in parts:                                              # gradients live in one flat bucket for each block, as a
            ps = list(part.parameters())                                # data-parallel trainer keeps them
            flat = torch.zeros(sum(p.numel() for p in ps), device="cuda")
            at = 0
            for p in ps:
                p.grad = flat[at:at + p.numel()].view_as(p)
                at += p.numel()
            buckets.append(flat)
        ids = torch.randint(0, 50261, (B, T + 1), device="cuda", generator=g)
        return dict(kind=kind, net=net, buckets=buckets, x=ids[:, :-1].contiguous(), y=ids[:, 1:].contiguous())
    cfg = _config(case["K"], vocab_size=50261, dim=768, n_heads=12, n_layers=12, max_seq_len=2048)
    net = _model(cfg, seed, torch.bfloat16, True).eval()
    eng = ContinuousBatcher(net, n_slots=case["users"], cuda_graph=True, max_position=2048)
    eng.warmup()
    lengths = _lengths(case, case["users"])
    flat = torch.randint(0, 50261, (sum(lengths),), device="cuda", generator=g).tolist()
    prompts = []
    for n in lengths:
        prompts.append(flat[:n])
        flat = flat[n:]
    return dict(kind=kind, eng=eng, prompts=prompts, new=case["new"])


# ------------------------------------------------------------------------------------ one pass
def run(s):
    kind = s["kind"]
    if kind == "scan":
        q, k, v, gamma = s["leaves"][:4]
        y, last = ops.pam_scan(q, k, v, gamma, coef=s["leaves"][4] if len(s["leaves"]) > 4 else None)
        return [y, last, *torch.autograd.grad(y, s["leaves"], s["dy"])]
    if kind == "prefill":
        return ops.pam_scan_tokens(s["q"], s["k"], s["v"], s["gamma"], coef=s["coef"], cu_seqlens=s["cu"])
    if kind == "ce":
        loss = fused_linear_cross_entropy(s["h"], s["w"], s["targets"], mask=s["mask"])
        return [loss, *torch.autograd.grad(loss, [s["h"], s["w"]])]
    if kind == "sample":
        return ops.sample_logits(s["logits"], s["uniforms"], history=s["history"], hist_len=s["hist_len"], return_stats=True, **s["settings"])
    if kind == "train":
        net = s["net"]
        for flat in s["buckets"]:
            flat.zero_()
        with torch.autocast("cuda", dtype=torch.bfloat16):
            loss, _ = net.fused_ce_loss(s["x"], s["y"])
        loss.backward()
        return [loss, *s["buckets"]]
    eng = s["eng"]
    rids = [eng.submit(p, s["new"]) for p in s["prompts"]]
    done = eng.run()
    eng.sched.finished.clear()
    return [torch.tensor([done[r] for r in rids]), eng.pool]


# ------------------------------------------------------------------------------------ what a pass cannot do without
def _scan_flops(d, K):
    """Causal-useful flops of the forward scan for one token and head, in chunks of 64."""
    return 8 * 65 * d + K * 16 * d * d


def _block_macs(D, H, K, hidden):
    """Real multiply-adds of one block for one token."""
    inner = H * 64
    return 4 * D * (2 * hidden) + 4 * hidden * D + 4 * D * 3 * inner + 4 * inner * D + 2 * D * H * 2 + (D * H * K if K > 1 else 0)


def work(case):
    kind = case["kind"]
    if kind == "scan":
        B, H, T, d, K = (case[k] for k in "BHTdK")
        n = B * H * T
        return {"bytes": n * (16 * d * SIZES[case["dtype"]] + K * (8 + (16 if K > 1 else 0))) + K * B * H * d * d * 8, "flops": 3 * n * _scan_flops(d, K)}
    if kind == "prefill":
        K, H = case["K"], case["H"]
        n = H * sum(_lengths(case, case["sequences"]))
        return {"bytes": n * (8 * 64 * 2 + K * (4 + (8 if K > 1 else 0))) + K * H * case["sequences"] * 64 * 64 * 8, "flops": n * _scan_flops(64, K)}
    if kind == "ce":
        N, F, V = case["N"], 2 * case["D"], case["V"]
        return {"bytes": 2 * 2 * (N * F + V * F) + 8 * N + (4 * N if case["masked"] else 0), "flops": 6 * N * V * F}
    if kind == "sample":
        return {"bytes": case["rows"] * (case["V"] * SIZES[case["dtype"]] + 8 * 264 + 28), "flops": 4 * case["rows"] * case["V"]}
    if kind == "train":
        B, T, K, L, D, H, V = case["B"], case["T"], case["K"], case["blocks"], 384, 6, 50261
        macs = L * _block_macs(D, H, K, 3 * D) + 4 * D * D + 2 * D * V
        params = L * _block_macs(D, H, K, 3 * D) / 2 + 2 * D * D + 2 * D * V
        return {"bytes": 8 * params + 16 * B * T, "flops": 6 * macs * B * T + 3 * L * B * T * H * _scan_flops(64, K)}
    n, new, K, L, D, H, V = case["users"], case["new"], case["K"], 12, 768, 12, 50261
    total = sum(_lengths(case, n))
    macs = L * _block_macs(D, H, K, 3 * D) + 4 * D * D
    weights = 2 * (macs / 2 + 2 * D * V)                                # bf16, real and imaginary part once each
    state = n * L * K * H * 64 * 64 * 2 * 2
    tokens = total + n * (new - 1)
    return {"bytes": new * weights + state * (2 * new - 1), "flops": 2 * macs * tokens + 4 * D * V * n * new + L * H * (total * _scan_flops(64, K) + n * (new - 1) * K * 16 * 64 * 64)}


def tolerance(case):
    kind = case["kind"]
    if kind == "scan":
        return {"rel": 1e-2} if case["dtype"] == "bf16" else {"rel": 2e-5}
    if kind in ("prefill", "ce"):
        return {"rel": 1e-2}
    if kind == "sample":
        return {"rel": 1e-4, "differ": 0.01}                            # a draw on the edge between two tokens may fall to the other
    return {"rel": 2e-2, "max": 0.9, "differ": 0.01}                    # bf16 through a whole model
