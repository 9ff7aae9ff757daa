"""Device-side token sampling (qpam_sample_logits) against the CPU restatement of the reference's sampling block
(v11/model.py:1221-1244): the filtered distribution (kept count, kept mass) and the inverse-CDF draw."""
import numpy as np
import pytest
import torch

from oracle import sampling_oracle as so
from qllm2_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _check_rows(logits, hist, hist_len, u, ids, stats, cfg, count_exact=True):
    """Kept count: exact where only integer logic decides it (top-k, no filter).  Where the nucleus closes, the
    float32 mass sums of the kernel and the float64 sums here may put the boundary a few negligible tokens apart
    (the tail tokens there weigh ~1e-6 of the total, the rounding noise of any float32 cumulative sum, the
    reference's included): then the kept MASS must agree to 5e-5 of the total."""
    lg = logits.float().cpu().numpy()
    nucleus = 0 < cfg["top_p"] < 1
    for r in range(lg.shape[0]):
        h = None if hist is None else hist[r, :(hist.shape[1] if hist_len is None else int(hist_len[r]))].tolist()
        p = so.filtered_probs(lg[r], h, **cfg)
        kept = int((p > 0).sum())
        if count_exact and not nucleus:
            assert int(stats[r, 2]) == kept, (r, int(stats[r, 2]), kept)
        else:
            full = so.filtered_probs(lg[r], h, **{**cfg, "top_p": 0.0})       # distribution before the nucleus filter
            assert abs(float(stats[r, 1]) / float(stats[r, 3]) - full[p > 0].sum()) < 5e-5, (r, stats[r], kept)
            assert abs(int(stats[r, 2]) - kept) <= max(3, 0.02 * kept), (r, int(stats[r, 2]), kept)
        c = np.cumsum(p)
        i = int(ids[r])
        if int(stats[r, 2]) == kept:
            assert p[i] > 0, (r, i)
        lo, hi = (c[i - 1] if i > 0 else 0.0), c[i]
        assert lo - 5e-5 <= float(u[r]) <= hi + 5e-5, (r, i, lo, float(u[r]), hi)


@pytest.mark.parametrize("cfg", [
    dict(temperature=0.8, top_k=50, top_p=0.9, repetition_penalty=1.1),
    dict(temperature=1.0, top_k=0, top_p=0.95, repetition_penalty=1.0),
    dict(temperature=1.3, top_k=20, top_p=0.0, repetition_penalty=1.2),
    dict(temperature=1.0, top_k=0, top_p=0.0, repetition_penalty=1.0),
    dict(temperature=0.7, top_k=1, top_p=0.5, repetition_penalty=1.0),
])
@pytest.mark.parametrize("V", [50261, 97, 70001])
def test_rows_match_reference_filter_and_inverse_cdf(cfg, V):
    n = 24
    g = torch.Generator().manual_seed(V + int(cfg["top_k"]))
    logits = (torch.randn(n, V, generator=g) * 3.0).to(DEV)
    hist = torch.randint(0, V, (n, 40), generator=g)
    u = torch.rand(n, generator=g)
    ids, stats = ops.sample_logits(logits, u.to(DEV), history=hist.to(DEV), return_stats=True, **cfg)
    _check_rows(logits, hist.numpy(), None, u.numpy(), ids.cpu().numpy(), stats.cpu().numpy(), cfg)


def test_bf16_logits_with_ties():
    """bf16 logits repeat values many times over 50k entries: the whole tie group at either threshold stays."""
    n, V = 16, 50261
    g = torch.Generator().manual_seed(5)
    logits = (torch.randn(n, V, generator=g) * 2.0).bfloat16().to(DEV)
    u = torch.rand(n, generator=g)
    cfg = dict(temperature=0.9, top_k=40, top_p=0.9, repetition_penalty=1.0)
    ids, stats = ops.sample_logits(logits, u.to(DEV), return_stats=True, **cfg)
    _check_rows(logits, None, None, u.numpy(), ids.cpu().numpy(), stats.cpu().numpy(), cfg, count_exact=False)


def test_frequencies_follow_the_filtered_distribution():
    """One row, 8192 evenly spaced uniforms: every token is drawn as often as its probability says (to 2 / n)."""
    V, n = 1000, 8192
    g = torch.Generator().manual_seed(9)
    row = torch.randn(V, generator=g) * 2.5
    cfg = dict(temperature=1.1, top_k=64, top_p=0.92, repetition_penalty=1.0)
    u = (torch.arange(n, dtype=torch.float32) + 0.5) / n
    ids = ops.sample_logits(row[None].expand(n, V).contiguous().to(DEV), u.to(DEV), **cfg).cpu().numpy()
    p = so.filtered_probs(row.numpy(), None, **cfg)
    freq = np.bincount(ids, minlength=V) / n
    assert np.abs(freq - p).max() <= 2.0 / n + 2e-5, float(np.abs(freq - p).max())
    assert set(np.nonzero(freq)[0]) <= set(np.nonzero(p)[0])


def test_slots_lengths_and_append():
    """Rows map to history rows through slot ids; only hist_len[slot] entries count for the penalty; the drawn id is
    appended behind them; a slot of -1 is a padded row (id 0, nothing appended)."""
    V, rows, cap = 311, 6, 12
    g = torch.Generator().manual_seed(21)
    logits = torch.randn(4, V, generator=g) * 4.0
    hist = torch.randint(0, V, (rows, cap), generator=g)
    hist_len = torch.tensor([3, 0, 12, 5, 7, 1], dtype=torch.int32)
    slots = torch.tensor([4, -1, 0, 2], dtype=torch.int32)
    u = torch.rand(4, generator=g)
    cfg = dict(temperature=1.0, top_k=0, top_p=0.0, repetition_penalty=1.5)
    hd, ld = hist.to(DEV), hist_len.to(DEV)
    ids = ops.sample_logits(logits.to(DEV), u.to(DEV), history=hd, hist_len=ld, slot_ids=slots.to(DEV), append=True, **cfg)
    ids = ids.cpu().numpy()
    assert ids[1] == 0
    new_len, new_hist = ld.cpu().numpy(), hd.cpu().numpy()
    for r, s in enumerate(slots.tolist()):
        if s < 0:
            continue
        ln = int(hist_len[s])
        p = so.filtered_probs(logits[r].numpy(), hist[s, :ln].tolist(), **cfg)
        c = np.cumsum(p)
        lo, hi = (c[ids[r] - 1] if ids[r] > 0 else 0.0), c[ids[r]]
        assert lo - 2e-5 <= float(u[r]) <= hi + 2e-5
        if ln < cap:
            assert new_len[s] == ln + 1 and new_hist[s, ln] == ids[r]
        else:       # a full row keeps its length and its entries
            assert new_len[s] == ln and (new_hist[s] == hist[s].numpy()).all()
    untouched = [s for s in range(rows) if s not in slots.tolist()]
    assert (new_len[untouched] == hist_len.numpy()[untouched]).all()


def test_bad_arguments_are_refused():
    from qllm2_b200._lib import QPamError
    logits = torch.zeros(2, 10, device=DEV)
    with pytest.raises(QPamError):
        ops.sample_logits(logits, temperature=0.0)
    with pytest.raises(QPamError):
        ops.sample_logits(logits, torch.zeros(3, device=DEV))
    with pytest.raises(QPamError):
        ops.sample_logits(logits, append=True)


@pytest.mark.parametrize("n,V,dtype,shift,cfg", [
    (3, 5, "fp32", 1, dict(top_k=2, top_p=0.9, repetition_penalty=1.3)),           # fewer groups than lanes
    (150, 333, "bf16", 3, dict(top_k=50, top_p=0.9, repetition_penalty=1.1)),      # 512 threads a row; rows start anywhere
    (150, 5003, "fp32", 0, dict(top_k=384, top_p=0.95, repetition_penalty=1.1)),   # the largest top-k of the list
    (4, 5003, "fp32", 2, dict(top_k=385, top_p=0.95, repetition_penalty=1.1)),     # the first beyond it
    (150, 5003, "bf16", 1, dict(top_k=0, top_p=0.9, repetition_penalty=1.1)),
    (2, 700001, "fp32", 1, dict(top_k=50, top_p=0.9, repetition_penalty=1.1)),     # a block is more than four groups
    (2, 700001, "bf16", 0, dict(top_k=0, top_p=0.6, repetition_penalty=1.1)),
    (4, 50261, "bf16", 0, dict(top_k=0, top_p=0.999, repetition_penalty=1.0)),
    (4, 4096, "fp32", 0, dict(top_k=0, top_p=1e-6, repetition_penalty=1.0)),       # the largest value alone
])
def test_blocks_stretches_and_marks(n, V, dtype, shift, cfg):
    """Where the passes can go wrong: rows off 16 bytes, blocks of several steps, both widths of a CTA, every route, penalised
    tokens (the row's largest among them, and tokens on the edges of the warps' stretches)."""
    g = torch.Generator().manual_seed(V + n)
    wide = (torch.randn(n, V + 5, generator=g) * 3.0)
    wide = wide.bfloat16() if dtype == "bf16" else wide
    logits = wide.to(DEV)[:, shift:shift + V]
    hist = torch.randint(0, V, (n, 40), generator=g)
    hist[:, 0] = logits.float().argmax(1).cpu()
    hist[:, 1], hist[:, 2], hist[:, 3] = 0, V - 1, V // 2
    hist[:, 4] = hist[:, 0]                       # the penalty applies once
    u = torch.rand(n, generator=g)
    cfg = dict(temperature=0.8, **cfg)
    ids, stats = ops.sample_logits(logits, u.to(DEV), history=hist.to(DEV), return_stats=True, **cfg)
    _check_rows(logits, hist.numpy(), None, u.numpy(), ids.cpu().numpy(), stats.cpu().numpy(), cfg, count_exact=dtype == "fp32")


def test_infinite_temperature_and_masked_logits():
    V = 1000
    logits = torch.randn(3, V, device=DEV)
    u = torch.tensor([0.0, 0.5, 0.9999], device=DEV)
    ids, stats = ops.sample_logits(logits, u, temperature=float("inf"), history=torch.zeros(3, 4, dtype=torch.int64, device=DEV),
                                   repetition_penalty=1.1, return_stats=True)
    assert (stats[:, 2] == V).all() and ids.tolist() == [0, 500, 999]      # uniform over the vocabulary
    logits[:, 10:] = float("-inf")
    for cfg in (dict(top_k=20), dict(top_p=0.9), dict()):
        ids, stats = ops.sample_logits(logits, u, return_stats=True, **cfg)
        assert (ids < 10).all() and (stats[:, 2] <= 10).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("cfg", [dict(), dict(top_k=20), dict(top_k=500), dict(repetition_penalty=1.2)])
def test_tokens_far_below_the_maximum_at_a_low_temperature(dtype, cfg):
    """At temperature 0.05 a logit 4.5 below the maximum has the mass e^-90, a denormal number: it is counted and can be drawn
    (fp32 masses reach down to e^-103), whichever way the row takes; beyond that a token has no mass."""
    V = 1000
    gaps = torch.full((V,), 130.0)
    gaps[:12] = torch.tensor([95.0, 0.0, 20.0, 50.0, 86.0, 88.5, 91.0, 99.0, 100.5, 106.0, 107.0, 110.0])
    gaps[V - 1] = 98.0
    logits = (gaps * -0.05).to(dtype).to(DEV)[None].expand(3, V).contiguous()
    scaled = logits[0].double().cpu() / 0.05
    far = scaled.max() - scaled
    assert not ((far > 102.5) & (far < 104.5)).any()            # e^-102.5 is above the smallest number, e^-104.5 below its half
    massive = far < 103.5
    u = torch.tensor([0.0, 0.5, 1.0 - 2.0 ** -24], device=DEV)
    hist = torch.tensor([[V - 2]] * 3, device=DEV)              # (a token without mass, whatever the penalty)
    ids, stats = ops.sample_logits(logits, u, temperature=0.05, history=hist, return_stats=True, **cfg)
    assert (stats[:, 2] == int(massive.sum())).all(), (stats[:, 2], int(massive.sum()))
    assert ids.tolist() == [0, 1, 1]                            # u = 0: the first token with any mass
    assert torch.allclose(stats[:, 1].double().cpu(), torch.exp(-far).sum().expand(3), rtol=1e-6)
