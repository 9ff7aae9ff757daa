"""Which form a packed forward-only scan takes, told by what it leaves in its workspace: short batches that finish one-chunk sequences in
the chunk sums, batches that walk, and the sequences that are split among them; with the states that each form puts into pool slots."""
import ctypes as C

import pytest
import torch

from qllm2_b200 import _lib, ops
from qllm2_b200._lib import check, dtype_code, ptr, stream_ptr

pytestmark = pytest.mark.gpu
DEV = "cuda"
LONGEST_BIN = 1023


def _inputs(K, H, lens, with_s0=False):
    g = torch.Generator(device=DEV).manual_seed(K * 11 + H)
    T = sum(lens)
    q, k, v = ((torch.randn(1, H, T, 64, 2, device=DEV, generator=g) * 0.1).bfloat16() for _ in range(3))
    gamma = torch.sigmoid(torch.randn(K, 1, H, T, device=DEV, generator=g) + 2)
    coef = torch.randn(K, 1, H, T, 2, device=DEV, generator=g) if K > 1 else None
    cu = torch.tensor([0] + lens, device=DEV).cumsum(0).int()
    s0 = torch.randn(K, len(lens), H, 64, 64, 2, device=DEV, generator=g) if with_s0 else None
    return q, k, v, gamma, coef, cu, s0


def _align(n):
    return (n + 255) // 256 * 256


def _prefill(K, H, lens, x, dtype):
    """y, the pool, the workspace's state slots as bytes, and the six counters of a call that walks."""
    q, k, v, gamma, coef, cu, s0 = x
    n, T = len(lens), sum(lens)
    pool = torch.full((n + 1, 1, K, H, 64, 64, 2), 7.0, device=DEV, dtype=dtype)
    slots = torch.arange(n, device=DEV, dtype=torch.int32)
    y = torch.empty(1, T, H * 64, 2, device=DEV, dtype=torch.bfloat16)
    a = _lib.ScanArgs()
    a.q, a.k, a.v, a.gamma, a.coef, a.s0, a.cu_seqlens, a.y = (ptr(t) for t in (q, k, v, gamma, coef, s0, cu, y))
    a.B, a.H, a.T, a.d, a.K, a.S, a.chunk, a.io_dtype, a.q_scale, a.gamma_eps = 1, H, T, 64, K, n, 64, 1, 0.125, 1e-6
    total = _lib.lib().qpam_scan_workspace_bytes(C.byref(a), 0)
    ws = torch.full((total,), 0x5A, dtype=torch.uint8, device=DEV)
    a.workspace, a.workspace_bytes = ws.data_ptr(), ws.numel()
    n0 = _lib.launch_count()
    check(_lib.lib().qpam_scan_prefill(C.byref(a), pool.data_ptr(), dtype_code(dtype), n + 1, 1, 0, ptr(slots), stream_ptr()), "qpam_scan_prefill")
    launches = _lib.launch_count() - n0
    first, state_slots = _align(4 * (n + 1)), K * H * (T // 128 + 2 * n)      # chunk prefix | state slots | decays | counters and list
    jobs = first + _align(state_slots * 64 * 64 * 8) + _align(state_slots * 4)
    states = ws[first:first + state_slots * 64 * 64 * 8]
    assert bool((pool[n] == 7).all()) and _lib.device_status() == 0
    return y, pool[:n, 0], states, ws[jobs:jobs + 24].view(torch.int32).tolist(), launches


def _training_form(K, x):
    q, k, v, gamma, coef, cu, s0 = x
    return ops.pam_scan(q, k, v, gamma.clone().requires_grad_(True), coef=coef, cu_seqlens=cu, s0=s0, token_major=True)


@pytest.mark.parametrize("K", [1, 3])
@pytest.mark.parametrize("with_s0", [False, True])
def test_one_chunk_sequences_finish_in_the_sums(K, with_s0):
    """Few short prompts: their sums go to the pool and nowhere else; a state before them takes the carry."""
    lens, H = [1, 128, 64, 0, 127], 2
    x = _inputs(K, H, lens, with_s0)
    y_ref, s_ref = _training_form(K, x)
    for dtype in (torch.float32, torch.bfloat16):
        y, pool, states, _, launches = _prefill(K, H, lens, x, dtype)
        assert launches == 4
        assert torch.equal(y, y_ref.detach()) and torch.equal(pool, s_ref.detach().transpose(0, 1).to(dtype))
        assert bool((states == 0x5A).all()) != with_s0


@pytest.mark.parametrize("K", [1, 3])
def test_a_long_sequence_beside_short_ones_keeps_three_passes_for_itself(K):
    """The final state of a split sequence in its pool slot, behind a list of walked ones."""
    lens, H = [5, 3000, 0] + [100 + i for i in range(26)], 12
    x = _inputs(K, H, lens)
    y_ref, s_ref = _training_form(K, x)
    for dtype in (torch.float32, torch.bfloat16):
        y, pool, _, (_, _, jobs, split_jobs, carry, above), launches = _prefill(K, H, lens, x, dtype)
        assert launches == 4 and carry == 1 and 1 <= above < 24 and jobs - split_jobs == 27 and split_jobs == 24
        assert torch.equal(y, y_ref.detach()) and torch.equal(pool, s_ref.detach().transpose(0, 1).to(dtype))


def _cost(chunks, above, H, ctas):
    walked, split = [c for c in chunks if c <= above], [c for c in chunks if c > above]
    per = H / ctas
    t = max(0.6 * max(walked, default=0) + 0.4 * min(max(walked, default=0), per * sum(chunks)), per * (sum(walked) + 0.8 * sum(split)))
    return t + 1 + 0.7 * per * sum(split) + 0.01 * max(split) if split else t


@pytest.mark.parametrize("K,H,lens", [
    (1, 16, [128 * (1 + i) for i in range(24)]),                                                   # evenly spread: all of them walk
    (1, 12, [3000] * 8 + [60] * 24),                                                               # a quarter is long
    (3, 6, [int(60 * 1.09 ** i) for i in range(56)]),                                              # a tail of ever longer ones
    (2, 12, [9000, 700] + [90] * 30),
    (1, 1, [int(1 + (37 * i) % 128) for i in range(1500)] + [128 * 1100, 128 * 1023, 128 * 40]),   # past the last bin, more than threads
])
def test_the_cheapest_split(K, H, lens):
    x = _inputs(K, H, lens)
    ctas = 2 * torch.cuda.get_device_properties(0).multi_processor_count
    assert len(lens) * H * 37 >= ctas * 40 or (K == 1 and len(lens) * H > ctas)
    _, _, _, (_, _, jobs, split_jobs, carry, above), _ = _prefill(K, H, lens, x, torch.bfloat16)
    chunks = [-(-n // 128) for n in lens]
    split = [c for c in chunks if c > above]
    assert split_jobs == sum(split) and jobs == sum(split) + len(chunks) - len(split) and carry == (1 if split else 0)
    best = min(_cost(chunks, min(c, LONGEST_BIN - 1) if c < LONGEST_BIN else 1 << 29, H, ctas) for c in [0] + chunks)
    assert _cost(chunks, above, H, ctas) <= best * (1 + 1e-5)      # (fp32 on the device: 24 bits)


@pytest.mark.parametrize("K", [1, 3])
@pytest.mark.parametrize("with_s0", [False, True])
def test_final_states_alone(K, with_s0):
    """A call for final states: the carry passes over the chunk sums and writes none of the slots that only an output would read."""
    lens, H = [300, 1, 0, 128, 513], 2
    q, k, v, gamma, coef, cu, s0 = x = _inputs(K, H, lens, with_s0)
    n, T = len(lens), sum(lens)
    s = torch.empty(K, n, H, 64, 64, 2, device=DEV)
    a = _lib.ScanArgs()
    a.q, a.k, a.v, a.gamma, a.s0, a.cu_seqlens, a.s_final = (ptr(t) for t in (q, k, v, gamma, s0, cu, s))
    a.B, a.H, a.T, a.d, a.K, a.S, a.chunk, a.io_dtype, a.q_scale, a.gamma_eps = 1, H, T, 64, K, n, 64, 1, 0.125, 1e-6
    ws = torch.full((_lib.lib().qpam_scan_workspace_bytes(C.byref(a), 0),), 0x5A, dtype=torch.uint8, device=DEV)
    a.workspace, a.workspace_bytes = ws.data_ptr(), ws.numel()
    check(_lib.lib().qpam_scan_fwd(C.byref(a), stream_ptr()), "qpam_scan_fwd")
    assert torch.equal(s, _training_form(K, x)[1].detach()) and torch.equal(s, ops.pam_scan_states(k, v, gamma, s0=s0, cu_seqlens=cu))
    slots = T // 128 + 2 * n
    first = _align(4 * (n + 1))
    states = ws[first:first + K * H * slots * 64 * 64 * 8].view(K, H, slots, 64 * 64 * 8)
    at = 0
    for length in lens:                                    # a sequence's first slot is the state before it
        assert bool((states[:, :, at] == 0x5A).all())
        at += -(-length // 128) + 1


@pytest.mark.parametrize("K", [1, 3])
@pytest.mark.parametrize("with_s0", [False, True])
def test_refused_descriptor(K, with_s0):
    """Lengths that decrease, in a batch that would walk: the status word says so, no token is touched, and every sequence counts as
    empty, as in the batches that do not walk."""
    lens, H = [60] * 30, 12
    q, k, v, gamma, coef, cu, s0 = _inputs(K, H, lens, with_s0)
    cu[5] = cu[4] - 1
    n, T = len(lens), sum(lens)
    y, s = torch.full((1, T, H * 64, 2), 3.0, device=DEV, dtype=torch.bfloat16), torch.full((K, n, H, 64, 64, 2), 3.0, device=DEV)
    a = _lib.ScanArgs()
    a.q, a.k, a.v, a.gamma, a.coef, a.s0, a.cu_seqlens, a.y, a.s_final = (ptr(t) for t in (q, k, v, gamma, coef, s0, cu, y, s))
    a.B, a.H, a.T, a.d, a.K, a.S, a.chunk, a.io_dtype, a.q_scale, a.gamma_eps = 1, H, T, 64, K, n, 64, 1, 0.125, 1e-6
    ws = torch.empty(_lib.lib().qpam_scan_workspace_bytes(C.byref(a), 0), dtype=torch.uint8, device=DEV)
    a.workspace, a.workspace_bytes = ws.data_ptr(), ws.numel()
    assert _lib.device_status() == 0
    try:
        check(_lib.lib().qpam_scan_fwd_tokens(C.byref(a), stream_ptr()), "qpam_scan_fwd_tokens")
        torch.cuda.synchronize()
    finally:
        assert _lib.device_status(clear=True) == 301
    assert bool((y == 3).all()) and torch.equal(s, torch.zeros_like(s) if s0 is None else s0)
