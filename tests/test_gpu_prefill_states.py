"""Final states of a forward-only scan: a sequence of no, one, two or more chunks, with and without an initial state, into the
s_final tensor and straight into pool slots, against the training forward (which writes every state) and a host copy."""
import ctypes as C

import pytest
import torch

from qllm2_b200 import _lib, ops
from qllm2_b200._lib import check, dtype_code, ptr, stream_ptr

pytestmark = pytest.mark.gpu
DEV = "cuda"
LENS = [0, 1, 128, 129, 300, 64, 256, 257]


def _inputs(K, H, lens, with_s0):
    g = torch.Generator(device=DEV).manual_seed(K * 7 + H)
    T = sum(lens)
    mk = lambda: (torch.randn(1, H, T, 64, 2, device=DEV, generator=g) * 0.1).bfloat16()
    q, k, v = mk(), mk(), mk()
    gamma = torch.sigmoid(torch.randn(K, 1, H, T, device=DEV, generator=g) + 2)
    coef = torch.randn(K, 1, H, T, 2, device=DEV, generator=g) if K > 1 else None
    cu = torch.tensor([0] + lens, device=DEV).cumsum(0).int()
    s0 = torch.randn(K, len(lens), H, 64, 64, 2, device=DEV, generator=g) if with_s0 else None
    return q, k, v, gamma, coef, cu, s0


@pytest.mark.parametrize("with_s0", [False, True])
@pytest.mark.parametrize("K,H,copies", [(1, 2, 1), (3, 2, 1), (3, 12, 5), (1, 16, 10)])      # the last two: a wave of carries and more
def test_forward_only_states(K, H, copies, with_s0):
    lens = LENS * copies
    q, k, v, gamma, coef, cu, s0 = _inputs(K, H, lens, with_s0)
    y_ref, s_ref = ops.pam_scan(q, k, v, gamma.clone().requires_grad_(True), coef=coef, cu_seqlens=cu, s0=s0, token_major=True)
    y, s = ops.pam_scan_tokens(q, k, v, gamma, coef=coef, cu_seqlens=cu, s0=s0)
    assert torch.equal(y, y_ref) and torch.equal(s, s_ref)
    for dtype in (torch.float32, torch.bfloat16):
        n = len(lens)
        slots = torch.randperm(n + 2, device=DEV)[:n].int()
        slots[3] = -1
        slots[4] = n + 2
        pool = torch.full((n + 2, 2, K, H, 64, 64, 2), 7.0, device=DEV, dtype=dtype)
        want = pool.clone()
        ops.pam_pool_store(want, slots, s_ref, layer=1)
        a = _lib.ScanArgs()
        y2 = torch.empty_like(y)
        a.q, a.k, a.v, a.gamma, a.coef, a.s0, a.cu_seqlens, a.y = (ptr(t) for t in (q, k, v, gamma, coef, s0, cu, y2))
        a.B, a.H, a.T, a.d, a.K, a.S, a.chunk, a.io_dtype, a.q_scale, a.gamma_eps = 1, H, q.shape[2], 64, K, n, 64, 1, 0.125, 1e-6
        ws = torch.empty(_lib.lib().qpam_scan_workspace_bytes(C.byref(a), 0), dtype=torch.uint8, device=DEV)
        a.workspace, a.workspace_bytes = ws.data_ptr(), ws.numel()
        check(_lib.lib().qpam_scan_prefill(C.byref(a), pool.data_ptr(), dtype_code(dtype), n + 2, 2, 1, ptr(slots), stream_ptr()), "qpam_scan_prefill")
        assert torch.equal(y2, y) and torch.equal(pool, want)


@pytest.mark.parametrize("lens", [[0, 1, 128, 129] + [1000 + 37 * i for i in range(20)],          # wide: the chunk sums carry
                                  [20000, 0] + [255 + i for i in range(22)]])                    # one long chain: they do not
def test_carry_in_the_chunk_sums(lens):
    H = 16
    q, k, v, gamma, _, cu, _ = _inputs(1, H, lens, False)
    assert len(lens) * H >= 384 and sum(lens) >= 1024 * len(lens)      # the batches the carrying form is chosen for
    y_ref, s_ref = ops.pam_scan(q, k, v, gamma.clone().requires_grad_(True), cu_seqlens=cu, token_major=True)
    for _ in range(3):
        y, s = ops.pam_scan_tokens(q, k, v, gamma, cu_seqlens=cu)
        assert torch.equal(s, s_ref) and torch.equal(y, y_ref)
