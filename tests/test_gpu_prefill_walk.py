"""Forward-only scans that walk over a sequence's chunks, at the edges of their dispatch: lengths around a chunk, a sequence that is
split, empty ones, more sequences than a tile of the list's kernel, equal lengths -- for every number of states, against the training
forward (chunk sums, carry, outputs as separate passes), whose bits they have."""
import pytest
import torch

from qllm2_b200 import _lib, ops

pytestmark = pytest.mark.gpu
DEV = "cuda"
EDGES = [0, 1, 127, 128, 129, 255, 256, 257, 384, 511, 0, 64]


def _inputs(B, H, T, K, S, with_s0, strong, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    mk = lambda: (torch.randn(B, H, T, 64, 2, device=DEV, generator=g) * 0.1).bfloat16()
    q, k, v = mk(), mk(), mk()
    gamma = torch.sigmoid(torch.randn(K, B, H, T, device=DEV, generator=g) + torch.linspace(-1.0 if strong else 1.5, 4.0, K, device=DEV).view(K, 1, 1, 1))
    coef = torch.randn(K, B, H, T, 2, device=DEV, generator=g) if K > 1 else None
    s0 = torch.randn(K, S, H, 64, 64, 2, device=DEV, generator=g) if with_s0 else None
    return q, k, v, gamma, coef, s0


@pytest.mark.parametrize("K", [1, 2, 3, 4])
@pytest.mark.parametrize("lens,H", [(EDGES * 2, 16),                              # walked
                                    (EDGES * 2 + [4000], 16),                     # the last one is split
                                    ([(7 * i) % 5 for i in range(1100)], 1)])     # tiny, and more of them than threads
@pytest.mark.parametrize("with_s0,strong", [(False, False), (True, True)])
def test_packed(K, lens, H, with_s0, strong):
    q, k, v, gamma, coef, s0 = _inputs(1, H, sum(lens), K, len(lens), with_s0, strong, K * 5 + H)
    cu = torch.tensor([0] + lens, device=DEV).cumsum(0).int()
    assert len(lens) * H >= 384
    y_ref, s_ref = ops.pam_scan(q, k, v, gamma.clone().requires_grad_(True), coef=coef, cu_seqlens=cu, s0=s0, token_major=True)
    for _ in range(2):
        y, s = ops.pam_scan_tokens(q, k, v, gamma, coef=coef, cu_seqlens=cu, s0=s0)
        assert torch.equal(s, s_ref) and torch.equal(y, y_ref)
    assert _lib.device_status() == 0


@pytest.mark.parametrize("K", [1, 3])
@pytest.mark.parametrize("B,H,T", [(48, 6, 100), (48, 6, 128), (98, 6, 300), (40, 6, 1025)])
def test_equal_lengths(K, B, H, T):
    q, k, v, gamma, coef, s0 = _inputs(B, H, T, K, B, T == 300, False, T + K)
    y_ref, s_ref = ops.pam_scan(q, k, v, gamma.clone().requires_grad_(True), coef=coef, s0=s0)
    with torch.no_grad():
        n0 = _lib.launch_count()
        y, s = ops.pam_scan(q, k, v, gamma, coef=coef, s0=s0)
        assert _lib.launch_count() - n0 == 1
    assert torch.equal(s, s_ref) and torch.equal(y, y_ref)
    assert _lib.device_status() == 0
