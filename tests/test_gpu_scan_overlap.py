"""The kernels of a scan overlap (programmatic dependent launch): a call whose inputs are still being written when it is issued,
between other calls, gives the bits of the same call on a device that is idle before and after it."""
import pytest
import torch

from qllm2_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,T,d,K,dtype", [
    (1, 6, 93, 64, 1, torch.bfloat16),       # one chunk: the chunk kernel begins the backward
    (2, 3, 128, 64, 3, torch.bfloat16),
    (4, 6, 129, 64, 1, torch.bfloat16),      # a second chunk of one token
    (8, 6, 1100, 64, 1, torch.bfloat16),     # more chunk jobs than fit the device at once
    (4, 6, 1100, 64, 3, torch.bfloat16),
    (2, 4, 50, 32, 1, torch.float32),
    (2, 4, 300, 32, 2, torch.float32),
])
def test_overlapped_calls_have_the_bits_of_separate_ones(B, H, T, d, K, dtype):
    g = torch.Generator(device="cuda").manual_seed(T)
    base = [(torch.randn(B, H, T, d, 2, device="cuda", generator=g) * (2 * d) ** -0.5).to(dtype) for _ in range(4)]
    gamma = torch.sigmoid(torch.randn(K, B, H, T, device="cuda", generator=g) + 2.0)
    coef = torch.randn(K, B, H, T, 2, device="cuda", generator=g) if K > 1 else None

    def call(i, wait):
        q, k, v, dy = ((t * (1.0 + i)).requires_grad_(True) for t in base)      # written right before the call
        gm = gamma.clone().requires_grad_(True)
        cf = None if coef is None else (coef * (1.0 + i)).requires_grad_(True)
        if wait:
            torch.cuda.synchronize()
        y, last = ops.pam_scan(q, k, v, gm, coef=cf)
        if wait:
            torch.cuda.synchronize()
        out = [y, last, *torch.autograd.grad(y, [q, k, v, gm] + ([] if cf is None else [cf]), dy.detach())]
        if wait:
            torch.cuda.synchronize()
        return out

    want = [call(i, True) for i in range(4)]
    got = [call(i, False) for i in range(4)]
    for a, b in zip(want, got):
        assert all(torch.equal(x, y) for x, y in zip(a, b))
