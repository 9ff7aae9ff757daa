"""Tensors that start off a 16-byte boundary (views into a flat buffer): the fused operators copy what their vector accesses
need aligned, forward and backward, and give the same results."""
import pytest
import torch

from qllm2_b200 import fused_elementwise as FE

DEV = "cuda"


def _off(t):
    """The same values, one element behind an aligned address."""
    buf = torch.empty(t.numel() + 8, dtype=t.dtype, device=t.device)
    v = buf[1:1 + t.numel()].view(t.shape)
    v.copy_(t)
    return v


def test_dense_gives_an_aligned_start():
    for dtype in (torch.float32, torch.bfloat16):
        t = torch.arange(24).to(dtype).view(2, 3, 4)
        assert FE._dense(t).data_ptr() == t.data_ptr()
        for u in (_off(t), t.transpose(0, 2), _off(t).transpose(0, 1)):
            d = FE._dense(u)
            assert d.is_contiguous() and d.data_ptr() % 16 == 0 and torch.equal(d, u)
        rows, _, _, _ = FE._rows(_off(torch.randn(3, 4, 2).to(dtype)))
        assert rows.data_ptr() % 16 == 0


OPS = {
    "norm": (lambda z, s: FE.fused_complex_norm(z, s), [(2, 9, 12, 2), (12,)]),
    "swish": (lambda z, b, be: FE.fused_mod_swish(z, b, be), [(2, 9, 12, 2), (12,), (12,)]),
    "gate": (lambda a, b: FE.fused_cgu_gate(a, b), [(2, 9, 12, 2), (2, 9, 12, 2)]),
    "residual": (lambda x, d, s: FE.scaled_residual(x, d, s), [(2, 9, 12, 2), (2, 9, 12, 2), ()]),
    "magnitude": (lambda z: FE.complex_magnitude(z), [(2, 9, 12, 2)]),
    "prep": (lambda qkv, omp: torch.stack(FE.pam_prep(qkv, _off(ROPE.to(DEV)), omp, n_heads=2, head_dim=4)), [(2, 9, 24, 2), (2, 9, 2)]),
}
ROPE = torch.randn(9, 4, 2, generator=torch.Generator().manual_seed(1))


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("name", OPS)
def test_operators_on_unaligned_tensors(name, dtype):
    fn, shapes = OPS[name]
    g = torch.Generator().manual_seed(4)
    data = [torch.randn(s, generator=g).to(DEV) for s in shapes]
    data = [t.to(dtype) if t.dim() == 4 else t for t in data]
    res = []
    for place in (torch.clone, _off):
        leaves = [place(t).requires_grad_() for t in data]
        y = fn(*leaves)
        dy = torch.ones_like(y) * 0.5
        res.append([y, *torch.autograd.grad(y, leaves, place(dy))])
    for a, b in zip(*res):
        assert torch.equal(a, b)
