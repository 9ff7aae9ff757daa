"""Parameters that a fused operator has to convert (bf16, or a strided view): each backward pass reads its own copies."""
import pytest
import torch

from qllm2_b200 import fused_elementwise as FE

pytestmark = pytest.mark.gpu
DEV = "cuda"
OPS = {"swish": (FE.fused_mod_swish, 2), "relu": (FE.fused_mod_relu, 1), "norm": (FE.fused_complex_norm, 1)}


@pytest.mark.parametrize("form", ["bf16", "strided"])
@pytest.mark.parametrize("name", OPS)
def test_converted_parameters_give_the_same_gradients(name, form):
    fn, n = OPS[name]
    C = 24
    g = torch.Generator().manual_seed(2)
    z = torch.randn(3, 11, C, 2, generator=g).to(DEV)
    dy = torch.randn(3, 11, C, 2, generator=g).to(DEV)
    vals = [(torch.randn(C, generator=g) + i).bfloat16().to(DEV) for i in range(n)]
    res = []
    for convert in (False, True):
        zi = z.clone().requires_grad_()
        ps = [v.float() for v in vals]
        if convert:
            ps = [v.clone() if form == "bf16" else v.float().repeat_interleave(2)[::2] for v in vals]
        ps = [p.detach().requires_grad_() for p in ps]
        y = fn(zi, *ps)
        res.append([y, *torch.autograd.grad(y, [zi, *ps], dy)])
    for a, b in zip(*res):
        assert torch.equal(a.to(b.dtype), b)
