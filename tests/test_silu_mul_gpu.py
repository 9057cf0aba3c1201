"""Output gate of the recurrent mixers: y * silu(gate) with the gate read in place from a wider row."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,extra", [((1, 8), 0), ((3, 5, 264), 16), ((2, 33, 4096), 8), ((7, 2056), 3)])
def test_silu_mul(shape, extra):
    from lm_engine_b200.ops import silu_mul

    g = torch.Generator(device="cuda").manual_seed(shape[-1])
    y = torch.randn(shape, generator=g, device="cuda").to(torch.bfloat16).requires_grad_(True)
    wide = (4 * torch.randn(*shape[:-1], shape[-1] + extra, generator=g, device="cuda")).to(torch.bfloat16).requires_grad_(True)
    dout = torch.randn(shape, generator=g, device="cuda").to(torch.bfloat16)
    out = silu_mul(y, wide[..., extra:])
    got = torch.autograd.grad(out, (y, wide), dout)
    y64, w64 = (t.detach().double().requires_grad_(True) for t in (y, wide))
    want = y64 * torch.nn.functional.silu(w64[..., extra:])
    ref = torch.autograd.grad(want, (y64, w64), dout.double())
    # two roundings to bf16 (of the activation or its gradient, and of the result), each at most 2^-8 of a value
    for a, b in zip((out, *got), (want, *ref)):
        assert float((a.double() - b).norm() / b.norm()) < 2.0 ** -7
