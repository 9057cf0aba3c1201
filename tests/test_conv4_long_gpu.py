"""Four-tap convolution of a sequence with more runs of 16 steps than a grid dimension holds."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_a_million_steps():
    from lm_engine_b200.ops.conv1d import causal_conv1d, causal_conv1d_reference

    S = 16 * 65535 + 21
    g = torch.Generator(device="cuda").manual_seed(0)
    x, w, dy = (torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16) for s in ((1, S, 8), (8, 4), (1, S, 8)))
    x, w = x.requires_grad_(True), w.requires_grad_(True)
    y = causal_conv1d(x, w, None, None, "silu")
    ref_in = [t.detach().double().requires_grad_(True) for t in (x, w)]
    ref = causal_conv1d_reference(*ref_in, None, None, "silu")
    got, want = torch.autograd.grad(y, (x, w), dy), torch.autograd.grad(ref, ref_in, dy.double())
    # one rounding of each result to bf16; the weight gradient adds a million fp32 terms first (sqrt(S) 2^-24 = 6e-5)
    for a, b in zip((y.detach(), *got), (ref.detach(), *want)):
        assert float((a.double() - b).norm() / b.norm()) < 2.0 ** -8
