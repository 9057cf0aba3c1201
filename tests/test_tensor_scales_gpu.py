"""Scales given as tensors keep the operations that differentiate them."""

import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def test_delta_rule_scale():
    from lm_engine_b200.ops.recurrence import gated_delta_rule

    q, k, v = (torch.randn(1, 70, 2, n, device="cuda").to(BF) for n in (128, 128, 64))
    g, beta = -0.1 * torch.rand(1, 70, 2, device="cuda"), torch.rand(1, 70, 2, device="cuda")
    scale = torch.tensor(0.2, device="cuda", requires_grad=True)
    y, _ = gated_delta_rule(q, k, v, g, beta, scale)
    dy = torch.randn_like(y)
    grad, = torch.autograd.grad(y, scale, dy)
    # y is linear in the scale; the chain multiplies bf16 roundings
    terms = y.detach().double() * dy.double() / 0.2
    assert float((grad.double() - terms.sum()).abs()) < 2e-2 * float(terms.norm())
    plain, _ = gated_delta_rule(q, k, v, g, beta, 0.2)
    assert float((y.detach().float() - plain.float()).norm() / plain.float().norm()) < 2e-2


@pytest.mark.parametrize("kind", ["tensor", "numpy"])
def test_one_token_attention_scale(kind):
    import numpy as np

    from lm_engine_b200.ops import attention

    q, k, v = (torch.randn(2, n, 4, 64, device="cuda").to(BF) for n in (1, 33, 33))
    want = attention(q, k, v, softmax_scale=0.25)
    if kind == "numpy":
        assert torch.equal(attention(q, k, v, softmax_scale=np.float32(0.25)), want)
        return
    scale = torch.tensor(0.25, device="cuda", requires_grad=True)
    out = attention(q, k, v, softmax_scale=scale)
    assert float((out.detach().float() - want.float()).norm() / want.float().norm()) < 2.0 ** -8
    assert torch.autograd.grad(out.float().square().sum(), scale)[0].isfinite()
