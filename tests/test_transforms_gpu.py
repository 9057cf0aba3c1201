"""Tracing, transforms and forward-mode derivatives of operators whose kernels take tensors by address: they see the
PyTorch operations."""

import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _gate():
    from lm_engine_b200.ops import silu_mul

    return silu_mul, [torch.randn(4, 64, device="cuda").to(BF) for _ in range(2)]


def _one_token():
    from lm_engine_b200.ops import attention

    q, k, v = (torch.randn(2, n, 4, 64, device="cuda").to(BF) for n in (1, 33, 33))
    return (lambda q, k, v: attention(q, k, v, causal=True)), [q, k, v]


# (the attention statement itself cannot be traced by torch.jit on a GPU: its head repetition gets an index on the CPU)
@pytest.mark.parametrize("make,trace", [(_gate, "make_fx"), (_gate, "make_fx fake"), (_gate, "jit"),
                                        (_one_token, "make_fx"), (_one_token, "make_fx fake")])
def test_traces_hold_for_other_inputs(make, trace):
    from torch.fx.experimental.proxy_tensor import make_fx

    f, ins = make()
    with torch.no_grad():
        if trace == "jit":
            g = torch.jit.trace(f, ins, check_trace=False)
        else:
            g = make_fx(f, tracing_mode="fake" if trace.endswith("fake") else "real")(*ins)
        others = [torch.randn_like(t) for t in ins]
        got, want = g(*others).float(), f(*others).float()
    # the same fp32 arithmetic, rounded to bf16 once or twice in both
    assert float((got - want).norm() / want.norm()) < 2.0 ** -7


def test_transforms_of_the_gate():
    f, (y, gate) = _gate()
    dy, dg = torch.randn_like(y), torch.randn_like(gate)
    _, tangent = torch.func.jvp(f, (y, gate), (dy, dg))
    y64, g64, dy64, dg64 = (t.double() for t in (y, gate, dy, dg))
    s = torch.sigmoid(g64)
    want = dy64 * g64 * s + y64 * dg64 * s * (1 + g64 * (1 - s))
    assert float((tangent.double() - want).norm() / want.norm()) < 2.0 ** -6       # a few roundings of 2^-9
    assert torch.equal(torch.func.vmap(f)(y, gate), f(y, gate)) or torch.allclose(
        torch.func.vmap(f)(y, gate).float(), f(y, gate).float(), rtol=2.0 ** -7)
    y, gate = y.requires_grad_(True), gate.requires_grad_(True)
    out = f(y, gate)
    first = torch.autograd.grad(out, (y, gate), dy, create_graph=True)
    second = torch.autograd.grad(first, (y, gate), (dg, dg))
    ins = [t.detach().double().requires_grad_(True) for t in (y, gate)]
    f64 = torch.autograd.grad(ins[0] * torch.nn.functional.silu(ins[1]), ins, dy64, create_graph=True)
    for a, b in zip(second, torch.autograd.grad(f64, ins, (dg64, dg64))):
        assert float((a.double() - b).norm() / b.norm()) < 2.0 ** -6
