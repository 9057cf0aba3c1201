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


def test_saved_tensors_that_come_back_with_other_strides():
    from lm_engine_b200.ops import silu_mul
    from lm_engine_b200.ops.conv1d import causal_conv1d
    from lm_engine_b200.ops.recurrence import gated_delta_rule
    from lm_engine_b200.ops.ssd import ssd_chunk_scan

    g = torch.Generator(device="cuda").manual_seed(0)

    def r(*s):
        return torch.randn(*s, generator=g, device="cuda").to(BF).requires_grad_(True)

    wide, w, y = r(2, 70, 1024), r(512, 4), r(2, 70, 512)
    f = (-0.1 * torch.rand(2, 70, 2, generator=g, device="cuda")).requires_grad_(True)

    def heads(a, b, n):
        return wide[..., a:b].unflatten(-1, (n, -1))

    one = torch.ones(4, device="cuda")
    cases = {
        "gate": (lambda: silu_mul(y, wide[..., 512:]), (y, wide)),
        "convolution": (lambda: causal_conv1d(wide[..., 512:], w, None, None, "silu"), (wide, w)),
        "delta rule": (lambda: gated_delta_rule(heads(0, 256, 2), heads(256, 512, 2), heads(512, 640, 2), f, -f)[0],
                       (wide, f)),
        "scan": (lambda: ssd_chunk_scan(heads(0, 128, 4), -f.repeat(1, 1, 2), -one, heads(128, 144, 1),
                                        heads(144, 160, 1), one, 32)[0], (wide, f)),
    }
    moved = []

    def pack(t):            # slices come back as rows of another pitch
        if t.dim() < 3 or t.is_leaf or t.is_contiguous():
            return t, False
        moved.append(t.shape)
        return torch.nn.functional.pad(t, (0, 3)), True

    for name, (run, wrt) in cases.items():
        out = run()
        dout = torch.randn(out.shape, generator=g, device="cuda").to(out.dtype)
        want = torch.autograd.grad(out, wrt, dout)
        with torch.autograd.graph.save_on_cpu():
            dense = run()
        results = [torch.autograd.grad(dense, wrt, dout)]
        if name != "scan":      # (the scan takes whole chunks as dense copies here)
            moved.clear()
            with torch.autograd.graph.saved_tensors_hooks(pack, lambda p: p[0][..., :-3] if p[1] else p[0]):
                padded = run()
            assert moved, name
            results.append(torch.autograd.grad(padded, wrt, dout))
        for got in results:     # equal but for the convolution's weight gradient, which is added in any order
            for a, b in zip(got, want):
                assert float((a.double() - b.double()).norm() / b.double().norm()) < 2.0 ** -8, name
