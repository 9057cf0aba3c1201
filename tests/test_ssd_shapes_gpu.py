"""One decay, skip weight or initial state for all heads or sequences in the SSD scan's kernels."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_shared_decay_skip_and_state():
    from lm_engine_b200.ops.ssd import ssd_chunk_scan

    b, S, N, P, G, Sd = 2, 70, 4, 32, 2, 16
    g = torch.Generator(device="cuda").manual_seed(0)

    def r(*s):
        return torch.randn(*s, generator=g, device="cuda")

    x, B, C = (r(*s).to(torch.bfloat16) for s in ((b, S, N, P), (b, S, G, Sd), (b, S, G, Sd)))
    dt = torch.rand(b, S, N, generator=g, device="cuda")
    shared = [(-r(1).abs()).requires_grad_(True), r(1).requires_grad_(True), r(1, N, P, Sd).requires_grad_(True)]
    full = [t.detach().expand(s).clone().requires_grad_(True) for t, s in zip(shared, ((N,), (N,), (b, N, P, Sd)))]
    dy, dh, outs = r(b, S, N, P).to(torch.bfloat16), r(b, N, P, Sd), []
    for A, D, h0 in (shared, full):
        y, h = ssd_chunk_scan(x, dt, A, B, C, D, 32, initial_state=h0)
        outs.append((y, h, *torch.autograd.grad((y, h), (A, D, h0), (dy, dh))))
    a, f = outs
    assert torch.equal(a[0], f[0]) and torch.equal(a[1], f[1])
    # the same fp32 gradients, added over heads or sequences in any order
    for got, want, dim in zip(a[2:], f[2:], (0, 0, 0)):
        torch.testing.assert_close(got, want.sum(dim, keepdim=True), rtol=1e-5, atol=1e-4 * float(want.abs().max()))


def test_a_step_width_that_does_not_fit_raises():
    from lm_engine_b200.ops.ssd import ssd_chunk_scan

    x, B = torch.zeros(1, 32, 4, 32, device="cuda", dtype=torch.bfloat16), torch.zeros(1, 32, 1, 16, device="cuda")
    with pytest.raises(RuntimeError):
        ssd_chunk_scan(x, torch.zeros(1, 32, 1, device="cuda"), -torch.ones(4, device="cuda"), B, B,
                       torch.ones(4, device="cuda"), 32)


def test_more_sequences_times_heads_than_a_grid_dimension_holds():
    from lm_engine_b200.ops import _lib
    from lm_engine_b200.ops.ssd import ssd_chunk_scan

    b, S, N, P, Sd = 2064, 40, 32, 32, 8
    g = torch.Generator(device="cuda").manual_seed(1)
    x, B, C = (torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)
               for s in ((b, S, N, P), (b, S, 1, Sd), (b, S, 1, Sd)))
    dt, A, D = torch.rand(b, S, N, generator=g, device="cuda"), -torch.rand(N, generator=g, device="cuda"), torch.ones(N, device="cuda")

    def run(s):
        ins = [t[s].detach().requires_grad_(True) for t in (x, dt, B, C)]
        before = _lib.launch_count
        y, h = ssd_chunk_scan(ins[0], ins[1], A, ins[2], ins[3], D, 32)
        grads = torch.autograd.grad((y.float().square().sum() + h.square().sum()), ins)
        return _lib.launch_count - before, [y.detach(), h.detach(), *grads]

    launches, whole = run(slice(0, b))
    halves = [run(slice(0, b // 2)), run(slice(b // 2, b))]
    assert launches == halves[0][0]                       # the same kernels
    for i, t in enumerate(whole):
        assert torch.equal(t, torch.cat([h[1][i] for h in halves]))


@pytest.mark.parametrize("Sd", [1, 12, 20])
def test_states_that_are_no_multiple_of_eight(Sd):
    from lm_engine_b200.ops import _lib
    from lm_engine_b200.ops.ssd import ssd_chunk_scan

    b, S, N, P, G = 2, 70, 4, 32, 2
    g = torch.Generator(device="cuda").manual_seed(Sd)
    x, B, C = (torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)
               for s in ((b, S, N, P), (b, S, G, Sd), (b, S, G, Sd)))
    dt, A, D = torch.rand(b, S, N, generator=g, device="cuda") * 0.3, -torch.rand(N, generator=g, device="cuda"), torch.ones(N, device="cuda")
    ins = [t.requires_grad_(True) for t in (x, dt, B, C, torch.randn(b, N, P, Sd, generator=g, device="cuda"))]
    before = _lib.launch_count
    y, h = ssd_chunk_scan(ins[0], ins[1], A, ins[2], ins[3], D, 32, initial_state=ins[4])
    assert _lib.launch_count > before
    dy, dh = torch.randn(y.shape, generator=g, device="cuda").to(torch.bfloat16), torch.randn(h.shape, generator=g, device="cuda")
    got = torch.autograd.grad((y, h), ins, (dy, dh))
    ref_in = [t.detach().double().requires_grad_(True) for t in ins]
    x, dt64, Bh, Ch = ref_in[0], ref_in[1], *(t.repeat_interleave(N // G, dim=2) for t in ref_in[2:4])
    state, ys = ref_in[4], []
    for t in range(S):
        state = state * torch.exp(dt64[:, t] * A.double())[..., None, None] + (
            (dt64[:, t, :, None] * x[:, t])[..., None] * Bh[:, t, :, None])
        ys.append((state * Ch[:, t, :, None]).sum(-1) + x[:, t])
    y64 = torch.stack(ys, dim=1)
    ref = torch.autograd.grad((y64, state), ref_in, (dy.double(), dh.double()))
    # products of bf16 roundings, a few 2^-9 along a path; dt collects sums that cancel over a chunk
    for name, a, e in zip(("y", "h", "dx", "ddt", "dB", "dC", "dh0"), (y, h, *got), (y64, state, *ref)):
        assert float((a.detach().double() - e.detach()).norm() / e.norm()) < (4e-2 if name == "ddt" else 2e-2), name
