"""The SSD scan's kernels on operands that are slices of one projection row, at lengths that do not fill a chunk, for one
and several groups; outputs, final state and every gradient against the token recurrence in 64 bits."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,S,N,P,G,Sd,L,offset", [(1, 32, 2, 32, 1, 8, 32, 0), (2, 70, 9, 64, 1, 16, 32, 8),
                                                   (2, 130, 8, 128, 2, 24, 64, 0), (1, 97, 33, 32, 3, 16, 96, 3)])
def test_scan_of_slices_matches_the_token_recurrence(b, S, N, P, G, Sd, L, offset):
    from lm_engine_b200.ops import _lib
    from lm_engine_b200.ops.ssd import ssd_chunk_scan

    g = torch.Generator(device="cuda").manual_seed(S)

    def r(*s):
        return torch.randn(*s, generator=g, device="cuda")

    wide = r(b, S, offset + N * P + 2 * G * Sd).to(torch.bfloat16).requires_grad_(True)
    dt = (torch.rand(b, S, N, generator=g, device="cuda") * 0.3 + 0.01).requires_grad_(True)
    A, D = (-torch.rand(N, generator=g, device="cuda") - 0.1).requires_grad_(True), r(N).requires_grad_(True)
    h0 = r(b, N, P, Sd).requires_grad_(True)

    def operands(w):
        x, B, C = w[..., offset:].split((N * P, G * Sd, G * Sd), dim=-1)
        return x.reshape(b, S, N, P), 0.5 * B.reshape(b, S, G, Sd), C.reshape(b, S, G, Sd)

    x, B, C = operands(wide)
    y, h = ssd_chunk_scan(x, dt, A, B, C, D, L, initial_state=h0)
    dy, dh = r(*y.shape).to(torch.bfloat16), r(*h.shape)
    ins = (wide, dt, A, D, h0)
    got = torch.autograd.grad((y, h), ins, (dy, dh))
    ref_in = [t.detach().double().requires_grad_(True) for t in ins]
    x, B, C = operands(ref_in[0])
    B, C = (t.repeat_interleave(N // G, dim=2) for t in (B, C))
    state, ys = ref_in[4], []
    for t in range(S):
        state = state * torch.exp(ref_in[1][:, t] * ref_in[2])[..., None, None] + (
            (ref_in[1][:, t, :, None] * x[:, t])[..., None] * B[:, t, :, None])
        ys.append((state * C[:, t, :, None]).sum(-1) + ref_in[3][:, None] * x[:, t])
    ref_y = torch.stack(ys, dim=1)
    ref = torch.autograd.grad((ref_y, state), ref_in, (dy.double(), dh.double()))
    assert _lib.read_status()[0] == 0
    # products of bf16 roundings (decay matrix, weighted inputs, carried states): a few 2^-9 along a path; dt and A
    # collect sums that cancel over a chunk
    for name, a, e in zip(("y", "h", "dwide", "ddt", "dA", "dD", "dh0"), (y, h, *got), (ref_y, state, *ref)):
        assert float((a.double() - e).norm() / e.norm()) < (4e-2 if name in ("ddt", "dA") else 2e-2), name
