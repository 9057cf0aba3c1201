"""Four-tap causal convolution kernels: time runs and channel groups that do not fill a block, a slice of a wider row
read in place, the initial state and its gradient; against 64-bit autograd."""

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,S,C,extra,state,silu", [(1, 1, 8, 0, True, True), (2, 2, 16, 8, True, False),
                                                    (1, 16, 136, 0, False, True), (3, 131, 264, 24, True, True),
                                                    (2, 257, 1032, 64, False, False), (1, 1000, 4352, 4096, False, True)])
def test_four_taps(B, S, C, extra, state, silu):
    from lm_engine_b200.ops.conv1d import causal_conv1d

    g = torch.Generator(device="cuda").manual_seed(S + C)

    def r(*s):
        return torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)

    wide, w, bias, dy = r(B, S, C + extra).requires_grad_(True), r(C, 4).requires_grad_(True), r(C).requires_grad_(True), r(B, S, C)
    init = r(B, C, 3).requires_grad_(True) if state else None
    ins = [wide, w, bias] + ([init] if state else [])
    y = causal_conv1d(wide[..., extra:], w, bias, init, "silu" if silu else None)
    got = torch.autograd.grad(y, ins, dy)
    r64 = [t.detach().double().requires_grad_(True) for t in ins]
    x64 = r64[0][..., extra:].transpose(1, 2)
    x64 = torch.cat((r64[3], x64), dim=-1) if state else F.pad(x64, (3, 0))
    z = F.conv1d(x64, r64[1].unsqueeze(1), r64[2], groups=C).transpose(1, 2)
    z = F.silu(z) if silu else z
    ref = torch.autograd.grad(z, r64, dy.double())
    # fp32 arithmetic, one rounding of each result to bf16
    for a, b in zip((y, *got), (z, *ref)):
        assert float((a.double() - b).norm() / (b.norm() + 1e-12)) < 2.0 ** -8
