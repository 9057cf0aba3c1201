"""The gated delta rule's block-local kernels (with the chain between them) against the tensor-operation form of the
same blocks in 64 bits, at ragged lengths, strided operands and every gradient."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _blocks64(q, k, v, g, beta, scale, h0, l2norm):
    """Token by token in 64 bits."""
    K = q.size(-1)
    if l2norm:
        q, k = (t / (t.norm(dim=-1, keepdim=True) + 1e-6) for t in (q, k))
    q = q * (K ** -0.5 if scale is None else scale)
    h, ys = h0, []
    for s in range(q.size(1)):
        h = h * torch.exp(g[:, s])[..., None, None]
        d = (v[:, s] - torch.einsum("bnkv,bnk->bnv", h, k[:, s])) * beta[:, s, :, None]
        h = h + k[:, s, :, :, None] * d[:, :, None, :]
        ys.append(torch.einsum("bnkv,bnk->bnv", h, q[:, s]))
    return torch.stack(ys, dim=1), h


@pytest.mark.parametrize("B,S,N,K,V,scale,l2norm", [(1, 8, 1, 128, 64, None, True), (2, 64, 2, 256, 128, None, True),
                                                    (1, 129, 3, 256, 192, 0.1, True), (2, 100, 1, 128, 512, None, False)])
def test_block_kernels_match_the_token_recurrence(B, S, N, K, V, scale, l2norm):
    from lm_engine_b200.ops import _lib
    from lm_engine_b200.ops.recurrence import gated_delta_blocks_usable, gated_delta_rule

    gen = torch.Generator(device="cuda").manual_seed(S)

    def r(*s):
        return torch.randn(*s, generator=gen, device="cuda")

    # slices of one projection row, as the layer makes them
    row = r(B, S, N * (2 * K + V)).to(torch.bfloat16)
    if not l2norm:
        row[..., :2 * N * K] *= K ** -0.5
    q, k, v = (t.reshape(B, S, N, -1) for t in row.split((N * K, N * K, N * V), dim=-1))
    g, beta = -0.3 * torch.rand(B, S, N, generator=gen, device="cuda"), 2 * torch.rand(B, S, N, generator=gen, device="cuda")
    ins = [t.detach().requires_grad_(True) for t in (q, k, v, g, beta, 0.3 * r(B, N, K, V))]
    assert gated_delta_blocks_usable(*ins[:5])
    y, h = gated_delta_rule(*ins[:5], scale, ins[5], l2norm)
    dy, dh = r(*y.shape).to(torch.bfloat16), r(*h.shape)
    got = torch.autograd.grad((y, h), ins, (dy, dh))
    ref_in = [t.detach().double().requires_grad_(True) for t in ins]
    y64, h64 = _blocks64(*ref_in[:5], scale, ref_in[5], l2norm)
    ref = torch.autograd.grad((y64, h64), ref_in, (dy.double(), dh.double()))
    assert _lib.read_status()[0] == 0
    # the chain multiplies bf16 roundings of its operands and state (2^-9 each, a handful of them along a path); the
    # bound is the one of the chain's own tests
    for name, a, b in zip(("y", "h", "dq", "dk", "dv", "dg", "dbeta", "dh0"), (y, h, *got), (y64, h64, *ref)):
        assert float((a.double() - b).norm() / (b.norm() + 1e-12)) < 2e-2, name
