"""RMSNorm kernels at the edges of their row layouts (one warp or one CTA per row, one to four vectors per thread, ring
shorter and longer than the rows) against 64-bit autograd."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("with_res", [False, True])
@pytest.mark.parametrize("T,H", [(1, 8), (3, 128), (3600, 256), (4001, 512), (445, 520), (1790, 1024), (1776, 2048), (1777, 2048), (1800, 8200), (2, 1032),
                                 (900, 2056), (1335, 4096), (333, 6144), (31, 8200), (450, 16384)])
def test_rmsnorm_layouts(T, H, with_res):
    from lm_engine_b200.ops import _lib, rmsnorm

    g = torch.Generator(device="cuda").manual_seed(T + H)

    def r(*s):
        return torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)

    x, res, dy, dh = r(T, H), r(T, H), r(T, H), r(T, H)
    w = (1 + 0.1 * r(H).float()).to(torch.bfloat16).requires_grad_(True)
    xs = [x.clone().requires_grad_(True)] + ([res.clone().requires_grad_(True)] if with_res else [])
    y, h = rmsnorm(xs[0], w, 1e-5, xs[1] if with_res else None)
    got = torch.autograd.grad((y, h) if with_res else (y,), (*xs, w), (dy, dh) if with_res else (dy,))
    h64 = (x + res if with_res else x).double().requires_grad_(True)      # the sum is rounded to bf16: an output
    w64 = w.detach().double().requires_grad_(True)
    y64 = h64 * torch.rsqrt(h64.square().mean(-1, keepdim=True) + 1e-5) * w64
    ref = torch.autograd.grad((y64, h64) if with_res else (y64,), (h64, w64),
                              (dy.double(), dh.double()) if with_res else (dy.double(),))

    def rel(a, b):
        return float((a.double() - b).norm() / b.norm())

    # one rounding to bf16 (2^-9 per element) of fp32 results
    assert rel(y, y64.detach()) < 2.0 ** -8 and rel(got[0], ref[0]) < 2.0 ** -8 and rel(got[-1], ref[1]) < 2.0 ** -8
    if with_res:
        assert torch.equal(h, x + res) and torch.equal(got[0], got[1])
    assert _lib.read_status()[0] == 0
