"""The split-contraction GEMM (few rows: generation, short prompts, small batches) at the edges of its tiles, clusters
and contraction shares, against the 64-bit product."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _operands(M, N, K, a_mn, b_mn):
    g = torch.Generator(device="cuda").manual_seed(M * 7919 + N * 31 + K)
    # 16-byte rows in either layout
    a = torch.randn((K, M) if a_mn else (M, K), generator=g, device="cuda").to(torch.bfloat16)
    b = torch.randn((K, N) if b_mn else (N, K), generator=g, device="cuda").to(torch.bfloat16)
    return a, b, (a.t() if a_mn else a).double() @ (b if b_mn else b.t()).double()


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
@pytest.mark.parametrize("M,N,K", [(8, 8, 64), (8, 4096, 4096), (128, 136, 1032), (136, 2048, 520), (256, 1000, 4104),
                                   (776, 2048, 2048), (24, 28672, 512)])
def test_products_of_few_rows(M, N, K, a_mn, b_mn):
    from lm_engine_b200.ops import _lib, gemm

    a, b, ref = _operands(M, N, K, a_mn, b_mn)
    out = gemm(a, b, a_mn=a_mn, b_mn=b_mn, out_dtype=torch.float32)
    # fp32 accumulation in any order: K roundings of 2^-24 relative to the sum of magnitudes, about 2e-6 in the norm
    assert float((out.double() - ref).norm() / ref.norm()) < 1e-5
    assert torch.equal(out, gemm(a, b, a_mn=a_mn, b_mn=b_mn, out_dtype=torch.float32))     # fixed order of the shares
    assert _lib.read_status()[0] == 0


@pytest.mark.parametrize("M", [1, 3, 129])
def test_epilogues_of_few_rows(M):
    from lm_engine_b200.ops import gemm, gemm_reference

    a, b, ref = _operands(M, 272, 2048, False, False)
    g = torch.Generator(device="cuda").manual_seed(1)
    bias, res = (torch.randn(s, generator=g, device="cuda").to(torch.bfloat16) for s in ((272,), (M, 272)))
    got = gemm(a, b, bias=bias, residual=res)
    assert float((got.double() - (ref + bias.double() + res.double())).norm() / ref.norm()) < 2.0 ** -8
    acc = torch.ones(M, 272, device="cuda")
    gemm(a, b, out=acc, accumulate=True)
    assert float((acc.double() - 1 - ref).norm() / ref.norm()) < 1e-5
    pre = torch.empty(M, 272, device="cuda", dtype=torch.bfloat16)
    y = gemm(a, b, swiglu=True, preact=pre)
    want = gemm_reference(a.float(), b.float(), swiglu=True)
    assert float((y.double() - want.double()).norm() / want.double().norm()) < 2.0 ** -7
    assert float((pre.double() - ref).norm() / ref.norm()) < 2.0 ** -8
