"""Attention of one new token per sequence over its cache: the kernel against the 64-bit statement at the edges of its
key blocks, splits and head groups, and what it does with rows and scores that are not ordinary."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs(B, Sk, Hq, Hkv, D, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)
            for s in ((B, 1, Hq, D), (B, Sk, Hkv, D), (B, Sk, Hkv, D))]


@pytest.mark.parametrize("B,Sk,Hq,Hkv,D,padded,window", [
    (1, 2, 4, 4, 64, False, None), (1, 15, 32, 8, 128, False, None), (2, 65, 20, 4, 128, True, None),
    (3, 1025, 16, 2, 128, True, None), (2, 129, 18, 2, 64, False, None), (1, 700, 32, 8, 128, False, 64),
    (2, 300, 8, 1, 64, True, 77), (40, 257, 16, 8, 128, False, None), (1, 5000, 32, 8, 128, False, None)])
def test_one_token_matches_the_statement(B, Sk, Hq, Hkv, D, padded, window):
    from lm_engine_b200.ops import _lib, attention, attention_reference

    q, k, v = _inputs(B, Sk, Hq, Hkv, D)
    mask = None
    if padded:
        mask = (torch.arange(Sk, device="cuda")[None] >= torch.randint(0, Sk, (B, 1), device="cuda")).long()
    before = _lib.launch_count
    out = attention(q, k, v, causal=True, attention_mask=mask, sliding_window=window)
    assert _lib.launch_count == before + 1
    ref = attention_reference(q.float(), k.float(), v.float(), causal=True, attention_mask=mask,
                              sliding_window=window)
    # the weights and sums are fp32: what is left is the rounding of the result, 2^-9 per element
    assert float((out.float() - ref).norm() / ref.norm()) < 2.0 ** -8.5


def test_strided_caches_and_hidden_rows():
    from lm_engine_b200.ops import attention, attention_reference

    q, k, v = _inputs(3, 90, 8, 2, 128)
    kv = torch.stack((k, v), dim=3)                       # [B, S, H, 2, D]: both caches are strided views
    mask = torch.ones(3, 90, dtype=torch.bool, device="cuda")
    mask[1] = False                                       # a sequence that attends to nothing
    out = attention(q, kv[:, :, :, 0], kv[:, :, :, 1], causal=True, attention_mask=mask)
    ref = attention_reference(q, k, v, causal=True, attention_mask=mask)
    assert bool((out[1] == 0).all()) and bool((ref[1] == 0).all())
    assert float((out.float() - ref.float()).norm() / ref.float().norm()) < 2.0 ** -8


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_scores_that_are_not_finite_give_the_statement_s_zero_rows(bad):
    from lm_engine_b200.ops import attention, attention_reference

    q, k, v = _inputs(1, 200, 8, 2, 64)
    q[..., 0] = 1.0
    k[0, 77, 0, 0] = bad                                  # reaches the four heads of the first group
    out, ref = attention(q, k, v, causal=True), attention_reference(q, k, v, causal=True)
    assert torch.equal(ref[0, 0, :4], torch.zeros_like(ref[0, 0, :4]))
    assert torch.equal(out[0, 0, :4], ref[0, 0, :4])
    assert float((out.float() - ref.float()).norm() / ref.float().norm()) < 2.0 ** -8


def test_gradients_keep_the_differentiable_path():
    from lm_engine_b200.ops import attention, attention_reference

    q, k, v = (t.requires_grad_(True) for t in _inputs(2, 40, 4, 4, 64))
    g = torch.autograd.grad(attention(q, k, v, causal=True).float().square().sum(), (q, k, v))
    r = torch.autograd.grad(attention_reference(q, k, v, causal=True).float().square().sum(), (q, k, v))
    assert all(torch.equal(a, b) for a, b in zip(g, r))


@pytest.mark.parametrize("Sk,D", [(2, 64), (40, 128), (1500, 128), (700, 64)])
def test_values_that_are_not_finite_reach_the_rows_that_attend_to_them(Sk, D):
    from lm_engine_b200.ops import attention, attention_reference

    q, k, v = _inputs(2, Sk, 12, 2, D)
    inf = float("inf")
    v[0, Sk // 2, 0, 3] = inf
    v[0, 0, 0, 9] = -inf
    v[0, Sk - 1, 0, 17] = float("nan")
    v[0, 0, 0, 33] = inf                                    # opposite infinities in one column: not a number
    v[0, Sk - 1, 0, 33] = -inf
    v[1, 1, 1, 0] = 3e38                                    # finite, with a finite average
    out = attention(q, k, v, causal=True).float()
    ref = attention_reference(q.double(), k.double(), v.double(), causal=True).double().float()
    # weights of this many random keys stay far above the smallest fp32 number, so no product is 0 * inf
    bad = ~torch.isfinite(ref)
    assert bool(bad[0, 0, :6, [3, 9, 17, 33]].all()) and int(bad.sum()) == 24
    torch.testing.assert_close(out[bad], ref[bad], rtol=0, atol=0, equal_nan=True)
    for b in range(2):      # (the rounding of the result, 2^-9 per element)
        o, r = (t[b].masked_fill(bad[b], 0.0).double() for t in (out, ref))
        assert float((o - r).norm() / r.norm()) < 2.0 ** -8.5
    o, r = (t[0].masked_fill(bad[0], 0.0) for t in (out, ref))
    assert float((o - r).norm() / r.norm()) < 2.0 ** -8.5


def test_values_behind_the_mask_are_not_read():
    from lm_engine_b200.ops import attention

    q, k, v = _inputs(2, 100, 8, 2, 128)
    mask = torch.ones(2, 100, dtype=torch.bool, device="cuda")
    mask[:, :40] = False
    want = attention(q, k, v, causal=True, attention_mask=mask)
    v[:, 7], v[:, 8], k[:, 9] = float("inf"), float("nan"), float("nan")
    assert torch.equal(attention(q, k, v, causal=True, attention_mask=mask), want)
