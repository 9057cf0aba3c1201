"""Generation of one sequence, one token per call, through the recurrent mixers: the projections' slices are single rows
whose widths need not be multiples of 8."""

import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _gated_deltanet(heads):
    from lm_engine_b200.models.config import GatedDeltaNetArgs
    from lm_engine_b200.models.layers.gated_deltanet import GatedDeltaNet

    return GatedDeltaNet(256, GatedDeltaNetArgs(k_head_dim=64, v_head_dim=128, num_k_heads=heads, num_v_heads=heads,
                                                use_gate=True, attention_multiplier=None, allow_neg_eigval=True,
                                                kernel_size=4),
                         0, "normal", 0.05, None, 4, False)


def _mamba2(heads, taps):
    from lm_engine_b200.models.config import Mamba2Args
    from lm_engine_b200.models.layers.mamba2 import Mamba2

    return Mamba2(256, Mamba2Args(state_size=16, intermediate_size=32 * heads, num_heads=heads, conv_kernel_size=taps,
                                  activation_function="silu", num_groups=1, chunk_size=32,
                                  normalization_function="rmsnorm"), 1e-5, 0.05, None, "normal", 4, 0)


MIXERS = {"mamba2-4": lambda: _mamba2(4, 4), "mamba2-3-three-taps": lambda: _mamba2(3, 3),
          "mamba2-8-three-taps": lambda: _mamba2(8, 3), "gated-deltanet-1": lambda: _gated_deltanet(1), "gated-deltanet-3": lambda: _gated_deltanet(3),
          "gated-deltanet-4": lambda: _gated_deltanet(4)}


@pytest.mark.parametrize("name", MIXERS)
def test_steps_of_one_sequence_match_the_whole(name):
    from lm_engine_b200.models import AttentionMaskInfo, GenerationCache, PositionInfo
    from lm_engine_b200.ops import _lib

    torch.manual_seed(0)
    with torch.device("cuda"):
        m = MIXERS[name]().to(BF).eval()
    x = torch.randn(1, 12, 256, device="cuda").to(BF)
    with torch.no_grad():
        whole = m(x)
        cache, parts = GenerationCache(), []
        for piece in x.split([9, 1, 1, 1], dim=1):
            parts.append(m(piece, cache_params=cache, attention_mask_info=AttentionMaskInfo(),
                           position_info=PositionInfo()))
    got = torch.cat(parts, dim=1)
    # two evaluations of the recurrence on bf16 operands: a few roundings of 2^-9 each along a path
    assert float((got.float() - whole.float()).norm() / whole.float().norm()) < 2e-2
    assert _lib.read_status()[0] == 0


@pytest.mark.parametrize("make", [lambda w: w[..., 6:], lambda w: w[..., 8:1544], lambda w: w[0, 0, :1536].view(24, 64)[None].transpose(0, 1)])
def test_gate_of_single_rows(make):
    from lm_engine_b200.ops import silu_mul

    wide = torch.randn(1, 1, 1547, device="cuda").to(BF).requires_grad_(True)
    gate = make(wide)
    gate = gate if gate.size(-1) % 8 == 0 else gate[..., :1536]
    y = torch.randn(gate.shape, device="cuda").to(BF).requires_grad_(True)
    out = silu_mul(y, gate)
    dout = torch.randn_like(out)
    got = torch.autograd.grad(out, (y, wide), dout)
    y64, w64 = (t.detach().double().requires_grad_(True) for t in (y, wide))
    g64 = make(w64)
    want = y64 * torch.nn.functional.silu(g64 if g64.size(-1) % 8 == 0 else g64[..., :1536])
    # two roundings to bf16, each at most 2^-8 of a value
    for a, b in zip((out.detach(), *got), (want.detach(), *torch.autograd.grad(want, (y64, w64), dout.double()))):
        assert float((a.double() - b).norm() / b.norm()) < 2.0 ** -7


@pytest.mark.parametrize("K", [3, 4])
@pytest.mark.parametrize("width,offset", [(1001, 8), (1008, 8), (1008, 4)])
def test_convolution_of_a_single_row(width, offset, K):
    from lm_engine_b200.ops.conv1d import causal_conv1d, causal_conv1d_reference

    wide = torch.randn(1, 1, width, device="cuda").to(BF).requires_grad_(True)
    w = torch.randn(64, K, device="cuda").to(BF).requires_grad_(True)
    state = torch.randn(1, 64, K - 1, device="cuda").to(BF).requires_grad_(True)
    y = causal_conv1d(wide[..., offset:offset + 64], w, None, state, "silu")
    dy = torch.randn(y.numel() + 1, device="cuda").to(BF)[1:].view(y.shape)
    ins = [t.detach().double().requires_grad_(True) for t in (wide, w, state)]
    want = causal_conv1d_reference(ins[0][..., offset:offset + 64], ins[1], None, ins[2], "silu")
    ref = torch.autograd.grad(want, ins, dy.double())
    # fp32 arithmetic, one rounding of each result to bf16
    for a, b in zip((y.detach(), *torch.autograd.grad(y, (wide, w, state), dy)), (want.detach(), *ref)):
        assert float((a.double() - b).norm() / b.norm()) < 2.0 ** -8
