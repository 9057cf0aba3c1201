"""Addresses that the wrappers hand to the kernels, with the library replaced by a recorder: what a kernel would read
has to lie inside the operand's storage, also where dimensions of size 1 carry strides of their own (contiguous() and
clone() keep those)."""

import pytest
import torch

from lm_engine_b200.ops import _lib

BF = torch.bfloat16


class _Recorder:
    def __init__(self):
        self.calls = {}

    def __getattr__(self, name):
        def call(*args):
            self.calls[name] = args
            return 0
        return call


@pytest.fixture
def lib(monkeypatch):
    rec = _Recorder()
    monkeypatch.setattr(_lib, "cuda_lib", lambda: rec)
    monkeypatch.setattr(_lib, "stream_ptr", lambda: 0)
    return rec


def _wide(B, S, W, offset, C):
    """Slice ``[B, S, C]`` of a projection's rows of W elements, that start at `offset`."""
    return torch.zeros(B, S, W, dtype=BF)[..., offset:offset + C]


GATES = {
    # (gate, rows the kernel may read in place at this pitch; None: a copy)
    "one row, odd width": (lambda: _wide(1, 1, 1542, 6, 1536), None),
    "one row, odd width, aligned": (lambda: _wide(1, 1, 1544 + 3, 8, 1536), 1536),
    "batch, one step": (lambda: _wide(5, 1, 528, 16, 512), 528),
    "rows of a batch": (lambda: _wide(2, 7, 528, 16, 512), 528),
    "odd width": (lambda: _wide(2, 7, 521, 8, 512), None),
    "transposed unit dimension": (lambda: torch.zeros(7, 64, dtype=BF)[None].transpose(0, 1), 64),
    "permuted": (lambda: torch.zeros(3, 5, 64, dtype=BF).transpose(0, 1), None),
    "expanded": (lambda: torch.zeros(1, 64, dtype=BF).expand(4, 64), None),
}


@pytest.mark.parametrize("name", GATES)
def test_gate_rows(lib, monkeypatch, name):
    from lm_engine_b200.ops import activation

    monkeypatch.setattr(activation, "_silu_mul_kernel_usable", lambda y, gate: True)
    make, in_place = GATES[name]
    gate = make().requires_grad_(True)
    y = torch.zeros(gate.shape, dtype=BF, requires_grad=True)
    read = {}
    out = activation.silu_mul(y, gate)
    read["fwd"] = lib.calls["lme_silu_mul_fwd"][1:3]
    out.backward(torch.zeros_like(out))
    read["bwd"] = lib.calls["lme_silu_mul_bwd"][2:4]
    assert y.grad.shape == y.shape and gate.grad.shape == gate.shape
    I, T = gate.size(-1), gate.numel() // gate.size(-1)
    base, n = gate.untyped_storage().data_ptr(), gate.untyped_storage().nbytes() // 2
    for ptr, pitch in read.values():
        assert ptr % 16 == 0 and pitch % 8 == 0
        if in_place is None:
            assert pitch == I        # a dense copy
        else:
            assert pitch == in_place and ptr == gate.data_ptr()
            assert 0 <= (ptr - base) // 2 and (ptr - base) // 2 + (T - 1) * pitch + I <= n


@pytest.mark.parametrize("wrt", [(0, 1), (0,), (1,)])
def test_gradients_of_the_gate_s_gradients(lib, monkeypatch, wrt):
    from lm_engine_b200.ops import activation

    monkeypatch.setattr(activation, "_silu_mul_kernel_usable", lambda y, gate: True)
    ins = [torch.randn(3, 16).to(BF).requires_grad_(i in wrt) for i in range(2)]
    dout, dd, results = torch.randn(3, 16).to(BF).requires_grad_(True), torch.randn(3, 16).to(BF), []
    for f in (activation.silu_mul, activation._silu_mul_statement):
        first = torch.autograd.grad(f(*ins), [ins[i] for i in wrt], dout, create_graph=True)
        second = torch.autograd.grad(first, [dout, *(ins[i] for i in wrt)], [dd] * len(wrt), allow_unused=True)
        results.append([*first, *(t for t in second if t is not None)])
    assert len(results[0]) == len(results[1]) >= 2 * len(wrt)
    assert all(torch.equal(a, b) for a, b in zip(*results))


ROWS = {
    # x [B, S, C], element strides (batch, time) of an in-place read at four taps; None: a dense copy
    "one row, odd width": (lambda: _wide(1, 1, 1001, 8, 16), (16, 16)),
    "one row, aligned width": (lambda: _wide(1, 1, 1008, 8, 16), (16, 16)),
    "one row, misaligned": (lambda: _wide(1, 1, 1008, 4, 16), None),
    "batch, one step": (lambda: _wide(3, 1, 1008, 8, 16), (1008, 16)),
    "batch, one step, odd width": (lambda: _wide(3, 1, 1001, 8, 16), None),
    "steps": (lambda: _wide(2, 5, 48, 8, 16), (240, 48)),
    "unit batch of odd stride": (lambda: torch.zeros(5 * 16 + 3, dtype=BF).as_strided((1, 5, 16), (83, 16, 1)), (80, 16)),
    "dense, misaligned": (lambda: torch.zeros(2 * 5 * 16 + 1, dtype=BF)[1:].view(2, 5, 16), None),
}


@pytest.mark.parametrize("K", [3, 4, 6])
@pytest.mark.parametrize("name", ROWS)
def test_convolution_rows(lib, name, K):
    from lm_engine_b200.ops.conv1d import _CausalConv1d

    make, in_place = ROWS[name]
    x = make().requires_grad_(True)
    B, S, C = x.shape
    y = _CausalConv1d.apply(x, torch.zeros(C, K, dtype=BF, requires_grad=True), None, None, True)
    dy = torch.zeros(y.numel() + 1, dtype=BF)[1:].view(y.shape)          # a contiguous gradient may start anywhere
    y.backward(dy)
    for ptr, x_b, x_t in (lib.calls["lme_causal_conv1d_fwd"][:3], lib.calls["lme_causal_conv1d_bwd"][:3]):
        assert ptr % 16 == 0
        if K == 4 and in_place is not None:
            assert (x_b, x_t) == in_place and ptr == x.data_ptr()
        else:
            assert (x_b, x_t) == (S * C, C)
    assert lib.calls["lme_causal_conv1d_bwd"][6] % 16 == 0


@pytest.mark.parametrize("shape,stride,in_place", [
    ((1, 9, 2, 128), (9 * 256 + 3, 256, 128), True), ((2, 9, 1, 128), (9 * 144, 144, 77), True),
    ((1, 9, 1, 128), (5, 128, 3), True), ((2, 9, 2, 128), (9 * 262, 262, 128), False),
    ((1, 9, 2, 128), (0, 262, 128), False), ((2, 9, 2, 128), (9 * 288, 288, 128), True)])
def test_delta_rule_operands(shape, stride, in_place):
    from lm_engine_b200.ops.recurrence import _delta_operand, _delta_strides

    t = torch.zeros(2 * 9 * 512, dtype=BF).as_strided(shape, (*stride, 1))
    u = _delta_operand(t)
    assert (u.data_ptr() == t.data_ptr()) == in_place
    got = tuple(_delta_strides(u))
    dense = (9 * shape[2] * 128, shape[2] * 128, 128)
    assert got == tuple((s if in_place and n > 1 else d) for s, n, d in zip(stride, shape, dense))


def test_one_token_attention_operands(lib):
    from lm_engine_b200.ops.attention_cuda import decode_attention

    flat = torch.zeros(4096, dtype=BF)
    q = flat.as_strided((1, 1, 4, 64), (1003, 77, 64, 1))          # a unit batch of any stride
    k = flat.as_strided((1, 6, 1, 64), (5, 72, 3, 1))              # and a single head
    v = flat.as_strided((1, 6, 1, 64), (5, 70, 3, 1))              # rows between 16-byte boundaries: a copy
    decode_attention(q, k, v, softmax_scale=1.0)
    args = lib.calls["lme_decode_attention"]
    assert args[:3] == (flat.data_ptr(), 256, 64)
    assert args[3:7] == (flat.data_ptr(), 384, 72, 64)
    assert args[7] != flat.data_ptr() and args[8:11] == (384, 64, 64)
