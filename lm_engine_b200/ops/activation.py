"""SwiGLU on the packed interleaved layout: ``y = x[..., 1::2] * silu(x[..., ::2])``.

Same layout as the reference's GLU activations (lm_engine/modeling_utils/activations/glu.py:52-59): gate at even
columns, up-projection at odd columns, which is what lets the GEMM epilogue fuse the activation (each accumulator
row holds adjacent gate/up pairs).
"""

from __future__ import annotations

import torch
import torch.nn.functional as F

from . import _lib


def swiglu_packed_reference(x: torch.Tensor) -> torch.Tensor:
    xf = x.float()
    return (xf[..., 1::2] * F.silu(xf[..., ::2])).to(x.dtype)


class _SwiGLU(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x):
        I2 = x.size(-1)
        x2 = x.reshape(-1, I2).contiguous()
        y = torch.empty((x2.size(0), I2 // 2), dtype=x.dtype, device=x.device)
        _lib.check(_lib.cuda_lib().lme_swiglu_fwd(x2.data_ptr(), y.data_ptr(), x2.size(0), I2 // 2,
                                                  _lib.stream_ptr()), "lme_swiglu_fwd")
        _lib.count_launch()
        ctx.save_for_backward(x2)
        ctx.shape = x.shape
        return y.view(*x.shape[:-1], I2 // 2)

    @staticmethod
    def backward(ctx, dy):
        (x2,) = ctx.saved_tensors
        dy2 = dy.reshape(x2.size(0), -1).contiguous()
        dx = torch.empty_like(x2)
        _lib.check(_lib.cuda_lib().lme_swiglu_bwd(x2.data_ptr(), dy2.data_ptr(), dx.data_ptr(), x2.size(0),
                                                  dy2.size(1), _lib.stream_ptr()), "lme_swiglu_bwd")
        _lib.count_launch()
        return dx.view(ctx.shape)


def swiglu_packed(x: torch.Tensor) -> torch.Tensor:
    if x.is_cuda and x.dtype == torch.bfloat16 and x.size(-1) % 16 == 0:
        return _SwiGLU.apply(x)
    return swiglu_packed_reference(x)


def swiglu_backward(preact: torch.Tensor, dy: torch.Tensor, tile_group: torch.Tensor | None = None) -> torch.Tensor:
    """d(preact) given the packed pre-activation and d(out) (used by the fused MLP op).  ``tile_group`` (int32, one
    entry per 128 rows): only tiles with an entry >= 0 are read and written (the grouped GEMMs' padded layout)."""
    if preact.is_cuda and preact.dtype == torch.bfloat16:
        p2 = preact.reshape(-1, preact.size(-1))
        d2 = dy.reshape(p2.size(0), -1).contiguous()
        dx = torch.empty_like(p2)
        if tile_group is not None and p2.size(0) == tile_group.numel() * 128:
            _lib.check(_lib.cuda_lib().lme_swiglu_bwd_tiles(p2.data_ptr(), d2.data_ptr(), dx.data_ptr(), p2.size(0),
                                                            d2.size(1), tile_group.data_ptr(), _lib.stream_ptr()),
                       "lme_swiglu_bwd_tiles")
            _lib.count_launch()
            return dx.view(preact.shape)
        _lib.check(_lib.cuda_lib().lme_swiglu_bwd(p2.data_ptr(), d2.data_ptr(), dx.data_ptr(), p2.size(0),
                                                  d2.size(1), _lib.stream_ptr()), "lme_swiglu_bwd")
        _lib.count_launch()
        return dx.view(preact.shape)
    g = preact[..., ::2].float()
    u = preact[..., 1::2].float()
    s = torch.sigmoid(g)
    d = dy.float()
    out = torch.empty_like(preact, dtype=torch.float32)
    out[..., ::2] = d * u * s * (1 + g * (1 - s))
    out[..., 1::2] = d * g * s
    return out.to(preact.dtype)


def _row_pitch(t: torch.Tensor) -> int | None:
    """Elements from row to row of ``t`` read as ``[rows, t.size(-1)]`` in place (16-byte accesses), ``None`` where no
    single pitch does it.  Dimensions of size 1 have no say: their strides are arbitrary, also in tensors that count as
    contiguous."""
    if t.stride(-1) != 1 or t.data_ptr() % 16:
        return None
    pitch = following = None
    for d in range(t.dim() - 2, -1, -1):
        if t.size(d) == 1:
            continue
        if pitch is None:
            pitch = t.stride(d)
        elif t.stride(d) != following:
            return None
        following = t.stride(d) * t.size(d)
    if pitch is None:
        return t.size(-1)
    return pitch if pitch % 8 == 0 and pitch >= t.size(-1) else None


def _rows(t: torch.Tensor) -> tuple[torch.Tensor, int]:
    """``t`` with its row pitch, copied where it has none."""
    pitch = _row_pitch(t)
    return (_lib.aligned(t), t.size(-1)) if pitch is None else (t, pitch)


class _SiLUMul(torch.autograd.Function):
    """y dense, gate with one row pitch (:func:`silu_mul` sees to both)."""

    @staticmethod
    def forward(ctx, y, gate, pitch):
        I = y.size(-1)
        out = torch.empty(y.shape, dtype=y.dtype, device=y.device)
        _lib.check(_lib.cuda_lib().lme_silu_mul_fwd(y.data_ptr(), gate.data_ptr(), pitch, out.data_ptr(),
                                                    y.numel() // I, I, _lib.stream_ptr()), "lme_silu_mul_fwd")
        _lib.count_launch()
        ctx.save_for_backward(y, gate)
        return out

    @staticmethod
    def backward(ctx, dout):
        y, gate = ctx.saved_tensors
        if torch.is_grad_enabled():         # a graph of the gradients is asked for
            y, gate = y.view_as(y), gate.view_as(gate)
            wrt = [t for t, needed in zip((y, gate), ctx.needs_input_grad) if needed]
            grads = iter(torch.autograd.grad(_silu_mul_statement(y, gate), wrt, dout, create_graph=True))
            return tuple(next(grads) if needed else None for needed in ctx.needs_input_grad)
        gate, pitch = _rows(gate)           # (a saved-tensor hook may return other strides)
        y, dout = _lib.aligned(y), _lib.aligned(dout)
        I = y.size(-1)
        dy, dg = (torch.empty(y.shape, dtype=y.dtype, device=y.device) for _ in range(2))
        _lib.check(_lib.cuda_lib().lme_silu_mul_bwd(dout.data_ptr(), y.data_ptr(), gate.data_ptr(), pitch,
                                                    dy.data_ptr(), dg.data_ptr(), y.numel() // I, I,
                                                    _lib.stream_ptr()), "lme_silu_mul_bwd")
        _lib.count_launch()
        return dy, dg, None


def _silu_mul_kernel_usable(y: torch.Tensor, gate: torch.Tensor) -> bool:
    return (y.dtype == gate.dtype == torch.bfloat16 and y.shape == gate.shape and y.dim() >= 2
            and y.size(-1) % 8 == 0 and y.numel() > 0 and _lib.eager(y, gate))


def _silu_mul_statement(y, gate):
    return y * torch.nn.functional.silu(gate.float()).to(gate.dtype)


def silu_mul(y: torch.Tensor, gate: torch.Tensor) -> torch.Tensor:
    """``y * silu(gate)``, the activation rounded to its input type; ``gate`` may be a slice of wider rows."""
    if _silu_mul_kernel_usable(y, gate):
        return _SiLUMul.apply(_lib.aligned(y), *_rows(gate))
    return _silu_mul_statement(y, gate)
