"""Mamba-2 state-space-duality (SSD) scan.

``y_t = C_t . h_t + D x_t``,  ``h_t = exp(dt_t A) h_{t-1} + dt_t B_t (x) x_t``  per head, evaluated chunk by chunk:
intra-chunk as a masked ``(C B^T) . decay`` product (tensor-core shaped), chunk summaries ``S_c``, a short sequential
pass over chunk boundaries, and the contribution of the carried state.  Same results as the token-by-token
recurrence (and as ``mamba_chunk_scan_combined`` / the reference's ``mamba2_torch``,
lm_engine/modeling_utils/sequence_mixer_blocks/mamba2/op.py:225-457) without materialising a
``[chunks, L, L, heads, state]`` tensor.
"""

from __future__ import annotations

import torch
import torch.distributed as dist

FUSED_INTRA_CHUNK = True   # tests switch it off to compare the two paths


def ssd_recurrent_step(x, dt, A, B, C, D, h):
    """One token.  x ``[b, N, P]``, dt ``[b, N]``, B/C ``[b, G, Sd]``, h ``[b, N, P, Sd]`` (fp32)."""
    N, G = x.size(1), B.size(1)
    Bh = B.float().repeat_interleave(N // G, dim=1)
    Ch = C.float().repeat_interleave(N // G, dim=1)
    dA = torch.exp(dt.float() * A.float())[..., None, None]
    h = h.float() * dA + (dt.float()[..., None] * x.float())[..., None] * Bh[:, :, None, :]
    y = (h * Ch[:, :, None, :]).sum(-1) + D.float()[None, :, None] * x.float()
    return y.to(x.dtype), h


def _group_mm(a: torch.Tensor, b: torch.Tensor, lowp: bool) -> torch.Tensor:
    """``a @ b`` over the leading (batch, chunk, group) dims with an fp32 result; bf16 operands on the tensor cores
    (the batched tcgen05 GEMM, ``b`` read as its MN-major operand) when the model computes in bf16, plain fp32
    otherwise."""
    lead = a.shape[:-2]
    a2, b2 = a.reshape(-1, *a.shape[-2:]), b.reshape(-1, *b.shape[-2:])
    if lowp:
        from .gemm import bmm

        out = bmm(a2.to(torch.bfloat16), b2.to(torch.bfloat16), b_mn=True)
    else:
        out = torch.bmm(a2.float(), b2.float())
    return out.view(*lead, a.size(-2), b.size(-1))


class _IntraChunk(torch.autograd.Function):
    """``y[l] = sum_{s<=l} exp(cum[l]-cum[s]) CB[l,s] xdt[s]`` per (batch, chunk, head) on CUDA: the decay-masked
    matrix is built in one kernel (bf16), the two products run as batched tensor-core GEMMs, and the backward needs
    one more kernel (group sum of ``dM * decay``); the gradient of ``cum`` follows from ``dy . y`` and
    ``xdt . dxdt`` without another L x L pass."""

    @staticmethod
    def forward(ctx, CB, ct, xdt):
        # CB [b, nc, G, L, L] bf16, ct [b, nc, N, L] fp32, xdt [b, nc, N, L, P] bf16
        from . import _lib

        b, nc, G, L, _ = CB.shape
        N, P = ct.size(2), xdt.size(-1)
        CB, ct, xdt = CB.contiguous(), ct.contiguous(), xdt.contiguous()
        M = torch.empty((b, nc, N, L, L), dtype=torch.bfloat16, device=CB.device)
        _lib.check(_lib.cuda_lib().lme_ssd_decay_matrix(CB.data_ptr(), ct.data_ptr(), M.data_ptr(), b * nc, N, G, L,
                                                        _lib.stream_ptr()), "lme_ssd_decay_matrix")
        _lib.count_launch()
        from .gemm import _bmm_kernel

        # y = M xdt: M is [l, s] (K-major), xdt is [s, P] = [K, N] (MN-major)
        y = _bmm_kernel(M.view(-1, L, L), xdt.view(-1, L, P), False, True, torch.float32).view(b, nc, N, L, P)
        ctx.save_for_backward(M, ct, xdt, y)
        ctx.G = G
        return y

    @staticmethod
    def backward(ctx, dy):
        from . import _lib

        M, ct, xdt, y = ctx.saved_tensors
        b, nc, N, L, P = xdt.shape
        G = ctx.G
        dy32 = dy.contiguous().float()
        dy = dy32.to(torch.bfloat16)
        dyv, xv = dy.view(-1, L, P), xdt.view(-1, L, P)
        from .gemm import _bmm_kernel

        dM = _bmm_kernel(dyv, xv, False, False, torch.bfloat16)          # dy xdt^T  [bcn, L, L]
        # M^T dy: M read as the MN-major A operand, dy [l, P] = [K, N] as the MN-major B operand
        dxdt = _bmm_kernel(M.view(-1, L, L), dyv, True, True, torch.float32).view(b, nc, N, L, P)
        dCB = torch.empty((b, nc, G, L, L), dtype=torch.bfloat16, device=dy.device)
        _lib.check(_lib.cuda_lib().lme_ssd_dcb(dM.data_ptr(), ct.data_ptr(), dCB.data_ptr(), b * nc, N, G, L,
                                               _lib.stream_ptr()), "lme_ssd_dcb")
        _lib.count_launch()
        dct = (dy32 * y).sum(-1) - (xdt.float() * dxdt).sum(-1)   # [b, nc, N, L]
        return dCB, dct, dxdt


class _BoundaryScan(torch.autograd.Function):
    """``h_{c+1} = decay[c] h_c + S_c`` over the chunks of every (batch, head) in one kernel each way.  Returns the
    state at every chunk start in bf16 (``[b, nc, N, P, Sd]``, the operand of the carried-state product) and the
    final state in fp32.  By itself: gradients of the states in fp32; :class:`_ChunkScan` runs the same kernels with
    gradients in the type that its products read."""

    @staticmethod
    def forward(ctx, states, decay, h_init):
        from . import _lib

        b, nc, N, P, Sd = states.shape
        states, decay = states.contiguous(), decay.contiguous()
        h_init = None if h_init is None else h_init.float().contiguous()
        h0 = torch.empty((b, nc, N, P, Sd), dtype=torch.bfloat16, device=states.device)
        keep = any(ctx.needs_input_grad)      # the backward pass walks the fp32 states
        h0f = torch.empty((b, nc, N, P, Sd), dtype=torch.float32, device=states.device) if keep else None
        hf = torch.empty((b, N, P, Sd), dtype=torch.float32, device=states.device)
        _lib.check(_lib.cuda_lib().lme_ssd_boundary_fwd(states.data_ptr(), decay.data_ptr(), _lib.ptr(h_init),
                                                        h0.data_ptr(), _lib.ptr(h0f), hf.data_ptr(), b, nc, N,
                                                        P * Sd, _lib.stream_ptr()), "lme_ssd_boundary_fwd")
        _lib.count_launch()
        ctx.save_for_backward(h0f, decay)
        ctx.has_init = h_init is not None
        return h0, hf

    @staticmethod
    def backward(ctx, dh0, dhf):
        from . import _lib

        h0f, decay = ctx.saved_tensors
        b, nc, N, P, Sd = h0f.shape
        dh0 = None if dh0 is None else dh0.float().contiguous()
        dhf = None if dhf is None else dhf.float().contiguous()
        dstates = torch.empty_like(h0f)
        parts = torch.empty((*decay.shape, (P * Sd + 127) // 128), dtype=torch.float32, device=h0f.device)
        dinit = torch.empty((b, N, P, Sd), dtype=torch.float32, device=h0f.device) if ctx.has_init else None
        _lib.check(_lib.cuda_lib().lme_ssd_boundary_bwd(_lib.ptr(dh0), _lib.ptr(dhf), h0f.data_ptr(),
                                                        decay.data_ptr(), dstates.data_ptr(), 0, parts.data_ptr(),
                                                        _lib.ptr(dinit), b, nc, N, P * Sd, _lib.stream_ptr()),
                   "lme_ssd_boundary_bwd")
        _lib.count_launch()
        return dstates, parts.sum(-1), dinit


def scan_glue_eligible(x: torch.Tensor, L: int) -> bool:
    b, S, N, P = x.shape
    return (x.is_cuda and x.dtype == torch.bfloat16 and L % 32 == 0 and L <= 1024 and P in (32, 64, 128)
            and b * N > 0 and 0 < b * ((S + L - 1) // L) <= 65535 and FUSED_INTRA_CHUNK)


def _per_head(t: torch.Tensor, N: int) -> bool:
    """One value per head, or one for all; other shapes that broadcast take the general path."""
    return t.shape == (N,) or (t.numel() in (1, N) and t.shape[-1:].numel() == t.numel())


def _intra_chunk_fused(Cc, Bc, ct, xdt):
    """CUDA path of the intra-chunk term.  Cc / Bc ``[b, nc, L, G, Sd]``, ct ``[b, nc, N, L]`` fp32,
    xdt ``[b, nc, L, N, P]`` fp32 -> ``[b, nc, L, N, P]`` fp32."""
    Cg = Cc.permute(0, 1, 3, 2, 4).to(torch.bfloat16)                    # [b, nc, G, L, Sd]
    Bg = Bc.permute(0, 1, 3, 2, 4).to(torch.bfloat16)
    from .gemm import bmm

    CB = bmm(Cg.reshape(-1, *Cg.shape[-2:]), Bg.reshape(-1, *Bg.shape[-2:]),
             out_dtype=torch.bfloat16).view(*Cg.shape[:-1], Cg.size(-2))  # [b, nc, G, L, L] bf16
    xh = xdt.permute(0, 1, 3, 2, 4).to(torch.bfloat16)                   # [b, nc, N, L, P]
    y = _IntraChunk.apply(CB, ct, xh)
    return y.permute(0, 1, 3, 2, 4)


def ssd_chunk_scan(x, dt, A, B, C, D, chunk_size: int, initial_state=None):
    """x ``[b, S, N, P]``, dt ``[b, S, N]`` (already softplus'ed), A ``[N]`` (negative), B/C ``[b, S, G, Sd]``,
    D ``[N]``.  Returns ``(y [b, S, N, P], final_state [b, N, P, Sd] fp32)``."""
    b, S, N, P = x.shape
    G, Sd = B.shape[-2:]
    dtype = x.dtype
    L = chunk_size
    pad = (L - S % L) % L
    if scan_glue_eligible(x, L) and _per_head(A, N) and _per_head(D, N):
        return _chunk_scan_kernels(x, dt, A, B, C, D, L, initial_state)
    xf, dtf, Bf, Cf = x.float(), dt.float(), B.float(), C.float()
    if pad:
        xf = torch.nn.functional.pad(xf, (0, 0, 0, 0, 0, pad))
        dtf = torch.nn.functional.pad(dtf, (0, 0, 0, pad))
        Bf = torch.nn.functional.pad(Bf, (0, 0, 0, 0, 0, pad))
        Cf = torch.nn.functional.pad(Cf, (0, 0, 0, 0, 0, pad))
    nc = (S + pad) // L
    xc = xf.view(b, nc, L, N, P)
    dtc = dtf.view(b, nc, L, N)
    Bc = Bf.view(b, nc, L, G, Sd)
    Cc = Cf.view(b, nc, L, G, Sd)
    rep = N // G
    dA = dtc * A.float()                                      # [b, nc, L, N]
    cum = torch.cumsum(dA, dim=2)
    # ---- intra-chunk: y[t] = sum_{s<=t} exp(cum[t]-cum[s]) (C_t.B_s) dt_s x_s
    ct = cum.permute(0, 1, 3, 2)                              # [b, nc, N, L]
    xdt = xc * dtc[..., None]                                 # [b, nc, L, N, P]
    if x.is_cuda and dtype == torch.bfloat16 and L % 8 == 0 and L <= 1024 and FUSED_INTRA_CHUNK:
        y = _intra_chunk_fused(Cc, Bc, ct, xdt)
    else:
        CB = torch.einsum("bclgn,bcsgn->bcgls", Cc, Bc)       # [b, nc, G, L, L]
        CB = CB.repeat_interleave(rep, dim=2)                 # [b, nc, N, L, L]
        seg = ct[..., :, None] - ct[..., None, :]             # cum[t] - cum[s]
        causal = torch.ones(L, L, dtype=torch.bool, device=x.device).tril()
        decay = torch.exp(seg.masked_fill(~causal, float("-inf")))
        y = torch.einsum("bcnls,bcsnp->bclnp", CB * decay, xdt)
    # ---- chunk summaries: S_c = sum_s exp(cum[L-1]-cum[s]) B_s (x) (dt_s x_s)
    # The heads of a group share B and C, so both state products are batched GEMMs over (batch, chunk, group) with
    # the group's heads folded into the GEMM's M / N dimension: no per-head copies of B or C are made.
    lowp = x.is_cuda and dtype == torch.bfloat16
    tail = torch.exp(cum[:, :, -1:, :] - cum)                 # [b, nc, L, N]
    xw = (xdt * tail[..., None]).view(b, nc, L, G, rep * P)   # [b, nc, L, G, rep*P]
    states = _group_mm(xw.permute(0, 1, 3, 4, 2), Bc.permute(0, 1, 3, 2, 4), lowp)   # [b, nc, G, rep*P, Sd]
    states = states.view(b, nc, N, P, Sd)
    # ---- boundary states: h_c = exp(sum dA of chunk c-1) h_{c-1} + S_{c-1}
    h = (torch.zeros(b, N, P, Sd, dtype=torch.float32, device=x.device) if initial_state is None
         else initial_state.float())
    chunk_decay = torch.exp(cum[:, :, -1, :])                 # [b, nc, N]
    starts = []
    for c in range(nc):
        starts.append(h)
        h = h * chunk_decay[:, c, :, None, None] + states[:, c]
    h0 = torch.stack(starts, dim=1)                           # [b, nc, N, P, Sd] state at chunk start
    # ---- carried state contribution: exp(cum[t]) C_t . h_c
    hg = h0.view(b, nc, G, rep * P, Sd)
    off = _group_mm(Cc.permute(0, 1, 3, 2, 4), hg.transpose(-1, -2), lowp)            # [b, nc, G, L, rep*P]
    off = off.permute(0, 1, 3, 2, 4).reshape(b, nc, L, N, P)
    y = y + off * torch.exp(cum)[..., None]
    y = y + D.float()[None, None, None, :, None] * xc
    y = y.reshape(b, nc * L, N, P)[:, :S]
    if pad:
        # padded steps have dt = 0: decay 1, no input, so ``h`` already is the state after the last real token
        pass
    return y.to(dtype), h


class _ChunkScan(torch.autograd.Function):
    """The CUDA composition of :func:`ssd_chunk_scan` for whole chunks.  Per-(token, head) decays, the element-wise
    passes, the decay matrix and the recurrence over chunk boundaries are the kernels of csrc/kernels/ssd.cu, every
    product is the batched tcgen05 GEMM on bf16 operands with fp32 results.  One function instead of a chain of them:
    what the kernels hand to the products' gradients is already in the type that they read, where autograd would cast
    every gradient to its forward tensor's type and back.  x, B and C may be slices of wider rows."""

    @staticmethod
    def forward(ctx, x, dt, A, B, C, D, L, h_init):
        from . import _lib
        from .gemm import _bmm_kernel

        b, S, N, P = x.shape
        G, Sd = B.shape[-2:]
        nc, rep, bf, f32, dev = S // L, N // G, torch.bfloat16, torch.float32, x.device
        bc = b * nc
        lib, st = _lib.cuda_lib(), _lib.stream_ptr()

        def new(*shape, dtype=f32):
            return torch.empty(shape, dtype=dtype, device=dev)

        ct, dtt, tail, ecum, decay = new(bc, N, L), new(bc, N, L), new(bc, N, L), new(bc, L, N), new(bc, N)
        _lib.check(lib.lme_ssd_decay_fwd(dt.data_ptr(), A.data_ptr(), ct.data_ptr(), dtt.data_ptr(), tail.data_ptr(),
                                         ecum.data_ptr(), decay.data_ptr(), bc, N, L, st), "lme_ssd_decay_fwd")
        xs = x.stride(1)
        xh, xwT = new(bc, N, L, P, dtype=bf), new(bc, N, P, L, dtype=bf)
        _lib.check(lib.lme_ssd_prep_fwd(x.data_ptr(), xs, dtt.data_ptr(), tail.data_ptr(), xh.data_ptr(),
                                        xwT.data_ptr(), bc, N, L, P, st), "lme_ssd_prep_fwd")
        Bg, Cg = _chunk_rows(B, bc, L), _chunk_rows(C, bc, L)                # [bc * G, L, Sd]
        CB = _bmm_kernel(Cg, Bg, False, False, bf)                           # C B^T  [bc * G, L, L]
        M = new(bc, N, L, L, dtype=bf)
        _lib.check(lib.lme_ssd_decay_matrix(CB.data_ptr(), ct.data_ptr(), M.data_ptr(), bc, N, G, L, st),
                   "lme_ssd_decay_matrix")
        yin = _bmm_kernel(M.view(-1, L, L), xh.view(-1, L, P), False, True, f32)          # [bc * N, L, P]
        # chunk summaries S_c [rep * P, Sd]: the heads of a group folded into the GEMM's M dimension
        states = _bmm_kernel(xwT.view(bc * G, rep * P, L), Bg, False, True, f32)
        h0, hf = new(b, nc, N, P, Sd, dtype=bf), new(b, N, P, Sd)
        keep = any(ctx.needs_input_grad)      # the backward pass walks the fp32 states
        h0f = new(b, nc, N, P, Sd) if keep else None
        h_init = None if h_init is None else h_init.float().contiguous()
        _lib.check(lib.lme_ssd_boundary_fwd(states.data_ptr(), decay.data_ptr(), _lib.ptr(h_init), h0.data_ptr(),
                                            _lib.ptr(h0f), hf.data_ptr(), b, nc, N, P * Sd, st),
                   "lme_ssd_boundary_fwd")
        h0 = h0.view(bc * G, rep * P, Sd)
        off = _bmm_kernel(Cg, h0, False, False, f32)                         # C_t . h_c  [bc * G, L, rep * P]
        y = new(b, S, N, P, dtype=bf)
        _lib.check(lib.lme_ssd_combine_fwd(yin.data_ptr(), off.data_ptr(), ecum.data_ptr(), D.data_ptr(), x.data_ptr(),
                                           xs, y.data_ptr(), bc, N, L, G, P, st), "lme_ssd_combine_fwd")
        _lib.count_launch(5)
        if keep:
            ctx.save_for_backward(x, dtt, A, D, Bg, Cg, ct, tail, ecum, decay, xh, xwT, M, yin, off, h0, h0f)
        ctx.cfg = (L, G, Sd, h_init is not None)
        return y, hf

    @staticmethod
    def backward(ctx, dy, dhf):
        from . import _lib
        from .gemm import _bmm_kernel

        x, dtt, A, D, Bg, Cg, ct, tail, ecum, decay, xh, xwT, M, yin, off, h0, h0f = ctx.saved_tensors
        L, G, Sd, has_init = ctx.cfg
        b, S, N, P = x.shape
        nc, rep, bf, f32, dev = S // L, N // G, torch.bfloat16, torch.float32, x.device
        bc = b * nc
        lib, st = _lib.cuda_lib(), _lib.stream_ptr()

        def new(*shape, dtype=f32):
            return torch.empty(shape, dtype=dtype, device=dev)

        dy, xs = _lib.aligned(dy.to(bf)), x.stride(1)
        dyin, doff = new(bc * N, L, P, dtype=bf), new(bc * G, L, rep * P, dtype=bf)
        sy, decum, dDp, ddt0, sw, sh, ddt = (new(bc * L * N) for _ in range(7))
        _lib.check(lib.lme_ssd_combine_bwd(dy.data_ptr(), yin.data_ptr(), off.data_ptr(), ecum.data_ptr(), x.data_ptr(),
                                           xs, dyin.data_ptr(), doff.data_ptr(), sy.data_ptr(), decum.data_ptr(),
                                           dDp.data_ptr(), bc, N, L, G, P, st), "lme_ssd_combine_bwd")
        xv = xh.view(-1, L, P)
        dM = _bmm_kernel(dyin, xv, False, False, bf)                         # dy xdt^T  [bc * N, L, L]
        dxh = _bmm_kernel(M.view(-1, L, L), dyin, True, True, f32)           # M^T dy
        dCB = new(bc * G, L, L, dtype=bf)
        _lib.check(lib.lme_ssd_dcb(dM.data_ptr(), ct.data_ptr(), dCB.data_ptr(), bc, N, G, L, st), "lme_ssd_dcb")
        # carried state: off = C h0^T
        dh0 = _bmm_kernel(doff, Cg, True, True, f32)                         # [bc * G, rep * P, Sd]
        dhf = None if dhf is None else dhf.float().contiguous()
        dstates = new(bc * G, rep * P, Sd, dtype=bf)
        parts = (P * Sd + 127) // 128
        ddecay = new(bc, N, parts)
        dinit = new(b, N, P, Sd) if has_init else None
        _lib.check(lib.lme_ssd_boundary_bwd(dh0.data_ptr(), _lib.ptr(dhf), h0f.data_ptr(), decay.data_ptr(),
                                            dstates.data_ptr(), 1, ddecay.data_ptr(), _lib.ptr(dinit), b, nc, N, P * Sd,
                                            st), "lme_ssd_boundary_bwd")
        # chunk summaries: S = xw^T B
        dxwT = _bmm_kernel(dstates, Bg, False, False, bf)                    # [bc * G, rep * P, L]
        dB = _bmm_kernel(xwT.view(bc * G, rep * P, L), dstates, True, True, f32) + _bmm_kernel(dCB, Cg, True, True, f32)
        dC = _bmm_kernel(doff, h0, False, True, f32) + _bmm_kernel(dCB, Bg, False, True, f32)
        dx = new(b, S, N, P, dtype=bf)
        _lib.check(lib.lme_ssd_prep_bwd(x.data_ptr(), xs, dtt.data_ptr(), tail.data_ptr(), dxh.data_ptr(),
                                        dxwT.data_ptr(), dy.data_ptr(), D.data_ptr(), dx.data_ptr(), ddt0.data_ptr(),
                                        sw.data_ptr(), sh.data_ptr(), bc, N, L, P, st), "lme_ssd_prep_bwd")
        dA, dD = new(bc, N), new(bc, N)
        _lib.check(lib.lme_ssd_decay_bwd(dtt.data_ptr(), A.data_ptr(), tail.data_ptr(), ecum.data_ptr(),
                                         decay.data_ptr(), sy.data_ptr(), decum.data_ptr(), ddt0.data_ptr(),
                                         sw.data_ptr(), sh.data_ptr(), ddecay.data_ptr(), parts, dDp.data_ptr(), ddt.data_ptr(),
                                         dA.data_ptr(), dD.data_ptr(), bc, N, L, st), "lme_ssd_decay_bwd")
        _lib.count_launch(5)

        def tokens(t):        # [bc * G, L, Sd] -> [b, S, G, Sd]
            return t.view(bc, G, L, Sd).permute(0, 2, 1, 3).reshape(b, S, G, Sd).to(bf)

        return dx, ddt.view(b, S, N), dA.sum(0), tokens(dB), tokens(dC), dD.sum(0), None, dinit


def _chunk_rows(t: torch.Tensor, bc: int, L: int) -> torch.Tensor:
    """B or C ``[b, S, G, Sd]`` as one ``[L, Sd]`` operand per (chunk, group); a single group is read in place."""
    b, S, G, Sd = t.shape
    if (G == 1 and t.stride(3) == 1 and t.stride(1) % 8 == 0 and t.data_ptr() % 16 == 0
            and (b == 1 or t.stride(0) == S * t.stride(1))):
        return t.as_strided((bc, L, Sd), (L * t.stride(1), t.stride(1), 1), t.storage_offset())
    from ._lib import aligned

    return aligned(t.reshape(bc, L, G, Sd).permute(0, 2, 1, 3).reshape(bc * G, L, Sd))


def _chunk_scan_kernels(x, dt, A, B, C, D, L: int, initial_state):
    """Pads to whole chunks (padded steps have dt = 0: decay 1, no input) and the state to a multiple of 8 (zero columns
    of B and C: the products read 16-byte rows), and runs :class:`_ChunkScan`.  The kernels get bare addresses, so every
    operand takes its full shape here (a mismatch raises)."""
    b, S, N, P = x.shape
    G, Sd = B.shape[-2:]
    if N % G:
        raise ValueError(f"ssd: {N} heads do not split into {G} groups")
    bf = torch.bfloat16
    pad = (L - S % L) % L
    B, C, dt = B.to(bf), C.to(bf), dt.float()
    if not (B.shape == C.shape == (b, S, G, Sd) and dt.shape == (b, S, N)):
        B, C, dt = B.reshape(b, S, G, Sd), C.reshape(b, S, G, Sd), dt.reshape(b, S, N)
    wide = -Sd % 8
    if pad or wide:
        B, C = (torch.nn.functional.pad(t, (0, wide, 0, 0, 0, pad)) for t in (B, C))
    if pad:
        x, dt = torch.nn.functional.pad(x, (0, 0, 0, 0, 0, pad)), torch.nn.functional.pad(dt, (0, 0, 0, pad))
    A, D = (t.float() if t.shape == (N,) else t.float().reshape(-1).expand(N) for t in (A, D))
    if initial_state is not None:
        if initial_state.shape != (b, N, P, Sd):
            initial_state = initial_state.expand(b, N, P, Sd)
        if wide:
            initial_state = torch.nn.functional.pad(initial_state, (0, wide))
    # rows of x: heads contiguous inside a token, one pitch from token to token over the whole batch
    ok = (x.stride(3) == 1 and x.stride(2) == P and x.stride(1) % 8 == 0 and x.data_ptr() % 16 == 0
          and (b == 1 or x.stride(0) == x.size(1) * x.stride(1)))
    from ._lib import aligned

    y, h = _ChunkScan.apply(x if ok else aligned(x), dt.contiguous(), A.contiguous(), B, C,
                            D.contiguous(), L, initial_state)
    return y[:, :S], h[..., :Sd] if wide else h


def ssd_context_parallel_initial_state(final_zero_init: torch.Tensor, total_decay: torch.Tensor, group) -> torch.Tensor:
    """State entering this rank's sequence shard.  ``final_zero_init [b, N, P, Sd]``: the shard's final state when
    started from zero; ``total_decay [b, N]``: ``exp(A sum dt)`` over the shard.  The entering state of rank r is
    ``sum_{j<r} (prod_{j<i<r} decay_i) final_j`` (lm_engine/modeling_utils/sequence_mixer_blocks/mamba2/op.py:73-145)."""
    return _CPPrefix.apply(final_zero_init, total_decay, group)


class _CPPrefix(torch.autograd.Function):
    @staticmethod
    def forward(ctx, f, d, group):
        world, r = dist.get_world_size(group), dist.get_rank(group)
        fs = [torch.empty_like(f) for _ in range(world)]
        ds = [torch.empty_like(d) for _ in range(world)]
        dist.all_gather(fs, f.contiguous(), group=group)
        dist.all_gather(ds, d.contiguous(), group=group)
        h = torch.zeros_like(f)
        for j in range(r):
            h = h * ds[j][..., None, None] + fs[j]
        ctx.group = group
        ctx.save_for_backward(torch.stack(fs), torch.stack(ds))
        return h

    @staticmethod
    def backward(ctx, g):
        fs, ds = ctx.saved_tensors
        group = ctx.group
        world, r = dist.get_world_size(group), dist.get_rank(group)
        # every rank needs d(loss_i)/d(f_r), d(loss_i)/d(d_r) for the later ranks i > r: exchange the incoming grads
        gs = [torch.empty_like(g) for _ in range(world)]
        dist.all_gather(gs, g.contiguous(), group=group)
        gf = torch.zeros_like(g)
        gd = torch.zeros_like(ds[0])
        for i in range(r + 1, world):
            # h_i = sum_{j<i} (prod_{j<k<i} d_k) f_j
            coef = torch.ones_like(ds[0])
            for k in range(r + 1, i):
                coef = coef * ds[k]
            gf = gf + gs[i] * coef[..., None, None]
            # dependence on d_r (r >= 1 contributes to h_i through the terms with j < r)
            if r >= 1:
                prefix = torch.zeros_like(g)
                for j in range(r):
                    prefix = prefix * ds[j][..., None, None] + fs[j]   # = h_r
                gd = gd + (gs[i] * prefix).sum((-1, -2)) * coef
        return gf, gd, None
