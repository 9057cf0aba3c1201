"""What the SSD scan's kernels get for operands that broadcast or do not fit: they read bare addresses, so shapes are
settled before them.  The autograd function over the kernels is replaced by a recorder."""

import pytest
import torch

from lm_engine_b200.ops import ssd

b, S, N, P, G, Sd, L = 2, 40, 4, 32, 2, 8, 32


@pytest.fixture
def calls(monkeypatch):
    seen = []

    def apply(x, dt, A, B, C, D, L, h):
        seen.append({k: None if t is None else tuple(t.shape)
                     for k, t in dict(x=x, dt=dt, A=A, B=B, C=C, D=D, h=h).items()})
        assert all(t.is_contiguous() for t in (dt, A, D))
        return x, torch.zeros(b, N, P, B.size(-1))

    monkeypatch.setattr(ssd, "scan_glue_eligible", lambda *a: True)
    monkeypatch.setattr(ssd._ChunkScan, "apply", staticmethod(apply))
    return seen


def _operands(**other):
    ops = dict(x=torch.zeros(b, S, N, P, dtype=torch.bfloat16), dt=torch.zeros(b, S, N), A=-torch.ones(N),
               B=torch.zeros(b, S, G, Sd), C=torch.zeros(b, S, G, Sd), D=torch.ones(N))
    ops.update(other)
    return ops


@pytest.mark.parametrize("other", [{}, dict(A=-torch.ones(1)), dict(A=-torch.ones(())), dict(D=torch.ones(1)),
                                   dict(initial_state=torch.zeros(1, N, P, Sd))])
def test_shapes_that_reach_the_kernels(calls, other):
    ssd.ssd_chunk_scan(**_operands(**other), chunk_size=L)
    T = 64
    assert calls == [dict(x=(b, T, N, P), dt=(b, T, N), A=(N,), B=(b, T, G, Sd), C=(b, T, G, Sd), D=(N,),
                          h=(b, N, P, Sd) if "initial_state" in other else None)]


@pytest.mark.parametrize("other", [dict(dt=torch.zeros(b, S, 1)), dict(dt=torch.zeros(b, S, N - 1)),
                                   dict(dt=torch.zeros(1, S, N)), dict(A=-torch.ones(N - 1)),
                                   dict(D=torch.ones(N + 1)), dict(C=torch.zeros(b, S, 1, Sd)),
                                   dict(C=torch.zeros(b, S, G, 2 * Sd)), dict(B=torch.zeros(1, S, G, Sd)),
                                   dict(initial_state=torch.zeros(b, N - 1, P, Sd)),
                                   dict(B=torch.zeros(b, S, 3, Sd), C=torch.zeros(b, S, 3, Sd))])
def test_shapes_that_do_not_fit_raise(calls, other):
    with pytest.raises((RuntimeError, ValueError)):
        ssd.ssd_chunk_scan(**_operands(**other), chunk_size=L)
    assert not calls


def test_other_broadcasts_take_the_general_path(calls):
    ops = _operands(A=-torch.rand(L, N))                   # a decay per position of the chunk
    y, h = ssd.ssd_chunk_scan(**ops, chunk_size=L)
    assert not calls and y.shape == ops["x"].shape


def test_states_of_any_width_reach_the_kernels(calls):
    y, h = ssd.ssd_chunk_scan(**_operands(B=torch.zeros(b, S, G, 12), C=torch.zeros(b, S, G, 12),
                                          initial_state=torch.zeros(b, N, P, 12)), chunk_size=L)
    assert calls[0]["B"] == calls[0]["C"] == (b, 64, G, 16) and calls[0]["h"] == (b, N, P, 16)
    assert h.shape == (b, N, P, 12)
