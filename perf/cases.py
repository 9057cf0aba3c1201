"""Performance cases: what training and serving programs ask of this framework, through its public entry points.

Layer and block sizes are those of the repository's benchmark models and configurations (hidden 2048 / 4096, head dim
128, 64 experts, Mamba-2 with state 128 and chunk 256, gated delta rule with key width 256).  Kinds:

``decode``    one generated token through a decoder block that holds a KV cache (norm, attention, norm, MLP)
``attend``    the attention operator for one new token per sequence over a long cache, plain or left-padded
``prompt``    a whole small model over a prompt, logits out
``block``     forward and backward of a dense decoder block, gradients of the input and of every weight
``norm``      residual add + RMSNorm, forward and backward
``head``      LM head + cross entropy from the hidden states, forward and backward
``moe``       mixture-of-experts layer with its router loss, forward and backward
``mamba2``    Mamba-2 mixer, forward and backward
``deltanet``  gated delta net mixer, forward and backward
``adamw``     one optimizer step on a flat shard

Activations and weights are bf16 as in the mixed-precision runs; decay parameters and optimizer state are fp32.
"""

from __future__ import annotations

import math

import torch
import torch.nn.functional as F

from lm_engine_b200 import ops
from lm_engine_b200.loss import get_autoregressive_language_modeling_loss
from lm_engine_b200.models import AttentionMaskInfo, GenerationCache, PositionInfo, build_model, dense_config
from lm_engine_b200.models.aux_loss import clear_aux_loss, get_aux_loss
from lm_engine_b200.models.blocks import Block
from lm_engine_b200.models.config import GatedDeltaNetArgs, Mamba2Args, MoEArgs
from lm_engine_b200.models.layers.gated_deltanet import GatedDeltaNet
from lm_engine_b200.models.layers.mamba2 import Mamba2
from lm_engine_b200.models.layers.moe import MoE
from lm_engine_b200.models.layers.norm import RMSNorm
from lm_engine_b200.models.layers.rope import RoPE

BF = torch.bfloat16
EPS = 1e-5
DEV = "cuda"


def listed() -> list[dict]:
    return [
        # interactive generation: one user, one token; launches and weight reads are all there is
        dict(name="decode-1x1023", kind="decode", batch=1, past=1023, hidden=4096, inter=14336, heads=32, kv=8),
        # served generation: a batch of users, each with a few hundred tokens behind them
        dict(name="decode-24x500", kind="decode", batch=24, past=500, hidden=4096, inter=14336, heads=32, kv=8),
        # attention of a generation step over long caches, the part of serving that grows with the context
        dict(name="attend-24x3001", kind="attend", batch=24, past=3000, heads=32, kv=8, padded=False),
        # time to first token of the 1B benchmark model's layers (4 of its 16) on a short prompt of odd length
        dict(name="prompt-1x333", kind="prompt", batch=1, seq=333, hidden=2048, inter=5632, heads=16, kv=8, layers=4,
             vocab=32000),
        # one layer of the 8B pretraining benchmark at its micro batch: the bulk of a training step
        dict(name="block-2x4096", kind="block", batch=2, seq=4096, hidden=4096, inter=14336, heads=32, kv=8),
        # fine-tuning of a 1B model on one short document of odd length
        dict(name="block-1x777", kind="block", batch=1, seq=777, hidden=2048, inter=8192, heads=16, kv=4),
        # residual add + norm between the sub-layers of the 8B model
        dict(name="norm-8191x4096", kind="norm", tokens=8191, hidden=4096),
        # LM head and loss of a 128k-vocabulary model
        dict(name="head-4095", kind="head", tokens=4095, hidden=2048, vocab=128256),
        # one layer of the mixture-of-experts benchmark
        dict(name="moe-4096", kind="moe", tokens=4096, hidden=2048, inter=1024, experts=64, top=8),
        # one mixer of the hybrid Mamba-2 configuration at its sequence length
        dict(name="mamba2-1x4096", kind="mamba2", batch=1, seq=4096, hidden=2048, heads=64),
        # one gated delta net mixer, published head layout
        dict(name="deltanet-2x2048", kind="deltanet", batch=2, seq=2048, hidden=2048, heads=4),
        # the optimizer on one rank's shard of a decoder layer of the 8B model (half of it: two ranks)
        dict(name="adamw-109M", kind="adamw", n=109_056_003),
    ]


def _spread(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["decode", "decode", "attend", "prompt", "block", "norm", "head", "moe", "mamba2", "deltanet",
                       "adamw"])
    hidden, inter, heads, kv = rng.choice([(4096, 14336, 32, 8), (2048, 5632, 16, 8), (2048, 8192, 16, 4)])
    dense = dict(hidden=hidden, inter=inter, heads=heads, kv=kv)
    if kind == "decode":
        return dict(kind=kind, batch=_spread(rng, 1, 64), past=_spread(rng, 17, 1500), **dense)
    if kind == "attend":
        return dict(kind=kind, batch=_spread(rng, 1, 32), past=_spread(rng, 100, 4000), heads=heads, kv=kv,
                    padded=rng.random() < 0.5)
    if kind == "prompt":
        return dict(kind=kind, batch=rng.choice([1, 1, 2]), seq=_spread(rng, 64, 1000), layers=4, vocab=32000, **dense)
    if kind == "block":
        return dict(kind=kind, batch=rng.choice([1, 2]), seq=_spread(rng, 200, 4096), **dense)
    if kind == "norm":
        return dict(kind=kind, tokens=_spread(rng, 500, 16384), hidden=rng.choice([1024, 2048, 2560, 4096, 6144]))
    if kind == "head":
        return dict(kind=kind, tokens=_spread(rng, 500, 4096), hidden=2048, vocab=rng.choice([32000, 50304, 128256]))
    if kind == "moe":
        return dict(kind=kind, tokens=_spread(rng, 300, 8192), hidden=2048, inter=1024, experts=64, top=8)
    if kind == "mamba2":
        hidden = rng.choice([2048, 2560])
        return dict(kind=kind, batch=rng.choice([1, 2]), seq=_spread(rng, 500, 4096), hidden=hidden, heads=hidden // 32)
    if kind == "deltanet":
        return dict(kind=kind, batch=rng.choice([1, 2]), seq=_spread(rng, 300, 4096), hidden=2048,
                    heads=rng.choice([3, 4]))
    return dict(kind=kind, n=_spread(rng, 1_000_000, 109_000_000))


# ------------------------------------------------------------------------------------------------------ inputs
class _Random:
    def __init__(self, seed: int) -> None:
        self.g = torch.Generator(device=DEV).manual_seed(seed)

    def normal(self, *shape, std: float = 1.0, dtype=BF) -> torch.Tensor:
        return (torch.randn(*shape, generator=self.g, device=DEV) * std).to(dtype)

    def uniform(self, *shape, lo: float = 0.0, hi: float = 1.0) -> torch.Tensor:
        return torch.rand(*shape, generator=self.g, device=DEV) * (hi - lo) + lo

    def ints(self, hi: int, *shape) -> torch.Tensor:
        return torch.randint(hi, shape, generator=self.g, device=DEV)


def _dense(c: dict, layers: int = 1, vocab: int = 512):
    return dense_config(vocab_size=vocab, hidden_size=c["hidden"], num_layers=layers, num_attention_heads=c["heads"],
                        num_key_value_heads=c["kv"], intermediate_size=c["inter"], head_dim=128,
                        rope_theta=500000, max_position_embeddings=4096)


def _fill(module, r: _Random) -> None:
    """Weights of a model in training: projections normal with std 0.02, norm weights around one, decay parameters
    and short convolutions at the scale of their initialisation."""
    with torch.no_grad():
        for name, p in module.named_parameters():
            leaf = name.split(".")[-1]
            if leaf == "A_log":
                p.data = torch.log(r.uniform(p.numel(), lo=1.0, hi=16.0))
            elif leaf == "dt_bias":
                dt = torch.exp(r.uniform(p.numel(), lo=math.log(1e-3), hi=math.log(1e-1)))
                p.data = dt + torch.log(-torch.expm1(-dt))
            elif leaf == "D" or "norm" in name or ".ln_" in name or name.startswith("ln_"):
                p.data = (1 + r.normal(*p.shape, std=0.1, dtype=torch.float32)).to(BF)
            elif "conv1d" in name:
                p.data = r.uniform(*p.shape, lo=-0.5, hi=0.5).to(BF)
            elif name == "weight" or p.dim() == 1:
                p.data = (1 + r.normal(*p.shape, std=0.1, dtype=torch.float32)).to(BF)
            else:
                p.data = r.normal(*p.shape, std=0.02)


def _module(c: dict, r: _Random):
    kind, H = c["kind"], c["hidden"]
    mix = dict(init_method="normal", initializer_range=0.02, m_width=None, num_layers=4, layer_idx=0)
    with torch.device(DEV):
        if kind in ("decode", "block"):
            m = Block(_dense(c), False, 0)
        elif kind == "norm":
            m = RMSNorm(H, eps=EPS)
        elif kind == "moe":
            m = MoE(H, MoEArgs(mlp_type="MoE", intermediate_size=c["inter"], activation_function="swiglu",
                               num_experts=c["experts"], num_experts_per_tok=c["top"],
                               shared_intermediate_size=None), "normal", 0.02, None, 4, False)
        elif kind == "mamba2":
            m = Mamba2(H, Mamba2Args(state_size=128, intermediate_size=2 * H, num_heads=c["heads"],
                                     conv_kernel_size=4, activation_function="silu", num_groups=1, chunk_size=256,
                                     normalization_function="rmsnorm"), layer_norm_epsilon=EPS, **mix)
        else:
            m = GatedDeltaNet(H, GatedDeltaNetArgs(k_head_dim=256, v_head_dim=512, num_k_heads=c["heads"],
                                                   num_v_heads=c["heads"], use_gate=True, attention_multiplier=None,
                                                   allow_neg_eigval=True, kernel_size=4),
                              use_depth_scaled_init=False, layer_norm_epsilon=EPS, **mix)
    _fill(m, r)
    return m


def _rope_tables():
    with torch.device(DEV):
        return RoPE(128, 4096, base=500000).tables(4096)


def prepare(case: dict, seed: int) -> dict:
    c, r = case, _Random(seed)
    kind = c["kind"]
    s = {"case": c}
    if kind == "decode":
        s["module"] = _module(c, r).eval()
        s["x"] = r.normal(c["batch"], 1, c["hidden"])
        s["key"] = r.normal(c["batch"], c["past"], c["kv"], 128)
        s["value"] = r.normal(c["batch"], c["past"], c["kv"], 128)
        s["positions"] = torch.full((1, 1), c["past"], dtype=torch.long, device=DEV)
        s["tables"] = _rope_tables()
    elif kind == "attend":
        s["q"] = r.normal(c["batch"], 1, c["heads"], 128)
        s["k"] = r.normal(c["batch"], c["past"] + 1, c["kv"], 128)
        s["v"] = r.normal(c["batch"], c["past"] + 1, c["kv"], 128)
        s["mask"] = None
        if c["padded"]:     # prompts of different lengths, padded on the left
            first = (r.uniform(c["batch"], 1) * 0.6 * c["past"]).long()
            s["mask"] = (torch.arange(c["past"] + 1, device=DEV)[None] >= first).long()
    elif kind == "prompt":
        with torch.device(DEV):
            s["module"] = build_model(_dense(c, c["layers"], c["vocab"])).eval()
        _fill(s["module"], r)
        s["tokens"] = r.ints(c["vocab"], c["batch"], c["seq"])
    elif kind == "head":
        s["x"] = r.normal(c["tokens"], c["hidden"]).requires_grad_(True)
        s["weight"] = r.normal(c["vocab"], c["hidden"], std=0.02).requires_grad_(True)
        s["labels"] = r.ints(c["vocab"], c["tokens"])
        s["labels"][r.uniform(c["tokens"]) < 0.05] = -100
        s["scale"] = torch.tensor(1.0 / c["tokens"], device=DEV)
    elif kind == "adamw":
        n = c["n"]
        s["p"], s["m"] = r.normal(n, std=0.02, dtype=torch.float32), r.normal(n, std=1e-3, dtype=torch.float32)
        s["v"] = r.normal(n, std=1e-3, dtype=torch.float32).square_()
        s["g"], s["lp"] = r.normal(n, std=1e-3), torch.empty(n, dtype=BF, device=DEV)
        s["gscale"] = torch.tensor([0.7], device=DEV)
    else:
        s["module"] = m = _module(c, r).train()
        if kind == "norm" or kind == "moe":
            shape = (c["tokens"], c["hidden"])
        else:
            shape = (c["batch"], c["seq"], c["hidden"])
        x = r.normal(*shape)
        if kind == "moe":
            # a trained router is decided: every token leans on `top` experts, some of which are popular
            load = (1 + torch.arange(c["experts"], device=DEV).float()) ** -0.3
            sel = torch.multinomial(load.expand(c["tokens"], -1), c["top"], generator=r.g)
            gate = F.normalize(m.gate.weight.detach().float(), dim=-1)
            x = (x.float() + 9.0 * gate[sel].sum(1)).to(BF)
        s["x"] = x.requires_grad_(True)
        s["dy"] = r.normal(*shape)
        if kind == "norm":
            s["residual"] = r.normal(*shape).requires_grad_(True)
            s["dh"] = r.normal(*shape)
        if kind == "block":
            s["positions"] = torch.arange(c["seq"], device=DEV).view(1, -1)
            s["tables"] = _rope_tables()
        s["wrt"] = [s["x"]] + ([s["residual"]] if kind == "norm" else []) + list(m.parameters())
        if kind == "moe":
            s["daux"] = torch.tensor(0.01, device=DEV, dtype=BF)
    return s


# --------------------------------------------------------------------------------------------------------- one pass
def run(s: dict):
    c = s["case"]
    kind = c["kind"]
    if kind == "decode":
        with torch.no_grad():
            cache = GenerationCache()
            cache.update(0, "key", s["key"])
            cache.update(0, "value", s["value"])
            y = s["module"](s["x"], cache_params=cache, attention_mask_info=AttentionMaskInfo(),
                            position_info=PositionInfo(position_ids=s["positions"], rope_tables=s["tables"],
                                                       sequence_length=c["past"] + 1))
            return y, cache.get(0, "key"), cache.get(0, "value")
    if kind == "attend":
        with torch.no_grad():
            return ops.attention(s["q"], s["k"], s["v"], causal=True, attention_mask=s["mask"])
    if kind == "prompt":
        with torch.no_grad():
            return s["module"](s["tokens"]).logits
    if kind == "head":
        loss = get_autoregressive_language_modeling_loss(None, s["labels"], hidden_states=s["x"],
                                                         vocab_weight=s["weight"], shift_logits_and_labels=False)
        return (loss.detach(), *torch.autograd.grad(loss, (s["x"], s["weight"]), s["scale"]))
    if kind == "adamw":
        ops.adamw_step(s["p"], s["m"], s["v"], s["g"], s["lp"], lr=3e-4, betas=(0.9, 0.95), eps=1e-10,
                       weight_decay=0.1, step=100, gscale=s["gscale"])
        return s["p"], s["m"], s["v"], s["lp"]
    if kind == "norm":
        y, h = s["module"].forward_with_residual(s["x"], s["residual"])
        return (y.detach(), h.detach(), *torch.autograd.grad((y, h), s["wrt"], (s["dy"], s["dh"])))
    if kind == "moe":
        clear_aux_loss()
        y = s["module"](s["x"])
        aux = get_aux_loss()
        clear_aux_loss()
        return (y.detach(), *torch.autograd.grad((y, aux), s["wrt"], (s["dy"], s["daux"])))
    if kind == "block":
        y = s["module"](s["x"], attention_mask_info=AttentionMaskInfo(),
                        position_info=PositionInfo(position_ids=s["positions"], rope_tables=s["tables"],
                                                   sequence_length=c["seq"]))
    else:
        y = s["module"](s["x"])
    return (y.detach(), *torch.autograd.grad(y, s["wrt"], s["dy"]))


# ------------------------------------------------------------------------------------------------ what it takes
def work(case: dict) -> dict:
    c = case
    kind = c["kind"]
    if kind == "adamw":
        return {"bytes": 28 * c["n"], "flops": 12 * c["n"]}
    if kind == "attend":
        kvb = 4 * c["batch"] * (c["past"] + 1) * c["kv"] * 128
        return {"bytes": kvb + 4 * c["batch"] * c["heads"] * 128,
                "flops": 4 * c["batch"] * c["heads"] * (c["past"] + 1) * 128}
    H = c["hidden"]
    if kind == "norm":
        # forward: x, residual -> y, h; backward: dy, dh, h -> dx (the gradient of both summands)
        return {"bytes": 16 * c["tokens"] * H, "flops": 20 * c["tokens"] * H}
    if kind == "head":
        T, V = c["tokens"], c["vocab"]
        return {"bytes": 4 * T * H + 4 * V * H, "flops": 6 * T * H * V}
    if kind == "moe":
        T, W = c["tokens"], 3 * H * c["inter"]
        return {"bytes": 8 * T * H + 4 * c["experts"] * W, "flops": 6 * T * c["top"] * W}
    if kind in ("decode", "prompt", "block"):
        W = H * (c["heads"] + 2 * c["kv"]) * 128 + c["heads"] * 128 * H + 3 * H * c["inter"]
        if kind == "decode":
            B, P = c["batch"], c["past"] + 1
            kvb = 4 * B * P * c["kv"] * 128
            # the cache is read once and comes back one token longer
            return {"bytes": 2 * W + 2 * kvb + 4 * B * H, "flops": 2 * B * W + 4 * B * c["heads"] * P * 128}
        T = c["batch"] * c["seq"]
        att = 2 * T * c["seq"] * c["heads"] * 128          # causal: half of 4 T S d
        if kind == "prompt":
            V, n = c["vocab"], c["layers"]
            return {"bytes": 2 * (n * W + V * H) + 2 * T * V, "flops": 2 * T * (n * W + V * H) + n * att}
        return {"bytes": 4 * W + 8 * T * H, "flops": 6 * T * W + 3.5 * att}
    B, S = c["batch"], c["seq"]
    T = B * S
    if kind == "mamba2":
        inner, state, chunk = 2 * H, 128, 256
        W = H * (2 * inner + 2 * state + c["heads"]) + inner * H
        scan = 2 * T * (chunk // 2) * (state + inner) + 4 * T * inner * state
    else:
        N, K, V, chunk = c["heads"], 256, 512, 64
        W = H * N * (2 * K + V) + H * (2 * N + N * V) + N * V * H
        scan = 2 * T * N * (chunk * (K + K // 2 + V) + 3 * K * V)
    return {"bytes": 4 * W + 8 * T * H, "flops": 6 * T * W + 3 * scan}


def tolerance(case: dict):
    # About four times what the outputs of the kind are off the 64-bit results on the B200: bf16 results carry 2^-9 of
    # rounding each, gradients pass through two or three bf16 intermediates, router weights through bf16 logits.
    kind = case["kind"]
    if kind in ("adamw", "attend", "norm", "head"):
        return {"rel": 7e-3, "max": 0.1}      # seen: 1.7e-3, one rounding (the fp32 states of adamw: 5e-8)
    if kind == "decode":
        return {"rel": 1.6e-2, "max": 0.2}    # seen: 4e-3
    if kind in ("prompt", "moe"):
        return {"rel": 3e-2, "max": 0.8}      # seen: 1.2e-2 after four layers, 1.4e-2 behind the router
    return {"rel": 2.8e-2, "max": 0.8}        # seen: 6e-3 to 9e-3 in the gradients, single values 0.17


# --------------------------------------------------------------------------------------------- 64-bit statements
def _d(t: torch.Tensor) -> torch.Tensor:
    return t.detach().double()


def _norm(x, w):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS) * w


def _rotate(x, cos, sin):
    a, b = x.chunk(2, dim=-1)
    return x * cos[:, None] + torch.cat((-b, a), dim=-1) * sin[:, None]


def _softmax_attention(q, k, v, mask=None):
    """q [B, Sq, N, D], k / v [B, Sk, Nkv, D]: the last Sq positions of a causal sequence of Sk."""
    rep = q.size(2) // k.size(2)
    q, k, v = q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2)
    Sq, Sk = q.size(2), k.size(2)
    hidden = torch.ones(Sq, Sk, dtype=torch.bool, device=DEV).triu(1 + Sk - Sq)
    if mask is not None:
        hidden = hidden[None, None] | (mask == 0)[:, None, None]
    out = []
    for h in range(q.size(1)):
        s = q[:, h] @ k[:, h // rep].transpose(1, 2) / math.sqrt(q.size(-1))
        s = s.masked_fill(hidden if hidden.dim() == 2 else hidden[:, 0], float("-inf"))
        out.append(torch.softmax(s, dim=-1) @ v[:, h // rep])
    return torch.stack(out, dim=2)


def _block(x, w, c, cos, sin, past=None):
    """Pre-norm decoder block; ``w`` maps the block's parameter names to 64-bit tensors."""
    B, S, H = x.shape
    N, KV, G = c["heads"], c["kv"], c["heads"] // c["kv"]
    qkv = (_norm(x, w["ln_1.weight"]) @ w["sequence_mixer.c_attn.weight"].t()).view(B, S, KV, G + 2, 128)
    q = _rotate(qkv[..., :G, :].reshape(B, S, N, 128), cos, sin)
    k, v = _rotate(qkv[..., G, :], cos, sin), qkv[..., G + 1, :]
    if past is not None:
        k, v = torch.cat((past[0], k), dim=1), torch.cat((past[1], v), dim=1)
    x = x + _softmax_attention(q, k, v).reshape(B, S, N * 128) @ w["sequence_mixer.c_proj.weight"].t()
    u = _norm(x, w["ln_2.weight"]) @ w["mlp_block.c_fc.weight"].t()
    return x + (F.silu(u[..., 0::2]) * u[..., 1::2]) @ w["mlp_block.c_proj.weight"].t(), k, v


def _moe(x, w, c):
    logits = x @ w["gate.weight"].t()
    top, sel = logits.topk(c["top"], dim=-1)
    gates = torch.softmax(top, dim=-1)
    y = torch.zeros_like(x)
    for e in range(c["experts"]):
        t, j = (sel == e).nonzero(as_tuple=True)
        if t.numel():
            u = x[t] @ w["c_fc.weight"][e].t()
            h = (F.silu(u[:, 0::2]) * u[:, 1::2]) @ w["c_proj.weight"][e].t()
            y = y.index_add(0, t, h * gates[t, j, None])
    count = torch.bincount(sel.flatten(), minlength=c["experts"]).double()
    share = F.normalize(torch.softmax(logits, dim=-1).sum(0), p=1, dim=0)
    aux = c["experts"] * (share * F.normalize(count, p=1, dim=0)).sum()
    return y, aux + 0.1 * torch.logsumexp(logits, dim=-1).square().mean()


def _conv(x, weight, bias):
    k = weight.size(-1)
    return F.silu(F.conv1d(F.pad(x.transpose(1, 2), (k - 1, 0)), weight, bias, groups=x.size(-1))).transpose(1, 2)


def _blocks_of(t, L):
    """[B, S, N, ...] -> [B, N, S / L, L, ...], padded with zeros to whole blocks."""
    B, S, N = t.shape[:3]
    t = torch.cat((t, t.new_zeros(B, -S % L, *t.shape[2:])), dim=1)
    return t.view(B, -1, L, *t.shape[2:]).movedim(3, 1)


def _decays(cum, strict):
    hidden = torch.ones(cum.size(-1), cum.size(-1), dtype=torch.bool, device=DEV).triu(0 if strict else 1)
    return torch.exp((cum[..., :, None] - cum[..., None, :]).masked_fill(hidden, float("-inf")))


def _mamba2(x, w, c):
    B, S, H = x.shape
    I, N, P, Z, L = 2 * H, c["heads"], 2 * H // c["heads"], 128, 128
    z, u, dt = (x @ w["in_proj.weight"].t()).split((I, I + 2 * Z, N), dim=-1)
    xs, b, cc = _conv(u, w["conv1d.weight"], w["conv1d.bias"]).split((I, Z, Z), dim=-1)
    dt = F.softplus(dt + w["decay_gate.dt_bias"])
    xs = xs.reshape(B, S, N, P)
    xb, bb, cb = _blocks_of(xs * dt[..., None], L), _blocks_of(b[:, :, None], L), _blocks_of(cc[:, :, None], L)
    cum = torch.cumsum(_blocks_of(-torch.exp(w["decay_gate.A_log"]) * dt, L), dim=-1)       # [B, N, n, L]
    y = (_decays(cum, False) * (cb @ bb.transpose(-1, -2))) @ xb
    add = (xb * torch.exp(cum[..., -1:] - cum)[..., None]).transpose(-1, -2) @ bb           # [B, N, n, P, Z]
    h, starts = torch.zeros_like(add[:, :, 0]), []
    for i in range(add.size(2)):
        starts.append(h)
        h = h * torch.exp(cum[:, :, i, -1])[..., None, None] + add[:, :, i]
    y = y + torch.exp(cum)[..., None] * (cb @ torch.stack(starts, dim=2).transpose(-1, -2))
    y = y.movedim(1, 3).reshape(B, -1, N, P)[:, :S] + w["D"][:, None] * xs
    return _norm(y.reshape(B, S, I) * F.silu(z), w["norm.weight"]) @ w["out_proj.weight"].t()


def _deltanet(x, w, c):
    B, S, _ = x.shape
    N, K, V, L = c["heads"], 256, 512, 64
    qkv = _conv(x @ w["qkv_proj.weight"].t(), w["qkv_conv1d.weight"], None)
    q, k, v = (t.reshape(B, S, N, -1) for t in qkv.split((N * K, N * K, N * V), dim=-1))
    a, b, gate = (x @ w["ab_proj.weight"].t()).split((N, N, N * V), dim=-1)
    beta = 2 * torch.sigmoid(b)
    g = -torch.exp(w["decay_gate.A_log"]) * F.softplus(a + w["decay_gate.dt_bias"])
    q = q / (q.norm(dim=-1, keepdim=True) + 1e-6) / math.sqrt(K)
    k = k / (k.norm(dim=-1, keepdim=True) + 1e-6)
    q, k, v, g, beta = (_blocks_of(t, L) for t in (q, k, v, g, beta))
    cum = torch.cumsum(g, dim=-1)
    lower = torch.eye(L, device=DEV, dtype=torch.float64) + beta[..., None] * _decays(cum, True) * (
        k @ k.transpose(-1, -2))
    right = torch.cat((beta[..., None] * v, (beta * torch.exp(cum))[..., None] * k), dim=-1)
    solved = torch.linalg.solve_triangular(lower, right, upper=False, unitriangular=True)
    within = _decays(cum, False) * (q @ k.transpose(-1, -2))
    h, ys = torch.zeros(B, N, K, V, device=DEV, dtype=torch.float64), []
    for i in range(q.size(2)):
        u = solved[:, :, i, :, :V] - solved[:, :, i, :, V:] @ h
        e = torch.exp(cum[:, :, i])
        ys.append(e[..., None] * (q[:, :, i] @ h) + within[:, :, i] @ u)
        left = torch.exp(cum[:, :, i, -1:] - cum[:, :, i])[..., None] * k[:, :, i]
        h = e[..., -1, None, None] * h + left.transpose(-1, -2) @ u
    y = torch.stack(ys, dim=2).movedim(1, 3).reshape(B, -1, N, V)[:, :S]
    y = _norm(y * F.silu(gate.reshape(B, S, N, V)), w["o_norm.weight"])
    return y.reshape(B, S, N * V) @ w["o_proj.weight"].t()


def exact(case: dict, seed: int):
    c, s = case, prepare(case, seed)
    kind = c["kind"]
    if kind == "adamw":
        p, m, v, g = (_d(s[n]) for n in "pmvg")
        g = g * _d(s["gscale"])
        p, m, v = p * (1 - 3e-4 * 0.1), 0.9 * m + 0.1 * g, 0.95 * v + 0.05 * g * g
        p = p - 3e-4 / (1 - 0.9**100) * m / (v.sqrt() / math.sqrt(1 - 0.95**100) + 1e-10)
        return p, m, v, p
    if kind == "attend":
        return _softmax_attention(_d(s["q"]), _d(s["k"]), _d(s["v"]), s["mask"])
    if kind == "head":
        x, w = _d(s["x"]), _d(s["weight"])
        valid = s["labels"] >= 0
        logits = x @ w.t()
        loss = F.cross_entropy(logits, s["labels"], reduction="sum")
        d = torch.softmax(logits, dim=-1)
        d[valid, s["labels"][valid]] -= 1
        d = d * (valid[:, None] * _d(s["scale"]))
        return loss, d @ w, d.t() @ x
    w = {n: _d(p).requires_grad_(True) for n, p in s["module"].named_parameters()}
    if kind == "prompt":
        with torch.no_grad():
            x = w["transformer.wte.weight"][s["tokens"]]
            cos, sin = (_d(t[:c["seq"]]) for t in s["module"].transformer.rope.tables(c["seq"]))
            for i in range(c["layers"]):
                pre = f"transformer.h.{i}."
                x = _block(x, {n[len(pre):]: t for n, t in w.items() if n.startswith(pre)}, c, cos, sin)[0]
            return _norm(x, w["transformer.ln_f.weight"]) @ w["lm_head.weight"].t()
    x = _d(s["x"]).requires_grad_(True)
    if kind == "decode":
        cos, sin = (_d(t[c["past"]:c["past"] + 1]) for t in s["tables"])
        with torch.no_grad():
            return _block(x, w, c, cos, sin, (_d(s["key"]), _d(s["value"])))
    wrt = [x, *w.values()]
    if kind == "norm":
        # the sum is rounded to bf16 before it is normalised: it is an output, and what the next layer adds to
        h = (s["x"].detach() + s["residual"].detach()).double().requires_grad_(True)
        y = _norm(h, w["weight"])
        dh, dw = torch.autograd.grad((y, h), (h, w["weight"]), (_d(s["dy"]), _d(s["dh"])))
        return y.detach(), h.detach(), dh, dh, dw
    if kind == "moe":
        y, aux = _moe(x, w, c)
        return (y.detach(), *torch.autograd.grad((y, aux), wrt, (_d(s["dy"]), _d(s["daux"]))))
    if kind == "block":
        y = _block(x, w, c, *(_d(t[:c["seq"]]) for t in s["tables"]))[0]
    else:
        y = {"mamba2": _mamba2, "deltanet": _deltanet}[kind](x, w, c)
    return (y.detach(), *torch.autograd.grad(y, wrt, _d(s["dy"])))
