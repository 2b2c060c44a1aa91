"""Performance cases of the framework: what its users have it do, with inputs, one pass, and the expected results.

The widths are those of the named presets of ``ksa_b200.config`` ("qwen3-1.9b-ksa", the training benchmark, and "ksa-4b",
the inference benchmark).  A case has one of eight kinds:

=============  =======================================================================================================
``proj``       the QKV projection of a few to a few hundred rows (``ops.linear``): one decode step of a batch
``mlp``        residual add, norm and feed-forward block of a few rows (``SwiGluMlp.forward_after_norm``): decoding
``layer``      one decoder layer without gradients (``KsaDecoderLayer``): prefill of a prompt
``attn``       attention alone on packed rows without gradients (``ops.attention_packed``): prefill of a long prompt
``train``      one decoder layer forward and backward, weight gradients in fp32 ``main_grad`` buffers as the training
               engine keeps them
``head``       output head and cross entropy, forward and backward (``ops.linear_cross_entropy``)
``adamw``      the optimizer of one unit of parameters (``ops.adamw_step``)
``serve``      a whole request on the inference engine: prefill, then decoding with given tokens; returns all logits
=============  =======================================================================================================
"""
from __future__ import annotations

import math

import torch

from ksa_b200 import ops
from ksa_b200.config import get_preset
from ksa_b200.inference.engine import KsaInferenceEngine
from ksa_b200.models import get_model_class
from ksa_b200.models.qwen3_ksa import BatchMeta, KsaDecoderLayer, SwiGluMlp

TRAIN, SERVE = "qwen3-1.9b-ksa", "ksa-4b"
BETA1, BETA2, ADAM_EPS, DECAY = 0.9, 0.95, 1e-8, 0.1


def listed():
    return [
        # one user decoding: the feed-forward block of one row, two launches that stream the weights
        {"name": "mlp_decode_1", "kind": "mlp", "model": SERVE, "rows": 1},
        # a small batch decoding
        {"name": "proj_decode_16", "kind": "proj", "model": SERVE, "rows": 16},
        # a server's batch of sequences decoding together: too many rows for a matrix-vector kernel, few for a GEMM tile
        {"name": "mlp_decode_48", "kind": "mlp", "model": SERVE, "rows": 48},
        # a chat prompt of odd length
        {"name": "layer_prompt_333", "kind": "layer", "model": SERVE, "batch": 1, "len": 333, "summary": True},
        # long-context prefill: the full-attention layers dominate it, the summary layers are the most numerous
        {"name": "attn_prompt_16k_full", "kind": "attn", "model": SERVE, "batch": 1, "len": 16384, "summary": False},
        {"name": "attn_prompt_32k_ksa", "kind": "attn", "model": SERVE, "batch": 1, "len": 32768, "summary": True},
        # fine-tuning on short ragged sequences
        {"name": "train_ksa_2x700", "kind": "train", "model": TRAIN, "batch": 2, "len": 700, "summary": True},
        # pretraining at the benchmark's length: both layer types of the hybrid stack
        {"name": "train_ksa_8k", "kind": "train", "model": TRAIN, "batch": 1, "len": 8192, "summary": True},
        {"name": "train_full_8k", "kind": "train", "model": TRAIN, "batch": 1, "len": 8192, "summary": False},
        # the loss of a training step (half of its tokens)
        {"name": "head_4k", "kind": "head", "model": TRAIN, "tokens": 4096},
        # the optimizer over the weights of one layer, as the training engine launches it per unit
        {"name": "adamw_layer", "kind": "adamw", "params": 58_724_608},
        # a request of a batch of four on the engine: prompts of about eight chunks, then tokens one by one across a
        # chunk boundary; four layers (three summary, one full) of the served width
        {"name": "serve_4x1000", "kind": "serve", "model": SERVE, "batch": 4, "len": 1000, "new": 32},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mlp", "proj", "layer", "attn", "train", "train", "head", "adamw", "serve"])
    if kind in ("mlp", "proj"):
        return {"kind": kind, "model": rng.choice([TRAIN, SERVE]), "rows": _log(rng, 1, 1024)}
    if kind in ("layer", "attn"):               # prompts of one or a few requests
        b = rng.choice([1, 1, 2, 3])
        return {"kind": kind, "model": rng.choice([TRAIN, SERVE]), "batch": b, "len": _log(rng, 130, 16000 // b),
                "summary": rng.random() < 0.7}
    if kind == "train":
        b = rng.choice([1, 1, 2, 4])
        return {"kind": kind, "model": TRAIN, "batch": b, "len": _log(rng, 130, 8192 // b), "summary": rng.random() < 0.7}
    if kind == "head":
        return {"kind": kind, "model": TRAIN, "tokens": _log(rng, 100, 4096)}
    if kind == "adamw":
        return {"kind": kind, "params": _log(rng, 1 << 16, 60_000_000)}
    return {"kind": kind, "model": SERVE, "batch": rng.randint(1, 6), "len": _log(rng, 130, 1000), "new": rng.randint(8, 32)}


# ------------------------------------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _normal(g, *shape, std=1.0, dtype=torch.bfloat16):
    return (torch.randn(*shape, generator=g, device="cuda") * std).to(dtype)


def _fill(module, g):
    """Benchmark initialisation: N(0, 0.02) matrices; norm scales spread around one, as trained ones are."""
    with torch.no_grad():
        for p in module.parameters():
            if p.dim() >= 2:
                p.normal_(0.0, 0.02, generator=g)
            else:
                p.copy_(1.0 + 0.1 * torch.randn(p.shape, generator=g, device="cuda"))
    return module


def _new(make, g):
    with torch.device("meta"):
        m = make()
    return _fill(m.to_empty(device="cuda").to(torch.bfloat16), g)


def _serve_config(case):
    cfg = get_preset(case["model"])
    return cfg.model_copy(update={"num_layers": 4, "summary_layer_freq": [1, 1, 1, 0]})


def _layer(case, g):
    cfg = get_preset(case["model"])
    return cfg, _new(lambda: KsaDecoderLayer(cfg, 0, case["summary"], cfg.summary_sliding_chunk_num, 0), g)


def _meta(case, cfg):
    layout = ops.get_layout(case["len"], cfg.summary_chunk_size, cfg.summary_token_num, cfg.summary_chunk_position_ids_type,
                            cfg.summary_token_position_ids_type, case["kind"] != "train")
    return BatchMeta(case["batch"], case["len"], layout, "cuda", False)


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    s = {"case": case}
    if kind in ("mlp", "proj", "layer", "attn", "head"):
        cfg = s["cfg"] = get_preset(case["model"])
        D = cfg.embed_dim
    if kind == "proj":
        s["w"] = _normal(g, (cfg.num_heads + 2 * cfg.num_kv_heads) * cfg.head_dim, D, std=0.02)
        s["x"] = _normal(g, case["rows"], D)
    elif kind == "mlp":
        s["mlp"] = _new(lambda: SwiGluMlp(D, cfg.intermediate_dim), g)
        s["norm"] = (1.0 + 0.1 * torch.randn(D, generator=g, device="cuda")).bfloat16()
        s["x"], s["delta"] = _normal(g, case["rows"], D, std=2.0), _normal(g, case["rows"], D)
    elif kind in ("layer", "train"):
        cfg, layer = _layer(case, g)
        s.update(cfg=cfg, layer=layer, meta=_meta(case, cfg))
        rows = case["batch"] * (case["len"] + s["meta"].Ns)
        # what the previous layer leaves: the residual stream and a feed-forward output that the first norm adds; a full
        # layer is followed by summary layers, so its input carries the summary rows too (its own output does not)
        s["x"], s["delta"] = _normal(g, rows, cfg.embed_dim, std=2.0), _normal(g, rows, cfg.embed_dim)
        if kind == "train":
            s["dx"] = _normal(g, rows, cfg.embed_dim, std=1e-2)
            n_out = rows if case["summary"] and s["meta"].Ns > 0 else case["batch"] * case["len"]
            s["dd"] = _normal(g, n_out, cfg.embed_dim, std=1e-2)
            for p in layer.parameters():
                p.main_grad = torch.zeros(p.shape, dtype=torch.float32, device="cuda")
    elif kind == "attn":
        layout = _meta(case, cfg)
        s["Ns"] = layout.Ns if case["summary"] else 0
        rows = case["batch"] * (case["len"] + s["Ns"])
        s["qkv"] = _normal(g, rows, (cfg.num_heads + 2 * cfg.num_kv_heads) * cfg.head_dim)
    elif kind == "head":
        s["w"] = torch.nn.Parameter(_normal(g, cfg.vocab_size, D, std=0.02))
        s["w"].main_grad = torch.zeros(s["w"].shape, dtype=torch.float32, device="cuda")
        s["h"] = _normal(g, case["tokens"], D)
        labels = torch.randint(0, cfg.vocab_size, (case["tokens"],), generator=g, device="cuda")
        labels[torch.rand(case["tokens"], generator=g, device="cuda") < 0.1] = -100          # masked positions
        s["labels"] = labels
    elif kind == "adamw":
        n = case["params"]
        s["master"] = _normal(g, n, std=0.02, dtype=torch.float32)
        s["grad"] = _normal(g, n, std=1e-3, dtype=torch.float32)
        s["m"] = _normal(g, n, std=1e-4, dtype=torch.float32)
        s["v"] = _normal(g, n, std=1e-3, dtype=torch.float32).square_()
        s["bf16"] = torch.empty(n, dtype=torch.bfloat16, device="cuda")
        s["hyper"] = torch.tensor([1e-3, 1 - BETA1 ** 10, 1 - BETA2 ** 10, 0.5], dtype=torch.float32, device="cuda")
        s["sumsq"] = torch.zeros(1, dtype=torch.float32, device="cuda")
    else:
        cfg = _serve_config(case)
        model = _new(lambda: get_model_class(cfg.model_class)(cfg), g)
        s["engine"] = KsaInferenceEngine(model, max_len=case["len"] + case["new"] + cfg.summary_chunk_size, batch=case["batch"])
        ids = torch.randint(0, 150000, (case["batch"], case["len"] + case["new"]), generator=g, device="cuda")
        s["prompt"], s["next"] = ids[:, :case["len"]].contiguous(), ids[:, case["len"]:].t().contiguous()
    return s


# ------------------------------------------------------------------------------------------------- one pass
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "proj":
        with torch.no_grad():
            return ops.linear(s["x"], s["w"])
    if kind == "mlp":
        with torch.no_grad():
            return s["mlp"].forward_after_norm(s["x"], s["delta"], s["norm"], s["cfg"].norm_eps)
    if kind == "layer":
        with torch.no_grad():
            return s["layer"](s["x"], s["delta"], s["meta"])
    if kind == "attn":
        cfg = s["cfg"]
        window = cfg.summary_sliding_chunk_num if s["Ns"] > 0 else ops.UNBOUNDED_WINDOW
        with torch.no_grad():
            return ops.attention_packed(s["qkv"], case["batch"], case["len"], s["Ns"], cfg.num_heads, cfg.num_kv_heads,
                                        cfg.head_dim, cfg.summary_chunk_size, cfg.summary_token_num, window)
    if kind == "train":
        params = dict(s["layer"].named_parameters())
        for p in params.values():
            p._grad_written = False                  # a new accumulation window: the first write overwrites
        x, delta = s["x"].detach().requires_grad_(), s["delta"].detach().requires_grad_()
        x2, out = s["layer"](x, delta, s["meta"])
        torch.autograd.backward([x2, out], [s["dx"], s["dd"]])
        return {"x": x2.detach(), "out": out.detach(), "dx": x.grad, "ddelta": delta.grad,
                "weights": {k: p.main_grad for k, p in params.items() if p._grad_written}}
    if kind == "head":
        s["w"]._grad_written = False
        h = s["h"].detach().requires_grad_()
        loss = ops.linear_cross_entropy(h, s["w"], s["labels"])
        loss.backward()
        return {"loss": loss.detach(), "dh": h.grad, "dw": s["w"].main_grad}
    if kind == "adamw":
        s["sumsq"].zero_()
        ops.adamw_step(s["master"], s["grad"], s["m"], s["v"], s["bf16"], s["hyper"], BETA1, BETA2, ADAM_EPS, DECAY, 0.0,
                       s["sumsq"])
        return {k: s[k] for k in ("master", "m", "v", "bf16", "sumsq")}
    engine = s["engine"]
    return torch.stack([engine.prefill(s["prompt"])] + [engine.decode_step(t) for t in s["next"]])


# ------------------------------------------------------------------------------------------------- what a pass needs
def _pairs(L, ns, cfg, summary):
    """(query, key) pairs of one sequence and head."""
    if not summary or ns == 0:
        return L * (L + 1) // 2
    C, S, W = cfg.summary_chunk_size, cfg.summary_token_num, cfg.summary_sliding_chunk_num
    n = 0
    for c in range((L + C - 1) // C):
        t = min(C, L - c * C)
        n += t * (t + 1) // 2 + t * (min(c, W) * C + max(0, c - W) * S)
        if c * S < ns:
            n += S * t + S * (S + 1) // 2
    return n


def _layer_work(cfg, B, L, ns, summary):
    """(weights, bytes of one row's input and output, flops of the forward pass) of one decoder layer."""
    D, F = cfg.embed_dim, cfg.intermediate_dim
    qkv, o = (cfg.num_heads + 2 * cfg.num_kv_heads) * cfg.head_dim, cfg.num_heads * cfg.head_dim
    per_row = D * qkv + o * D + 3 * D * F
    weights = per_row + (D * qkv if summary else 0)
    rows = B * (L + (ns if summary else 0))
    flops = 2.0 * rows * per_row + 4.0 * B * cfg.num_heads * cfg.head_dim * _pairs(L, ns, cfg, summary)
    return weights, rows, flops


def work(case):
    kind = case["kind"]
    if kind == "adamw":
        return {"bytes": 30.0 * case["params"], "flops": 15.0 * case["params"]}
    cfg = get_preset(case["model"])
    D, F = cfg.embed_dim, cfg.intermediate_dim
    qkv = (cfg.num_heads + 2 * cfg.num_kv_heads) * cfg.head_dim
    if kind == "proj":
        M = case["rows"]
        return {"bytes": 2.0 * (qkv * D + M * D + M * qkv), "flops": 2.0 * M * D * qkv}
    if kind == "mlp":
        M = case["rows"]
        return {"bytes": 2.0 * (3 * D * F + D + 4 * M * D), "flops": 6.0 * M * D * F}
    if kind == "head":
        T, V = case["tokens"], cfg.vocab_size
        return {"bytes": 2.0 * V * D + 4.0 * V * D + 4.0 * T * D + 8.0 * T, "flops": 6.0 * T * V * D}
    C, S = cfg.summary_chunk_size, cfg.summary_token_num
    if kind == "serve":
        B, L, new = case["batch"], case["len"], case["new"]
        V, layers = cfg.vocab_size, 4
        weights = sum(_layer_work(cfg, 1, 1, 0, i < 3)[0] for i in range(layers)) + V * D
        flops = sum(_layer_work(cfg, B, L, L // C * S, i < 3)[2] for i in range(layers)) + 2.0 * B * D * V
        flops += new * 2.0 * B * weights
        return {"bytes": 2.0 * weights * (1 + new) + 4.0 * B * V * (1 + new), "flops": flops}
    B, L = case["batch"], case["len"]
    ns = (L // C if kind != "train" else (L + C - 1) // C) * S
    if kind == "attn":
        ns = ns if case["summary"] else 0
        rows, H = B * (L + ns), cfg.num_heads
        return {"bytes": 2.0 * rows * (qkv + H * cfg.head_dim),
                "flops": 4.0 * B * H * cfg.head_dim * _pairs(L, ns, cfg, case["summary"])}
    weights, rows, flops = _layer_work(cfg, B, L, ns, case["summary"])
    every = B * (L + ns)
    if kind == "layer":
        return {"bytes": 2.0 * (weights + 3 * every * D + rows * D), "flops": flops}
    att = 4.0 * B * cfg.num_heads * cfg.head_dim * _pairs(L, ns, cfg, case["summary"])
    # weights read and their fp32 gradients written; inputs, outputs and the gradients of both
    return {"bytes": 6.0 * weights + 2.0 * (6 * every * D + 2 * rows * D), "flops": 3.0 * (flops - att) + 3.5 * att}


def tolerance(case):
    kind = case["kind"]
    if kind == "adamw":
        return {"rel": 4e-3, "max": 0.02}              # the bf16 copy of the weights; a value may round the other way
    if kind == "serve":
        return {"rel": 0.03, "max": 0.3}
    if kind == "train":
        return {"rel": 0.012, "max": 0.3}
    if kind == "head":
        return {"rel": 0.01, "max": 0.3}
    return {"rel": 0.01, "max": 0.2}


# ------------------------------------------------------------------------------------------------- the same in 64 bits
def _rms(x, w, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w


def _rope(x, pos, theta):
    """``x`` ``[rows, heads, d]``; halves rotated."""
    d = x.shape[-1]
    inv = theta ** (-torch.arange(0, d, 2, device=x.device, dtype=torch.float64) / d)
    ang = pos.double()[:, None] * inv[None, :]
    cos, sin = ang.cos()[:, None, :], ang.sin()[:, None, :]
    a, b = x[..., :d // 2], x[..., d // 2:]
    return torch.cat([a * cos - b * sin, b * cos + a * sin], dim=-1)


def _mask(q0, q1, L, ns, C, S, W, device):
    """Keys (``L`` text, then ``ns`` summary) that the queries ``q0 .. q1`` of the same numbering see."""
    q, k = torch.arange(q0, q1, device=device)[:, None], torch.arange(L + ns, device=device)[None, :]
    if ns == 0:
        return k <= q
    q_text, k_text = q < L, k < L
    qc = torch.where(q_text, q // C, (q - L) // S)
    kc = torch.where(k_text, k // C, (k - L) // S)
    text = torch.where(k_text, (k <= q) & (qc - kc <= W), qc - kc > W)
    return torch.where(q_text, text, (qc == kc) & (k_text | (k <= q)))


class _Attention64(torch.autograd.Function):
    """``q`` ``[H, T, d]``, ``k, v`` ``[Hkv, T, d]`` (text then summary rows of one sequence), one block at a time."""

    BLOCK = 2048

    @staticmethod
    def _probs(q, k, h, r, lo, hi, keys):
        L, ns, C, S, W = keys
        z = (q[h, lo:hi] @ k[h // r].t()) / math.sqrt(q.shape[-1])
        return z.masked_fill_(~_mask(lo, hi, L, ns, C, S, W, q.device), -math.inf).softmax(-1)

    @staticmethod
    def forward(ctx, q, k, v, keys):
        ctx.save_for_backward(q, k, v)
        ctx.keys = keys
        o = torch.empty_like(q)
        r = q.shape[0] // k.shape[0]
        for h in range(q.shape[0]):
            for lo in range(0, q.shape[1], _Attention64.BLOCK):
                hi = min(q.shape[1], lo + _Attention64.BLOCK)
                o[h, lo:hi] = _Attention64._probs(q, k, h, r, lo, hi, keys) @ v[h // r]
        return o

    @staticmethod
    def backward(ctx, do):
        q, k, v = ctx.saved_tensors
        r, sc = q.shape[0] // k.shape[0], 1 / math.sqrt(q.shape[-1])
        dq, dk, dv = torch.empty_like(q), torch.zeros_like(k), torch.zeros_like(v)
        for h in range(q.shape[0]):
            for lo in range(0, q.shape[1], _Attention64.BLOCK):
                hi = min(q.shape[1], lo + _Attention64.BLOCK)
                p = _Attention64._probs(q, k, h, r, lo, hi, ctx.keys)
                g = do[h, lo:hi]
                dv[h // r] += p.t() @ g
                dp = g @ v[h // r].t()
                ds = p * (dp - (dp * p).sum(-1, keepdim=True)) * sc
                dq[h, lo:hi] = ds @ k[h // r]
                dk[h // r] += ds.t() @ q[h, lo:hi]
        return dq, dk, dv, None


def _attend(qkv, B, L, ns, cfg, window):
    """Packed rows (text rows of all sequences, then summary rows), rotated -> ``[rows, Hq * d]``."""
    H, Hk, d = cfg.num_heads, cfg.num_kv_heads, cfg.head_dim
    keys = (L, ns, cfg.summary_chunk_size, cfg.summary_token_num, window)
    texts, sums = [], []
    for b in range(B):
        rows = torch.cat([qkv[b * L:(b + 1) * L], qkv[B * L + b * ns:B * L + (b + 1) * ns]]).view(L + ns, H + 2 * Hk, d)
        rows = rows.transpose(0, 1)
        o = _Attention64.apply(rows[:H].contiguous(), rows[H:H + Hk].contiguous(), rows[H + Hk:].contiguous(), keys)
        o = o.transpose(0, 1).reshape(L + ns, H * d)
        texts.append(o[:L])
        sums.append(o[L:])
    return torch.cat(texts + sums)


def _swiglu64(h, w13, w2):
    g, u = (h @ w13.t()).chunk(2, -1)
    return (torch.nn.functional.silu(g) * u) @ w2.t()


def _layer64(p, x, delta, cfg, B, L, ns, pos, summary):
    H, Hk, d, eps = cfg.num_heads, cfg.num_kv_heads, cfg.head_dim, cfg.norm_eps
    x = x + torch.cat([delta, delta.new_zeros(x.shape[0] - delta.shape[0], x.shape[1])])
    h = _rms(x, p["sa_norm.scale"], eps)
    n = B * L
    ns = ns if summary else 0
    qkv = h[:n] @ p["attn.wqkv.weight"].t()
    if ns > 0:
        qkv = torch.cat([qkv, h[n:] @ p["attn.wqkv_summary.weight"].t()])
    heads = qkv.view(qkv.shape[0], H + 2 * Hk, d)
    q = _rope(_rms(heads[:, :H], p["attn.q_norm.scale"], eps), pos[:len(heads)], cfg.rope_base)
    k = _rope(_rms(heads[:, H:H + Hk], p["attn.k_norm.scale"], eps), pos[:len(heads)], cfg.rope_base)
    rot = torch.cat([q, k, heads[:, H + Hk:]], 1).reshape(qkv.shape)
    a = _attend(rot, B, L, ns, cfg, cfg.summary_sliding_chunk_num) @ p["attn.output_proj.weight"].t()
    x = x + torch.cat([a, a.new_zeros(x.shape[0] - a.shape[0], x.shape[1])])
    h = _rms(x, p["mlp_norm.scale"], eps)
    return x, _swiglu64(h[:len(a)], p["mlp.w13.weight"], p["mlp.w2.weight"])


def _params64(module, grad=False):
    return {k: v.detach().double().requires_grad_(grad) for k, v in module.named_parameters()}


def exact(case, seed):
    s = prepare(case, seed)
    kind = case["kind"]
    if kind == "proj":
        return s["x"].double() @ s["w"].double().t()
    if kind == "mlp":
        res = s["x"].double() + s["delta"].double()
        p = _params64(s["mlp"])
        return res, _swiglu64(_rms(res, s["norm"].double(), s["cfg"].norm_eps), p["w13.weight"], p["w2.weight"])
    if kind == "attn":
        return _attend(s["qkv"].double(), case["batch"], case["len"], s["Ns"], s["cfg"], s["cfg"].summary_sliding_chunk_num)
    if kind == "layer":
        with torch.no_grad():
            return _layer64(_params64(s["layer"]), s["x"].double(), s["delta"].double(), s["cfg"], case["batch"], case["len"],
                            s["meta"].Ns, s["meta"].pos, case["summary"])
    if kind == "train":
        p = _params64(s["layer"], True)
        x, delta = s["x"].double().requires_grad_(), s["delta"].double().requires_grad_()
        x2, out = _layer64(p, x, delta, s["cfg"], case["batch"], case["len"], s["meta"].Ns, s["meta"].pos, case["summary"])
        torch.autograd.backward([x2, out], [s["dx"].double(), s["dd"].double()])
        return {"x": x2.detach(), "out": out.detach(), "dx": x.grad, "ddelta": delta.grad,
                "weights": {k: v.grad for k, v in p.items() if v.grad is not None}}
    if kind == "head":
        w, h, labels = s["w"].detach().double(), s["h"].double(), s["labels"]
        valid = labels != -100
        n, loss = int(valid.sum()), 0.0
        dh, dw = torch.empty_like(h), torch.zeros_like(w)
        for lo in range(0, len(h), 512):
            sl = slice(lo, lo + 512)
            z = torch.log_softmax(h[sl] @ w.t(), -1)
            at, ok = labels[sl].clamp_min(0)[:, None], valid[sl][:, None].double()
            loss = loss - (z.gather(1, at) * ok).sum() / n
            g = z.exp_()
            g.scatter_add_(1, at, -torch.ones_like(ok))
            g *= ok / n
            dh[sl] = g @ w
            dw.addmm_(g.t(), h[sl])
        return {"loss": loss, "dh": dh, "dw": dw}
    if kind == "adamw":
        lr, bc1, bc2, scale = s["hyper"].double().tolist()
        g = s["grad"].double() * scale
        m = BETA1 * s["m"].double() + (1 - BETA1) * g
        v = BETA2 * s["v"].double() + (1 - BETA2) * g * g
        w = s["master"].double() * (1 - lr * DECAY) - lr * (m / bc1) / ((v / bc2).sqrt() + ADAM_EPS)
        return {"master": w, "m": m, "v": v, "bf16": w, "sumsq": (g * g).sum().reshape(1)}
    model, cfg, B, L, new = s["engine"].model, s["engine"].cfg, case["batch"], case["len"], case["new"]
    T = L + new
    p = _params64(model)
    C, S = cfg.summary_chunk_size, cfg.summary_token_num
    layout = ops.get_layout(T, C, S, cfg.summary_chunk_position_ids_type, cfg.summary_token_position_ids_type, True)
    meta = BatchMeta(B, T, layout, "cuda", False)
    ids = torch.cat([s["prompt"], s["next"].t()], 1)
    x = p["tok_embeddings.weight"][ids.reshape(-1)]
    x = torch.cat([x, p["summary_embedding.weight"].repeat(B * (meta.Ns // S), 1)])
    delta = torch.zeros_like(x)
    with torch.no_grad():
        for i, layer in enumerate(model.layers):
            own = {k[len(f"layers.{i}."):]: v for k, v in p.items() if k.startswith(f"layers.{i}.")}
            x, delta = _layer64(own, x, delta, cfg, B, T, meta.Ns, meta.pos, layer.is_summary_layer)
        h = _rms(x[:B * T] + delta[:B * T], p["norm.scale"], cfg.norm_eps).view(B, T, -1)[:, L - 1:]
        return (h @ p["output.weight"].t()).transpose(0, 1).contiguous()
