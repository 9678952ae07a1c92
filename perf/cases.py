"""Timed workloads: single layers and operators of training and serving through the public entry points, over the sizes
users run them at.

``listed()`` names twelve of them, ``draw(rng)`` makes one more of the same ranges, ``prepare`` builds what a program has in
hand before the call (inputs from the seed, weights, caches), ``run`` is one pass, ``work`` what a pass cannot do without,
``tolerance`` how far another correct implementation may be away, ``exact`` the same outputs in 64 bits.

Widths, heads and vocabularies are those of the model presets (``llmctl_b200.models.config.PRESETS``) and of the serving
benchmark's latent-attention model; a training micro-batch is 8 sequences of 512 tokens, as in ``bench.py``.
"""
import math

import torch

# (heads, head_dim, hidden, ffn) of the presets gpt-125m, gpt-1b, gpt-7b, gpt-13b
_SMALL, _MEDIUM, _LARGE, _XL = (12, 64, 768, 2048), (16, 128, 2048, 5632), (32, 128, 4096, 11008), (40, 128, 5120, 13824)
_VOCAB = 32000
# latent-attention layers of the serving benchmark: (width, heads, query rank); rank 512 + 64 rotated, 128 per head
_LATENT = ((2048, 16, 768), (4096, 32, 1536))
_R, _DR, _DN, _DV, _PAGE = 512, 64, 128, 128, 64


def listed():
    return [
        # causal attention, forward and backward, of a training step: the smallest preset (heads of 64), the default micro-batch
        # of the 7B preset, and the 13B plan's micro-batch of long sequences
        {"name": "attention_train_small", "kind": "attention", "batch": 8, "seq": 512, "heads": 12, "dim": 64, "grad": True},
        {"name": "attention_train", "kind": "attention", "batch": 8, "seq": 512, "heads": 32, "dim": 128, "grad": True},
        {"name": "attention_train_long", "kind": "attention", "batch": 2, "seq": 2048, "heads": 40, "dim": 128, "grad": True},
        # a served prompt: one sequence of any length, forward only
        {"name": "attention_prompt", "kind": "attention", "batch": 1, "seq": 1777, "heads": 32, "dim": 128, "grad": False},
        # a decoding step's cache append and attention: one short conversation, a full batch of long ones
        {"name": "decode_one", "kind": "decode", "batch": 1, "context": 300, "heads": 12, "dim": 64},
        {"name": "decode_batch", "kind": "decode", "batch": 16, "context": 4096, "heads": 32, "dim": 128},
        # one decoder layer of a training step, forward and backward (norms, projections, rotation, attention, SwiGLU)
        {"name": "block_train", "kind": "block", "batch": 8, "seq": 512, "heads": 16, "dim": 128, "hidden": 2048, "ffn": 5632},
        # output head and loss of a training step, forward and backward
        {"name": "head_loss", "kind": "head", "tokens": 4096, "hidden": 2048},
        # optimizer update of one layer of the 7B preset
        {"name": "optimizer", "kind": "adamw", "n": 202383360, "grad_bits": 16},
        # a whole small model over one prompt: logits
        {"name": "model_logits", "kind": "model", "seq": 777, "layers": 12},
        # latent-attention layer of a served model: two whole prompts; 32 decoding sequences
        {"name": "latent_prompt", "kind": "latent", "batch": 2, "tokens": 2048, "start": 0, "width": 2048, "heads": 16, "q_rank": 768},
        {"name": "latent_decode", "kind": "latent", "batch": 32, "tokens": 1, "start": 4000, "width": 2048, "heads": 16, "q_rank": 768},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _length(rng, lo, hi):
    """A sequence length: whole tiles of 128 for packed training batches, any number otherwise."""
    n = _log(rng, lo, hi)
    return max(128, n // 128 * 128) if rng.random() < 0.4 else n


def draw(rng):
    kind = rng.choice(["attention_train", "attention_train", "attention_train", "attention_prompt", "decode", "decode", "block", "head",
                       "adamw", "model", "latent_prompt", "latent_decode"])
    heads, dim, hidden, ffn = rng.choice([_SMALL, _MEDIUM, _LARGE, _XL])
    if kind == "attention_train":
        seq = _length(rng, 64, 2048)
        batch = min(rng.choice([1, 2, 4, 8]), max(1, 4096 // seq))
        return {"kind": "attention", "batch": batch, "seq": seq, "heads": heads, "dim": dim, "grad": True}
    if kind == "attention_prompt":
        return {"kind": "attention", "batch": 1, "seq": _log(rng, 20, 4000), "heads": heads, "dim": dim, "grad": False}
    if kind == "decode":
        return {"kind": "decode", "batch": _log(rng, 1, 16), "context": _log(rng, 60, 4096), "heads": min(heads, 32), "dim": dim}
    if kind == "block":
        seq = _length(rng, 64, 2048)
        heads, dim, hidden, ffn = rng.choice([_SMALL, _MEDIUM])
        return {"kind": "block", "batch": min(rng.choice([1, 2, 4, 8]), max(1, 4096 // seq)), "seq": seq, "heads": heads, "dim": dim,
                "hidden": hidden, "ffn": ffn}
    if kind == "head":
        return {"kind": "head", "tokens": _log(rng, 64, 4096), "hidden": rng.choice([768, 2048])}
    if kind == "adamw":
        return {"kind": "adamw", "n": _log(rng, 100000, 200000000), "grad_bits": rng.choice([16, 32])}
    if kind == "model":
        return {"kind": "model", "seq": _log(rng, 20, 2000), "layers": rng.choice([4, 8, 12])}
    width, heads, q_rank = rng.choice(_LATENT)
    if kind == "latent_prompt":
        tokens = _log(rng, 100, 2048)
        return {"kind": "latent", "batch": rng.choice([1, 2]) if width == 2048 else 1, "tokens": tokens,
                "start": rng.choice([0, 0, _log(rng, 16, 1000)]) if tokens < 1000 else 0, "width": width, "heads": heads, "q_rank": q_rank}
    return {"kind": "latent", "batch": _log(rng, 1, 32), "tokens": 1, "start": _log(rng, 60, 4000), "width": width, "heads": heads,
            "q_rank": q_rank}


# ---------------------------------------------------------------------------------------------------------------------
# inputs: made from the seed alone
# ---------------------------------------------------------------------------------------------------------------------
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _randn(g, *shape, std=1.0, dtype=torch.bfloat16):
    out = torch.empty(*shape, device="cuda", dtype=dtype)
    return out.normal_(0.0, std, generator=g)


def _lengths(case):
    """Context lengths of a decoding batch: the longest first, the others spread down to a quarter of it."""
    n, c = case["batch"], case["context"]
    return [max(1, c - (3 * c * i) // (4 * max(n, 2))) for i in range(n)]


def _tables(g, pages):
    """Block tables of sequences that own ``pages[i]`` pages each, scattered over the pool."""
    perm = torch.randperm(sum(pages), generator=g, device="cuda").tolist()
    out, at = [], 0
    for n in pages:
        out.append(perm[at:at + n])
        at += n
    return out


def _inputs(case, seed):
    g, k = _generator(seed), case["kind"]
    if k == "attention":
        B, S, H, D = case["batch"], case["seq"], case["heads"], case["dim"]
        s = {"qkv": _randn(g, B, S, 3, H, D)}
        if case["grad"]:
            s["do"] = _randn(g, B, S, H, D)
        return s
    if k == "decode":
        B, H, D, bs = case["batch"], case["heads"], case["dim"], 16
        lens = _lengths(case)
        pages = [(n + bs - 1) // bs for n in lens]
        tables = _tables(g, pages)
        bt = torch.zeros(B, max(pages), dtype=torch.int32)
        for i, t in enumerate(tables):
            bt[i, :len(t)] = torch.tensor(t, dtype=torch.int32)
        slots = [t[(n - 1) // bs] * bs + (n - 1) % bs for t, n in zip(tables, lens)]
        return {"qkv": _randn(g, B, 3 * H * D), "k": _randn(g, sum(pages), bs, H, D), "v": _randn(g, sum(pages), bs, H, D),
                "tables": bt.cuda(), "lens": torch.tensor(lens, dtype=torch.int32, device="cuda"),
                "slots": torch.tensor(slots, dtype=torch.int64, device="cuda")}
    if k in ("block", "model"):
        layers = case.get("layers", 1)
        H, D, W, F = (case["heads"], case["dim"], case["hidden"], case["ffn"]) if k == "block" else _SMALL
        ws = []
        for _ in range(layers):
            ws.append({"norm1.weight": 1 + _randn(g, W, std=0.1), "attn.qkv.weight": _randn(g, 3 * H * D, W, std=W ** -0.5),
                       "attn.out.weight": _randn(g, W, H * D, std=(H * D) ** -0.5), "norm2.weight": 1 + _randn(g, W, std=0.1),
                       "mlp.up.weight": _randn(g, 2 * F, W, std=W ** -0.5), "mlp.down.weight": _randn(g, W, F, std=F ** -0.5)})
        if k == "model":
            return {"layers": ws, "embed": _randn(g, _VOCAB, W), "norm": 1 + _randn(g, W, std=0.1), "head": _randn(g, _VOCAB, W, std=W ** -0.5),
                    "tokens": torch.randint(0, _VOCAB, (1, case["seq"]), generator=g, device="cuda")}
        T = case["batch"] * case["seq"]
        return {"layers": ws, "x": _randn(g, T, W), "residual": _randn(g, T, W), "dy": _randn(g, T, W), "dres": _randn(g, T, W)}
    if k == "head":
        T, W = case["tokens"], case["hidden"]
        t = torch.randint(0, _VOCAB, (T,), generator=g, device="cuda")
        t[torch.rand(T, generator=g, device="cuda") < 0.05] = -100          # padding of a training batch
        t[0] = 7
        return {"x": _randn(g, T, W), "w": _randn(g, _VOCAB, W, std=W ** -0.5), "t": t}
    if k == "adamw":
        n = case["n"]
        f32 = torch.float32
        s = {"master": _randn(g, n, std=0.02, dtype=f32), "m": _randn(g, n, std=1e-3, dtype=f32),
             "v": torch.rand(n, generator=g, device="cuda").mul_(1e-5).add_(1e-7),
             "grad": _randn(g, n, std=1e-3, dtype=torch.bfloat16 if case["grad_bits"] == 16 else f32),
             "scale": torch.tensor([0.8], device="cuda")}
        return s
    if k == "latent":
        B, n, W, H, Q = case["batch"], case["tokens"], case["width"], case["heads"], case["q_rank"]
        starts = [case["start"] if n > 1 else max(0, case["start"] - (case["start"] * i) // (2 * B)) for i in range(B)]
        tables = _tables(g, [(s + n + _PAGE - 1) // _PAGE for s in starts])
        cache = _randn(g, sum(len(t) for t in tables), _PAGE, _R + _DR)
        return {"h": _randn(g, B * n, W), "cache": cache, "tables": tables, "starts": starts,
                "w_down": _randn(g, Q + _R + _DR, W, std=W ** -0.5), "q_norm": 1 + _randn(g, Q, std=0.1), "kv_norm": 1 + _randn(g, _R, std=0.1),
                "w_uq": _randn(g, H * (_DN + _DR), Q, std=Q ** -0.5), "w_uk": _randn(g, H, _DN, _R, std=_R ** -0.5),
                "w_uv": _randn(g, H, _DV, _R, std=_R ** -0.5), "w_o": _randn(g, W, H * _DV, std=(H * _DV) ** -0.5)}
    raise ValueError(k)


def _fill(module, tensors):
    with torch.no_grad():
        for name, p in module.named_parameters():
            p.copy_(tensors[name])


def prepare(case, seed):
    s, k = _inputs(case, seed), case["kind"]
    s["case"] = case
    if k == "attention":
        # q, k and v are column blocks of one packed projection, as a decoder layer has them
        s["q"], s["k"], s["v"] = (s["qkv"][:, :, i].detach().requires_grad_(case["grad"]) for i in range(3))
    elif k == "decode":
        # the engine rounds the longest context up to a power of two, the size its decoding step is captured at
        s["bound"] = 256
        while s["bound"] < case["context"]:
            s["bound"] *= 2
    elif k in ("block", "model"):
        from llmctl_b200.models.config import ModelConfig
        from llmctl_b200.models.gpt import GPTModel
        H, D, W, F = (case["heads"], case["dim"], case["hidden"], case["ffn"]) if k == "block" else _SMALL
        cfg = ModelConfig(name="timed", layers=len(s["layers"]), hidden=W, ffn=F, heads=H, head_dim=D, vocab_size=_VOCAB if k == "model" else 128,
                          max_position_embeddings=2048)
        m = GPTModel(cfg, device="cuda")
        for blk, w in zip(m.blocks, s["layers"]):
            _fill(blk, w)
        s["cos"], s["sin"] = m.rope_tables(torch.device("cuda"))
        if k == "model":
            with torch.no_grad():
                m.embed.weight.copy_(s["embed"])
                m.final_norm.weight.copy_(s["norm"])
                m.lm_head.weight.copy_(s["head"])
            s["model"] = m.eval()
        else:
            s["block"] = m.blocks[0]
            s["x"].requires_grad_(True)
            s["residual"].requires_grad_(True)
        del s["layers"]
    elif k == "head":
        s["x"].requires_grad_(True)
        s["w"].requires_grad_(True)
    elif k == "adamw":
        s["param"] = torch.empty(case["n"], device="cuda", dtype=torch.bfloat16)
    elif k == "latent":
        from llmctl_b200.models.mixers import LatentAttention, LatentAttentionSpec
        from llmctl_b200.serve.ragged import Portion, RaggedBatch
        n = case["tokens"]
        spec = LatentAttentionSpec(heads=case["heads"], dim=_DN, rot_dim=_DR, vdim=_DV, kv_rank=_R, q_rank=case["q_rank"],
                                   scale=(_DN + _DR) ** -0.5, rot_base=10000.0)
        layer = LatentAttention(case["width"], spec, 1e-5, torch.bfloat16, "cuda")
        _fill(layer, s)
        s["layer"] = layer
        s["batch"] = RaggedBatch([Portion(i, [1] * n, st, [n - 1], tb) for i, (st, tb) in enumerate(zip(s["starts"], s["tables"]))], _PAGE,
                                 torch.device("cuda"))
    return s


def run(s):
    from llmctl_b200.ops import functional as ops
    case = s["case"]
    k = case["kind"]
    if k == "attention":
        if not case["grad"]:
            with torch.no_grad():
                return ops.attention(s["q"], s["k"], s["v"], causal=True)
        o = ops.attention(s["q"], s["k"], s["v"], causal=True)
        return (o.detach(), *torch.autograd.grad(o, (s["q"], s["k"], s["v"]), s["do"]))
    if k == "decode":
        from llmctl_b200.ops import serving
        B, H, D = case["batch"], case["heads"], case["dim"]
        serving.kv_append(s["qkv"], s["k"], s["v"], s["slots"], H, D)
        o = serving.paged_attention_decode(s["qkv"][:, :H * D].reshape(B, H, D), s["k"], s["v"], s["tables"], s["lens"], s["bound"])
        return o, s["k"], s["v"]
    if k == "block":
        blk = s["block"]
        y, r = blk(s["x"], s["residual"], s["cos"], s["sin"], case["batch"], case["seq"])
        params = [blk.norm1.weight, blk.attn.qkv.weight, blk.attn.out.weight, blk.norm2.weight, blk.mlp.up.weight, blk.mlp.down.weight]
        return (y.detach(), r.detach(), *torch.autograd.grad((y, r), [s["x"], s["residual"]] + params, (s["dy"], s["dres"])))
    if k == "model":
        with torch.no_grad():
            return s["model"](s["tokens"])
    if k == "head":
        loss = ops.cross_entropy(ops.linear(s["x"], s["w"]), s["t"], assume_unit_grad=True)
        return (loss.detach(), *torch.autograd.grad(loss, (s["x"], s["w"])))
    if k == "adamw":
        from llmctl_b200.ops import optim
        optim.adamw_step(s["master"], s["m"], s["v"], s["grad"], s["param"], step=10, lr=2e-4, beta1=0.9, beta2=0.95, eps=1e-8,
                         weight_decay=0.1, scale_dev=s["scale"])
        return s["master"], s["m"], s["v"], s["param"]
    with torch.no_grad():
        return s["layer"](s["h"], s["batch"], s["cache"]), s["cache"]


# ---------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------------------------------
def _attention_flops(S, H, D, grad):
    return (14 if grad else 4) * H * D * S * (S + 1) / 2        # 2 products forward, 5 backward, over the visible pairs


def work(case):
    k = case["kind"]
    if k == "attention":
        B, S, H, D = case["batch"], case["seq"], case["heads"], case["dim"]
        return {"bytes": 2.0 * B * S * H * D * (8 if case["grad"] else 4), "flops": B * _attention_flops(S, H, D, case["grad"])}
    if k == "decode":
        n, w = sum(_lengths(case)), case["heads"] * case["dim"]
        return {"bytes": 4.0 * n * w + 12.0 * case["batch"] * w, "flops": 4.0 * n * w}
    if k == "block":
        T, W, a = case["batch"] * case["seq"], case["hidden"], case["heads"] * case["dim"]
        p = 4 * W * a + 3 * W * case["ffn"]
        return {"bytes": 2.0 * (2 * p + 8 * T * W), "flops": 6.0 * T * p + case["batch"] * _attention_flops(case["seq"], case["heads"], case["dim"], True)}
    if k == "model":
        H, D, W, F = _SMALL
        p, S = case["layers"] * (4 * W * H * D + 3 * W * F) + W * _VOCAB, case["seq"]
        return {"bytes": 2.0 * (p + S * _VOCAB), "flops": 2.0 * S * p + case["layers"] * _attention_flops(S, H, D, False)}
    if k == "head":
        T, W = case["tokens"], case["hidden"]
        return {"bytes": 4.0 * (T * W + _VOCAB * W), "flops": 6.0 * T * W * _VOCAB}
    if k == "adamw":
        return {"bytes": (24.0 + 2 + case["grad_bits"] / 8) * case["n"], "flops": 12.0 * case["n"]}
    B, n, W, H, Q = case["batch"], case["tokens"], case["width"], case["heads"], case["q_rank"]
    starts = [case["start"] if n > 1 else max(0, case["start"] - (case["start"] * i) // (2 * B)) for i in range(B)]
    pairs = sum(n * s + n * (n + 1) / 2 for s in starts)
    T = B * n
    p = W * (Q + _R + _DR) + Q * H * (_DN + _DR) + H * _R * (_DN + _DV) + W * H * _DV
    return {"bytes": 2.0 * (p + 2 * T * W + (sum(starts) + T) * (_R + _DR)), "flops": 2.0 * T * p + 2.0 * pairs * H * (2 * _R + _DR)}


def tolerance(case):
    """About four times the distance from 64 bits that rounding to the activation type at the present places shows."""
    return {"attention": {"rel": 1e-2}, "decode": {"rel": 7e-3}, "block": {"rel": 3e-2}, "model": {"rel": 5e-2}, "head": {"rel": 1e-2},
            "adamw": {"rel": 5e-5}, "latent": {"rel": 2e-2}}[case["kind"]]


# ---------------------------------------------------------------------------------------------------------------------
# the same outputs in 64 bits
# ---------------------------------------------------------------------------------------------------------------------
def _attend(q, k, v, scale):
    """Causal attention of [S, D] tensors."""
    s = (q @ k.t()) * scale
    s = s.masked_fill(torch.ones_like(s, dtype=torch.bool).triu(1), float("-inf"))
    return torch.softmax(s, -1) @ v


def _attend_heads(q, k, v):
    """[B, S, H, D] each; one head at a time."""
    B, S, H, D = q.shape
    return torch.stack([torch.stack([_attend(q[b, :, h], k[b, :, h], v[b, :, h], D ** -0.5) for h in range(H)], 1) for b in range(B)])


def _norm(x, w):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + 1e-5) * w


def _rotate(x, S):
    """[B, S, H, D] by halves, base 10000."""
    D = x.shape[-1]
    f = 10000.0 ** (-torch.arange(0, D // 2, dtype=torch.float64, device=x.device) * 2 / D)
    a = torch.outer(torch.arange(S, dtype=torch.float64, device=x.device), f)
    c, s = a.cos()[None, :, None], a.sin()[None, :, None]
    u, v = x.chunk(2, -1)
    return torch.cat([u * c - v * s, v * c + u * s], -1)


def _layer(x, residual, w, B, S, H, D):
    r = x if residual is None else x + residual
    qkv = (_norm(r, w["norm1.weight"]) @ w["attn.qkv.weight"].t()).view(B, S, 3, H, D)
    o = _attend_heads(_rotate(qkv[:, :, 0], S), _rotate(qkv[:, :, 1], S), qkv[:, :, 2]).reshape(B * S, H * D)
    r = r + o @ w["attn.out.weight"].t()
    gate, up = (_norm(r, w["norm2.weight"]) @ w["mlp.up.weight"].t()).chunk(2, -1)
    return (torch.nn.functional.silu(gate) * up) @ w["mlp.down.weight"].t(), r


def exact(case, seed):
    s, k, f64 = _inputs(case, seed), case["kind"], torch.float64
    if k == "attention":
        q, kk, v = (s["qkv"][:, :, i].to(f64) for i in range(3))
        if not case["grad"]:
            return _attend_heads(q, kk, v)
        outs = [torch.empty_like(q) for _ in range(4)]
        for b in range(case["batch"]):
            for h in range(case["heads"]):
                leaf = [t[b, :, h].clone().requires_grad_(True) for t in (q, kk, v)]
                o = _attend(*leaf, case["dim"] ** -0.5)
                for out, val in zip(outs, (o.detach(), *torch.autograd.grad(o, leaf, s["do"][b, :, h].to(f64)))):
                    out[b, :, h] = val
        return tuple(outs)
    if k == "decode":
        H, D, bs = case["heads"], case["dim"], 16
        q, kn, vn = s["qkv"].view(-1, 3, H, D).unbind(1)
        s["k"].view(-1, H, D)[s["slots"]] = kn
        s["v"].view(-1, H, D)[s["slots"]] = vn
        out = torch.empty(q.shape, dtype=f64, device="cuda")
        for i, n in enumerate(_lengths(case)):
            pages = s["tables"][i, :(n + bs - 1) // bs].long()
            kk, vv = (t[pages].reshape(-1, H, D)[:n].to(f64) for t in (s["k"], s["v"]))
            p = torch.softmax(torch.einsum("hd,nhd->hn", q[i].to(f64), kk) * D ** -0.5, -1)
            out[i] = torch.einsum("hn,nhd->hd", p, vv)
        return out, s["k"], s["v"]
    if k == "block":
        w = {n: t.to(f64).requires_grad_(True) for n, t in s["layers"][0].items()}
        x, r0 = (s[n].to(f64).requires_grad_(True) for n in ("x", "residual"))
        y, r = _layer(x, r0, w, case["batch"], case["seq"], case["heads"], case["dim"])
        names = ["norm1.weight", "attn.qkv.weight", "attn.out.weight", "norm2.weight", "mlp.up.weight", "mlp.down.weight"]
        return (y.detach(), r.detach(), *torch.autograd.grad((y, r), [x, r0] + [w[n] for n in names], (s["dy"].to(f64), s["dres"].to(f64))))
    if k == "model":
        H, D, W, _ = _SMALL
        with torch.no_grad():
            x, r = s["embed"].to(f64)[s["tokens"][0]], None
            for w in s["layers"]:
                x, r = _layer(x, r, {n: t.to(f64) for n, t in w.items()}, 1, case["seq"], H, D)
            return _norm(x + r, s["norm"].to(f64)) @ s["head"].to(f64).t()
    if k == "head":
        x, w = s["x"].to(f64).requires_grad_(True), s["w"].to(f64).requires_grad_(True)
        loss = torch.nn.functional.cross_entropy(x @ w.t(), s["t"])
        return (loss.detach(), *torch.autograd.grad(loss, (x, w)))
    if k == "adamw":
        b1, b2, lr = 0.9, 0.95, 2e-4
        g = s["grad"].to(f64) * s["scale"].to(f64)
        m = s["m"].to(f64) * b1 + (1 - b1) * g
        v = s["v"].to(f64) * b2 + (1 - b2) * g * g
        p = s["master"].to(f64) * (1 - lr * 0.1) - lr * (m / (1 - b1 ** 10)) / ((v / (1 - b2 ** 10)).sqrt() + 1e-8)
        return p, m, v, p
    B, n, H, Q = case["batch"], case["tokens"], case["heads"], case["q_rank"]
    w = {name: t.to(f64) for name, t in s.items() if isinstance(t, torch.Tensor) and name != "cache"}
    d = w["h"] @ w["w_down"].t()

    def rotate(x, pos):
        f = 10000.0 ** (-torch.arange(0, _DR // 2, dtype=torch.float64, device="cuda") * 2 / _DR)
        a = torch.outer(pos.to(f64), f)
        c, sn = a.cos(), a.sin()
        if x.dim() == 3:
            c, sn = c[:, None], sn[:, None]
        u, v = x[..., 0::2], x[..., 1::2]
        return torch.stack([u * c - v * sn, v * c + u * sn], -1).flatten(-2)
    q = (_norm(d[:, :Q], w["q_norm"]) @ w["w_uq"].t()).view(B * n, H, _DN + _DR)
    out = torch.empty(B * n, H, _DV, dtype=f64, device="cuda")
    cache = s["cache"].to(f64)
    for i in range(B):
        rows = slice(i * n, (i + 1) * n)
        at = torch.arange(s["starts"][i], s["starts"][i] + n, device="cuda")
        table = torch.tensor(s["tables"][i], device="cuda")
        slots = table[torch.arange(s["starts"][i] + n, device="cuda") // _PAGE] * _PAGE + torch.arange(s["starts"][i] + n, device="cuda") % _PAGE
        cache.view(-1, _R + _DR)[slots[at]] = torch.cat([_norm(d[rows, Q:Q + _R], w["kv_norm"]), rotate(d[rows, Q + _R:], at)], -1)
        kv = cache.view(-1, _R + _DR)[slots]
        qr = rotate(q[rows, :, _DN:], at)
        dark = torch.arange(len(slots), device="cuda")[None, :] > at[:, None]
        for h in range(H):
            ql = q[rows, h, :_DN] @ w["w_uk"][h]
            sc = (ql @ kv[:, :_R].t() + qr[:, h] @ kv[:, _R:].t()) * (_DN + _DR) ** -0.5
            out[rows, h] = torch.softmax(sc.masked_fill(dark, float("-inf")), -1) @ kv[:, :_R] @ w["w_uv"][h].t()
    return out.reshape(B * n, H * _DV) @ w["w_o"].t(), cache
