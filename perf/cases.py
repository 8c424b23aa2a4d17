"""Performance cases of nabla_b200 on one GPU.

Each case is one layer, block or step as a user's program runs it: the function is compiled once
with ``nb.compile`` (launch-bound chains of small kernels with ``cuda_graph=True``) and called again
with the inputs at hand. Sizes come from the training
configurations in ``nabla_b200/models`` (d_model 2048, 16 heads of 128, d_ff 8192, vocabulary 32000,
sequences of 2048; the 64-256-256-256-1 MLP; rank-16 LoRA) and their smaller relatives; ragged
sequence lengths, odd row counts and narrow widths stand beside the round ones.

``listed()`` gives the fixed cases, ``draw(rng)`` others of the same ranges, ``prepare`` the inputs
on the GPU, ``run`` one pass, ``work`` the bytes and operations it cannot do without, and ``exact``
the same outputs from plain torch in 64 bits.
"""
from __future__ import annotations

import functools
import math

import torch
import torch.nn.functional as TF

import nabla_b200 as nb
from nabla_b200 import nn
from nabla_b200.models import transformer as T
from nabla_b200.nn import functional as F
from nabla_b200.nn.finetune.qlora import qlora_linear
from nabla_b200.ops import fused

BF16, F32, F64 = torch.bfloat16, torch.float32, torch.float64
LAYER = ("ln1_g", "ln1_b", "wqkv", "bqkv", "wo", "bo", "ln2_g", "ln2_b", "w1", "b1", "w2", "b2")


# ---------------------------------------------------------------------------------------- inputs
class _Source:
    """Tensors of one seed, drawn on the GPU."""

    def __init__(self, seed: int):
        self.g = torch.Generator("cuda").manual_seed(int(seed))

    def normal(self, shape, std=1.0, mean=0.0, dtype=BF16):
        return (torch.randn(shape, generator=self.g, device="cuda") * std + mean).to(dtype)

    def uniform(self, shape, low, high, dtype=BF16):
        return (torch.rand(shape, generator=self.g, device="cuda") * (high - low) + low).to(dtype)

    def integers(self, shape, high):
        return torch.randint(0, high, shape, generator=self.g, device="cuda")

    def tokens(self, shape, vocab):
        """Token ids with the skew of text: the id of rank r turns up about 1 / r as often as the first."""
        u = torch.rand(shape, generator=self.g, device="cuda", dtype=F64)
        return (torch.exp(u * math.log(vocab + 1.0)) - 1.0).long().clamp_(0, vocab - 1)


def _dtype(case):
    return F32 if case.get("dtype") == "fp32" else BF16


def _size(case):
    return 4 if case.get("dtype") == "fp32" else 2


def _log_int(rng, low, high):
    """An integer spread over the logarithm of [low, high]."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _grads(f, primals, cot):
    """Outputs of ``f`` and the gradients of all its primals for one cotangent."""
    y, pull = nb.vjp(f, *primals, create_graph=False)
    return (y, *pull(cot))


def _grads64(f, primals, cot):
    ps = [p.to(F64).requires_grad_(True) for p in primals]
    y = f(*ps)
    return [y.detach()] + list(torch.autograd.grad(y, ps, cot.to(F64)))


# ---------------------------------------------------------------------------------- attention
# The self-attention of a training step on the packed projection (batch, seq, heads * 3 * head_dim).
@functools.lru_cache(None)
def _attn_train(head_dim):
    return nb.compile(lambda qkv, do: _grads(lambda t: fused.packed_self_attention(t, head_dim, causal=True), (qkv,), do))


def _attn_train_inputs(c, s):
    w = c["heads"] * c["head_dim"]
    return [s.normal((c["batch"], c["seq"], 3 * w)), s.normal((c["batch"], c["seq"], w))]


def _attend64(q, k, v, causal, mask=None):
    """One (batch, head) pair at a time: the scores in 64 bits of all of them would not fit."""
    out = []
    for i in range(q.shape[0]):
        rows = []
        for h in range(q.shape[1]):
            sc = q[i, h] @ k[i, h].T / math.sqrt(q.shape[-1])
            if causal:
                keep = torch.ones(sc.shape, dtype=torch.bool, device="cuda").tril(sc.shape[1] - sc.shape[0])
                sc = sc.masked_fill(~keep, float("-inf"))
            if mask is not None:
                sc = sc + mask[i, 0]
            rows.append(torch.softmax(sc, -1) @ v[i, h])
        out.append(torch.stack(rows))
    return torch.stack(out)


def _attn_train_exact(c, qkv, do):
    b, n, h, d = c["batch"], c["seq"], c["heads"], c["head_dim"]
    y, g = [], []
    for i in range(b):                      # per example, so that autograd keeps one example's scores
        r = _grads64(lambda t: _attend64(*(t.view(1, n, h, 3, d)[:, :, :, j].transpose(1, 2) for j in range(3)), True)
                     .transpose(1, 2).reshape(1, n, h * d), (qkv[i:i + 1],), do[i:i + 1])
        y.append(r[0])
        g.append(r[1])
    return [torch.cat(y), torch.cat(g)]


def _attn_train_work(c):
    t, w = c["batch"] * c["seq"], c["heads"] * c["head_dim"]
    # QK^T and PV forward, five products backward, the visible half of each
    return {"bytes": t * w * 2 * (3 + 1 + 1 + 3), "flops": 7 * c["batch"] * c["seq"] * c["seq"] * w}


# Attention of a padded batch: separate q, k, v (batch, heads, seq, head_dim) and an additive mask that
# hides the padding keys of each example.
@functools.lru_cache(None)
def _attn_padded():
    return nb.compile(lambda q, k, v, m, do: _grads(lambda a, b, c: F.scaled_dot_product_attention(a, b, c, attn_mask=m), (q, k, v), do))


def _attn_padded_inputs(c, s):
    shape = (c["batch"], c["heads"], c["seq"], c["head_dim"])
    length = s.integers((c["batch"],), max(1, c["seq"] // 2)) + (c["seq"] + 1) // 2
    mask = (torch.arange(c["seq"], device="cuda")[None] >= length[:, None]).float() * -1e9
    return [s.normal(shape), s.normal(shape), s.normal(shape), mask[:, None, None, :].contiguous(), s.normal(shape)]


def _attn_padded_exact(c, q, k, v, m, do):
    parts = [_grads64(lambda a, b, e: _attend64(a, b, e, False, m[i:i + 1].to(F64)), (q[i:i + 1], k[i:i + 1], v[i:i + 1]), do[i:i + 1])
             for i in range(c["batch"])]
    return [torch.cat(p) for p in zip(*parts)]


def _attn_padded_work(c):
    n = c["batch"] * c["heads"] * c["seq"] * c["head_dim"]
    return {"bytes": n * 2 * 8 + c["batch"] * c["seq"] * 4, "flops": 14 * n * c["seq"]}


# A few new queries against the keys and values of a long prefix, forward only (inference).
@functools.lru_cache(None)
def _attn_prefix():
    return nb.compile(lambda q, k, v: F.scaled_dot_product_attention(q, k, v, is_causal=True))


def _attn_prefix_inputs(c, s):
    b, h, d = c["batch"], c["heads"], c["head_dim"]
    return [s.normal((b, h, c["new"], d)), s.normal((b, h, c["prefix"], d)), s.normal((b, h, c["prefix"], d))]


def _attn_prefix_exact(c, q, k, v):
    return _attend64(q.to(F64), k.to(F64), v.to(F64), True)


def _attn_prefix_work(c):
    bhd = c["batch"] * c["heads"] * c["head_dim"]
    return {"bytes": bhd * 2 * (2 * c["prefix"] + 2 * c["new"]), "flops": 4 * bhd * c["new"] * c["prefix"]}


# ------------------------------------------------------------------------------------- layer norm
@functools.lru_cache(None)
def _norm():
    return nb.compile(lambda x, g, b, dy: _grads(lambda *a: F.layer_norm(*a), (x, g, b), dy))


def _norm_inputs(c, s):
    dt, d = _dtype(c), c["dim"]
    return [s.normal((c["rows"], d), 1.0, 0.1, dt), s.normal((d,), 0.1, 1.0, dt), s.normal((d,), 0.1, 0.0, dt),
            s.normal((c["rows"], d), 1.0, 0.0, dt)]


def _norm_exact(c, x, g, b, dy):
    return _grads64(lambda t, u, v: TF.layer_norm(t, (c["dim"],), u, v, 1e-5), (x, g, b), dy)


def _norm_work(c):
    return {"bytes": 5 * c["rows"] * c["dim"] * _size(c), "flops": 0}


# ------------------------------------------------------------------------------------ feed-forward
@functools.lru_cache(None)
def _mlp():
    def layer(x, w1, b1, w2, b2):
        return F.linear(F.linear(x, w1, b1, activation="gelu"), w2, b2)

    return nb.compile(lambda x, w1, b1, w2, b2, dy: _grads(layer, (x, w1, b1, w2, b2), dy))


def _mlp_inputs(c, s):
    t, d, f = c["tokens"], c["dim"], c["hidden"]
    return [s.normal((t, d)), s.normal((d, f), d ** -0.5), s.normal((f,), 0.02), s.normal((f, d), f ** -0.5),
            s.normal((d,), 0.02), s.normal((t, d))]


def _mlp_exact(c, x, w1, b1, w2, b2, dy):
    return _grads64(lambda t, u, v, y, z: TF.gelu(t @ u + v) @ y + z, (x, w1, b1, w2, b2), dy)


def _mlp_work(c):
    t, d, f = c["tokens"], c["dim"], c["hidden"]
    return {"bytes": 2 * (4 * t * d + 4 * d * f), "flops": 12 * t * d * f}


# ----------------------------------------------------------------------------- transformer block
def _layer_inputs(s, d, f):
    std = 0.02
    shapes = {"wqkv": (d, 3 * d), "bqkv": (3 * d,), "wo": (d, d), "bo": (d,), "w1": (d, f), "b1": (f,), "w2": (f, d), "b2": (d,)}
    p = {k: s.normal(v, max(std, v[0] ** -0.5) if len(v) == 2 else std) for k, v in shapes.items()}
    for i in ("1", "2"):
        p[f"ln{i}_g"], p[f"ln{i}_b"] = s.normal((d,), 0.1, 1.0), s.normal((d,), 0.1)
    return [p[k] for k in LAYER]


@functools.lru_cache(None)
def _block(dim, heads, hidden):
    cfg = T.TransformerConfig(n_layers=1, d_model=dim, n_heads=heads, d_ff=hidden)
    return nb.compile(lambda x, dy, *p: _grads(lambda t, *q: T.block(t, dict(zip(LAYER, q)), cfg), (x, *p), dy), cuda_graph=True)


def _block_inputs(c, s):
    d = c["heads"] * c["head_dim"]
    shape = (c["batch"], c["seq"], d)
    return [s.normal(shape), s.normal(shape)] + _layer_inputs(s, d, c["hidden"])


def _block64(x, p, heads):
    b, n, d = x.shape
    qkv = (TF.layer_norm(x, (d,), p["ln1_g"], p["ln1_b"]) @ p["wqkv"] + p["bqkv"]).view(b, n, heads, 3, d // heads)
    q, k, v = (qkv[:, :, :, i].transpose(1, 2) for i in range(3))
    x = x + _attend64(q, k, v, True).transpose(1, 2).reshape(b, n, d) @ p["wo"] + p["bo"]
    return x + TF.gelu(TF.layer_norm(x, (d,), p["ln2_g"], p["ln2_b"]) @ p["w1"] + p["b1"]) @ p["w2"] + p["b2"]


def _block_exact(c, x, dy, *p):
    return _grads64(lambda t, *q: _block64(t, dict(zip(LAYER, q)), c["heads"]), (x, *p), dy)


def _block_work(c):
    t, d, f = c["batch"] * c["seq"], c["heads"] * c["head_dim"], c["hidden"]
    return {"bytes": 2 * (4 * t * d + 2 * (4 * d * d + 2 * d * f)), "flops": 6 * t * (4 * d * d + 2 * d * f) + 7 * t * c["seq"] * d}


# ----------------------------------------------------------------------------- head and embedding
# Projection to the vocabulary and the mean cross-entropy, with the gradients of both operands.
@functools.lru_cache(None)
def _head():
    def loss(x, w, t):
        return F.cross_entropy_loss(F.linear(x, w), t)

    return nb.compile(lambda x, w, t: nb.value_and_grad(loss, argnums=(0, 1), create_graph=False)(x, w, t))


def _head_inputs(c, s):
    t, d, v = c["tokens"], c["dim"], c["vocab"]
    return [s.normal((t, d)), s.normal((d, v), d ** -0.5), s.tokens((t,), v)]


def _head_exact(c, x, w, t):
    x, w = x.to(F64).requires_grad_(True), w.to(F64).requires_grad_(True)
    loss = TF.cross_entropy(x @ w, t)
    return [loss.detach(), list(torch.autograd.grad(loss, (x, w)))]


def _head_work(c):
    t, d, v = c["tokens"], c["dim"], c["vocab"]
    return {"bytes": 2 * (2 * t * d + 2 * d * v) + 8 * t, "flops": 6 * t * d * v}


# Token plus position embedding of a batch and the gradients of both tables.
@functools.lru_cache(None)
def _embed():
    def look_up(table, pos, ids):
        return F.embedding(ids, table) + pos

    return nb.compile(lambda table, pos, ids, dy: _grads(lambda a, b: look_up(a, b, ids), (table, pos), dy))


def _embed_inputs(c, s):
    dt, d = _dtype(c), c["dim"]
    return [s.normal((c["vocab"], d), 0.02, 0.0, dt), s.normal((c["seq"], d), 0.02, 0.0, dt),
            s.tokens((c["batch"], c["seq"]), c["vocab"]), s.normal((c["batch"], c["seq"], d), 1.0, 0.0, dt)]


def _embed_exact(c, table, pos, ids, dy):
    return _grads64(lambda a, b: a[ids] + b, (table, pos), dy)


def _embed_work(c):
    t, d = c["batch"] * c["seq"], c["dim"]
    rows = min(t, c["vocab"])
    return {"bytes": _size(c) * d * (rows + 2 * t + 2 * c["seq"] + c["vocab"]) + 8 * t, "flops": 0}


# ---------------------------------------------------------------------------- convolutional network
# Training step of a small image classifier in fp32: two 3x3 convolutions with relu and 2x2 max pooling,
# then a linear layer. Gradients of every weight.
@functools.lru_cache(None)
def _cnn():
    def loss(w1, b1, w2, b2, w3, b3, x, t):
        h = nb.max_pool2d(nb.relu(nb.conv2d(x, w1, bias=b1, padding=1)), 2)
        h = nb.max_pool2d(nb.relu(nb.conv2d(h, w2, bias=b2, padding=1)), 2)
        return F.cross_entropy_loss(F.linear(nb.reshape(h, (int(h.shape[0]), -1)), w3, b3), t)

    return nb.compile(lambda *a: nb.value_and_grad(loss, argnums=tuple(range(6)), create_graph=False)(*a), cuda_graph=True)


def _cnn_inputs(c, s):
    dt, n, e, k = _dtype(c), c["batch"], c["edge"], c["channels"]
    flat = (e // 4) ** 2 * 2 * k
    return [s.normal((3, 3, c["planes"], k), (9 * c["planes"]) ** -0.5, 0.0, dt), s.normal((k,), 0.02, 0.0, dt),
            s.normal((3, 3, k, 2 * k), (9 * k) ** -0.5, 0.0, dt), s.normal((2 * k,), 0.02, 0.0, dt),
            s.normal((flat, c["classes"]), flat ** -0.5, 0.0, dt), s.normal((c["classes"],), 0.02, 0.0, dt),
            s.uniform((n, e, e, c["planes"]), 0.0, 1.0, dt), s.integers((n,), c["classes"])]


def _cnn_exact(c, w1, b1, w2, b2, w3, b3, x, t):
    ps = [p.to(F64).requires_grad_(True) for p in (w1, b1, w2, b2, w3, b3)]
    h = x.to(F64).permute(0, 3, 1, 2)
    for w, b in ((ps[0], ps[1]), (ps[2], ps[3])):
        h = TF.pad(h, (1, 1, 1, 1)).unfold(2, 3, 1).unfold(3, 3, 1)
        h = TF.max_pool2d(torch.relu(torch.einsum("nchwrs,rscf->nfhw", h, w) + b[:, None, None]), 2)
    loss = TF.cross_entropy(h.permute(0, 2, 3, 1).reshape(h.shape[0], -1) @ ps[4] + ps[5], t)
    return [loss.detach(), list(torch.autograd.grad(loss, ps))]


def _cnn_work(c):
    n, e, k, p = c["batch"], c["edge"], c["channels"], c["planes"]
    first, second = n * e * e * 9 * p * k, n * (e // 2) ** 2 * 9 * k * 2 * k
    return {"bytes": _size(c) * n * e * e * p, "flops": 2 * (2 * first + 3 * second)}


# ------------------------------------------------------------------------------------------ QLoRA
# Linear layer over a frozen NF4 weight with a LoRA adapter: output and the gradients of x, A and B.
@functools.lru_cache(None)
def _qlora(dim, out, block):
    def layer(x, a, b, codes, scales):
        q = {"indices": codes, "scales": scales, "original_shape": (dim, out), "original_numel": dim * out,
             "padded_numel": dim * out, "block_size": block}
        return qlora_linear(x, q, {"A": a, "B": b}, alpha=16.0, compute_dtype=nb.DType.bfloat16)

    return nb.compile(lambda x, a, b, codes, scales, dy: _grads(lambda *p: layer(*p, codes, scales), (x, a, b), dy), cuda_graph=True)


def _qlora_inputs(c, s):
    t, d, o, r = c["tokens"], c["dim"], c["out"], c["rank"]
    codes = s.normal((d * o,), 2.6, 7.5, F32).round().clamp(0, 15).to(torch.uint8)
    return [s.normal((t, d)), s.normal((d, r), 0.02), s.normal((r, o), 0.02), codes,
            s.uniform((d * o // c["block"],), 0.04, 0.08, F32), s.normal((t, o))]


def _qlora_exact(c, x, a, b, codes, scales, dy):
    book = torch.tensor([-1.0, -0.6962, -0.5251, -0.3949, -0.2844, -0.1848, -0.0911, 0.0, 0.0796, 0.1609, 0.2461, 0.3379,
                         0.4407, 0.5626, 0.7230, 1.0], dtype=F64, device="cuda")
    w = (book[codes.long()].view(-1, c["block"]) * scales.to(F64)[:, None]).view(c["dim"], c["out"])
    return _grads64(lambda t, u, v: t @ w + (t @ u) @ v * (16.0 / c["rank"]), (x, a, b), dy)


def _qlora_work(c):
    t, d, o, r = c["tokens"], c["dim"], c["out"], c["rank"]
    return {"bytes": d * o + 4 * d * o // c["block"] + 2 * (2 * t * d + 2 * t * o), "flops": 4 * t * d * o + 6 * t * r * (d + o)}


# ------------------------------------------------------------------------------------- whole calls
# One training step of a small MLP: mean squared error, gradients, AdamW (the smallest calls: latency
# and launches count), as a pure function: the program keeps the old state too.
@functools.lru_cache(None)
def _step(layers):
    def net(params, x):
        for i in range(layers):
            x = F.linear(x, params[f"w{i}"], params[f"b{i}"], activation="relu" if i + 1 < layers else None)
        return x

    def step(params, state, x, y):
        loss, grads = nb.value_and_grad(lambda p: F.mse_loss(net(p, x), y), create_graph=False)(params)
        params, state = nn.adamw_update(params, grads, state, lr=1e-3, weight_decay=0.01, realize=False)
        return loss, params, state

    return nb.compile(step, cuda_graph=True)


def _step_inputs(c, s):
    dims = [c["inputs"]] + [c["width"]] * c["layers"] + [1]
    p, m, v = {}, {}, {}
    for i, (a, b) in enumerate(zip(dims, dims[1:])):
        for name, shape, std in ((f"w{i}", (a, b), a ** -0.5), (f"b{i}", (b,), 0.02)):
            p[name] = s.normal(shape, std)
            m[name] = s.normal(shape, 1e-2, 0.0, F32)
            v[name] = s.uniform(shape, 1e-4, 1e-3, F32)
    x = s.uniform((c["batch"], c["inputs"]), 0.0, 1.0)
    y = torch.sin(2 * math.pi * x.float().mean(1, keepdim=True)).to(BF16)
    return [p, {"m": m, "v": v, "step": torch.tensor(100.0, device="cuda")}, x, y]


def _step_exact(c, p, state, x, y):
    n = c["layers"] + 1
    names = sorted(p)
    w = {k: p[k].to(F64).requires_grad_(True) for k in names}
    h = x.to(F64)
    for i in range(n):
        h = h @ w[f"w{i}"] + w[f"b{i}"]
        h = torch.relu(h) if i + 1 < n else h
    loss = ((h - y.to(F64)) ** 2).mean()
    new, ms, vs = {}, {}, {}
    for k, g in zip(names, torch.autograd.grad(loss, [w[k] for k in names])):
        ms[k] = 0.9 * state["m"][k].to(F64) + 0.1 * g
        vs[k] = 0.999 * state["v"][k].to(F64) + 0.001 * g * g
        up = (ms[k] / (1 - 0.9 ** 101)) / (torch.sqrt(vs[k] / (1 - 0.999 ** 101)) + 1e-8) + 0.01 * w[k].detach()
        new[k] = w[k].detach() - 1e-3 * up
    return [loss.detach(), new, {"m": ms, "v": vs, "step": state["step"].to(F64) + 1.0}]


def _step_work(c):
    dims = [c["inputs"]] + [c["width"]] * c["layers"] + [1]
    n = sum(a * b + b for a, b in zip(dims, dims[1:]))
    return {"bytes": n * (2 + 2 + 16) + 2 * c["batch"] * c["inputs"], "flops": 6 * c["batch"] * n}


# Logits of a whole decoder for a batch of prompts (inference).
@functools.lru_cache(None)
def _logits(layers, dim, heads, vocab):
    cfg = T.TransformerConfig(n_layers=layers, d_model=dim, n_heads=heads, d_ff=4 * dim, vocab=vocab)
    return nb.compile(lambda params, ids: T.forward(params, ids, cfg), cuda_graph=True)


def _logits_inputs(c, s):
    d = c["heads"] * c["head_dim"]
    params = {"tok_emb": s.normal((c["vocab"], d)), "pos_emb": s.normal((2048, d), 0.1),
              "layers": [dict(zip(LAYER, _layer_inputs(s, d, 4 * d))) for _ in range(c["layers"])],
              "lnf_g": s.normal((d,), 0.1, 1.0), "lnf_b": s.normal((d,), 0.1), "lm_head": s.normal((d, c["vocab"]), d ** -0.5)}
    return [params, s.tokens((c["batch"], c["seq"]), c["vocab"])]


def _logits_exact(c, params, ids):
    up = lambda t: t.to(F64)  # noqa: E731
    x = up(params["tok_emb"])[ids] + up(params["pos_emb"])[: c["seq"]]
    for p in params["layers"]:
        x = _block64(x, {k: up(v) for k, v in p.items()}, c["heads"])
    return TF.layer_norm(x, (x.shape[-1],), up(params["lnf_g"]), up(params["lnf_b"])) @ up(params["lm_head"])


def _logits_work(c):
    t, d, v = c["batch"] * c["seq"], c["heads"] * c["head_dim"], c["vocab"]
    return {"bytes": 2 * (12 * c["layers"] * d * d + d * v + t * d + t * v),
            "flops": 2 * t * (12 * c["layers"] * d * d + d * v) + 2 * c["layers"] * t * c["seq"] * d}


# ------------------------------------------------------------------------------------------ table
# kind: (inputs, compiled function of a case, exact, work, relative error of a correct bf16 result: about four
# times what the outputs differ by from 64 bits)
KINDS = {
    "attn_train": (_attn_train_inputs, lambda c: _attn_train(c["head_dim"]), _attn_train_exact, _attn_train_work, 1e-2),
    "attn_padded": (_attn_padded_inputs, lambda c: _attn_padded(), _attn_padded_exact, _attn_padded_work, 1e-2),
    "attn_prefix": (_attn_prefix_inputs, lambda c: _attn_prefix(), _attn_prefix_exact, _attn_prefix_work, 1e-2),
    "norm": (_norm_inputs, lambda c: _norm(), _norm_exact, _norm_work, 7e-3),
    "mlp": (_mlp_inputs, lambda c: _mlp(), _mlp_exact, _mlp_work, 1e-2),
    "block": (_block_inputs, lambda c: _block(c["heads"] * c["head_dim"], c["heads"], c["hidden"]), _block_exact, _block_work, 2.4e-2),
    "head": (_head_inputs, lambda c: _head(), _head_exact, _head_work, 7e-3),
    "embed": (_embed_inputs, lambda c: _embed(), _embed_exact, _embed_work, 7e-3),
    "cnn": (_cnn_inputs, lambda c: _cnn(), _cnn_exact, _cnn_work, 1e-5),
    "qlora": (_qlora_inputs, lambda c: _qlora(c["dim"], c["out"], c["block"]), _qlora_exact, _qlora_work, 1.2e-2),
    "step": (_step_inputs, lambda c: _step(c["layers"] + 1), _step_exact, _step_work, 2e-2),
    "logits": (_logits_inputs, lambda c: _logits(c["layers"], c["heads"] * c["head_dim"], c["heads"], c["vocab"]), _logits_exact,
               _logits_work, 2.7e-2),
}


def listed():
    return [
        # the training configuration's attention, a quarter of its batch
        {"name": "attention_train_2048", "kind": "attn_train", "batch": 4, "seq": 2048, "heads": 16, "head_dim": 128},
        # an encoder layer over a padded batch of ragged length
        {"name": "attention_padded_777", "kind": "attn_padded", "batch": 8, "seq": 777, "heads": 12, "head_dim": 64},
        # one new position for each of a few sequences (decoding)
        {"name": "attention_decode_4001", "kind": "attn_prefix", "batch": 4, "new": 1, "prefix": 4001, "heads": 16, "head_dim": 128},
        # the norms of the training configuration
        {"name": "layer_norm_16384", "kind": "norm", "rows": 16384, "dim": 2048, "dtype": "bf16"},
        # the feed-forward layer of the training configuration (the largest case)
        {"name": "mlp_16384", "kind": "mlp", "tokens": 16384, "dim": 2048, "hidden": 8192},
        # a whole block at a quarter of the width on sequences of odd length
        {"name": "block_train_1001", "kind": "block", "batch": 2, "seq": 1001, "heads": 8, "head_dim": 64, "hidden": 2048},
        # the head of the training configuration on one gradient-accumulation slice
        {"name": "head_4096", "kind": "head", "tokens": 4096, "dim": 2048, "vocab": 32000},
        # its embedding, whole batch
        {"name": "embedding_16384", "kind": "embed", "batch": 8, "seq": 2048, "dim": 2048, "vocab": 32000, "dtype": "bf16"},
        # the image classifier of the examples at a usual batch
        {"name": "cnn_step_256", "kind": "cnn", "batch": 256, "edge": 28, "planes": 1, "channels": 16, "classes": 10, "dtype": "fp32"},
        # QLoRA on the packed projection of the training configuration
        {"name": "qlora_2048", "kind": "qlora", "tokens": 2048, "dim": 2048, "out": 6144, "rank": 16, "block": 64},
        # the small MLP of the configurations, one whole step
        {"name": "mlp_step_512", "kind": "step", "batch": 512, "inputs": 64, "width": 256, "layers": 3},
        # logits of a small decoder for a batch of prompts
        {"name": "decoder_logits_333", "kind": "logits", "batch": 4, "seq": 333, "layers": 4, "heads": 8, "head_dim": 64, "vocab": 8192},
    ]


def draw(rng):
    kind = rng.choice(sorted(KINDS))
    hd = rng.choice([64, 128])
    if kind == "attn_train":
        seq = _log_int(rng, 64, 4096)
        most = 4 * 16 * 2048 * 2048 * 128 // (seq * seq * hd)          # no more work than the listed case
        heads = rng.choice([h for h in (4, 8, 12, 16, 32) if h <= max(4, most)])
        return {"kind": kind, "batch": rng.randint(1, max(1, min(16, most // heads))), "seq": seq, "heads": heads, "head_dim": hd}
    if kind == "attn_padded":
        seq = _log_int(rng, 40, 1500)
        return {"kind": kind, "batch": rng.randint(1, 8), "seq": seq, "heads": rng.choice([4, 8, 12, 16]), "head_dim": hd}
    if kind == "attn_prefix":
        prefix = _log_int(rng, 200, 8000)
        return {"kind": kind, "batch": _log_int(rng, 1, 16), "new": rng.choice([1, 1, 1, 2, 5, 16, 33]), "prefix": prefix,
                "heads": rng.choice([4, 8, 16]), "head_dim": hd}
    if kind == "norm":
        dtype = rng.choice(["bf16", "bf16", "fp32"])
        dim = rng.choice([256, 512, 768, 1000, 1024, 1536, 2048] + ([3072, 4096] if dtype == "bf16" else []))
        return {"kind": kind, "rows": _log_int(rng, 100, 16384 * 2048 // dim), "dim": dim, "dtype": dtype}
    if kind == "mlp":
        dim = rng.choice([256, 512, 768, 1024, 2048])
        return {"kind": kind, "tokens": _log_int(rng, 64, 16384), "dim": dim, "hidden": 4 * dim}
    if kind == "block":
        heads = rng.choice([4, 8, 12, 16])
        return {"kind": kind, "batch": rng.randint(1, 4), "seq": _log_int(rng, 64, 2048), "heads": heads, "head_dim": hd,
                "hidden": 4 * heads * hd}
    if kind == "head":
        return {"kind": kind, "tokens": _log_int(rng, 100, 4096), "dim": rng.choice([256, 512, 1024, 2048]),
                "vocab": rng.choice([1000, 8192, 32000, _log_int(rng, 1000, 32000)])}
    if kind == "embed":
        seq = _log_int(rng, 64, 2048)
        return {"kind": kind, "batch": rng.randint(1, 8), "seq": seq, "dim": rng.choice([256, 512, 768, 1024, 2048]),
                "vocab": rng.choice([1000, 8192, 32000, _log_int(rng, 1000, 32000)]), "dtype": rng.choice(["bf16", "bf16", "fp32"])}
    if kind == "cnn":
        return {"kind": kind, "batch": _log_int(rng, 16, 256), "edge": rng.choice([16, 28, 32]), "planes": rng.choice([1, 3]),
                "channels": rng.choice([8, 16]), "classes": rng.choice([10, 100]), "dtype": "fp32"}
    if kind == "qlora":
        dim = rng.choice([512, 768, 1024, 2048])
        return {"kind": kind, "tokens": _log_int(rng, 100, 2048), "dim": dim, "out": rng.choice([dim, 3 * dim, 4 * dim]),
                "rank": rng.choice([8, 16, 64]), "block": rng.choice([64, 128])}
    if kind == "step":
        return {"kind": kind, "batch": _log_int(rng, 32, 2048), "inputs": rng.choice([16, 64, 100]), "width": rng.choice([64, 128, 256, 512]),
                "layers": rng.randint(2, 4)}
    return {"kind": kind, "batch": rng.randint(1, 8), "seq": _log_int(rng, 16, 777), "layers": rng.choice([2, 4]),
            "heads": rng.choice([4, 8]), "head_dim": 64, "vocab": rng.choice([1000, 8192, 10001])}


# --------------------------------------------------------------------------------------- interface
def _wrap(v):
    if isinstance(v, dict):
        return {k: _wrap(x) for k, x in v.items()}
    if isinstance(v, list):
        return [_wrap(x) for x in v]
    return nb.Tensor.from_torch(v)


def _unwrap(v):
    if isinstance(v, dict):
        return {k: _unwrap(x) for k, x in v.items()}
    if isinstance(v, (list, tuple)):
        return [_unwrap(x) for x in v]
    return v.to_torch()


def _inputs(case, seed):
    return KINDS[case["kind"]][0](case, _Source(seed))


def prepare(case, seed):
    return {"call": KINDS[case["kind"]][1](case), "args": [_wrap(v) for v in _inputs(case, seed)]}


def run(state):
    return _unwrap(state["call"](*state["args"]))


def work(case):
    return KINDS[case["kind"]][3](case)


def tolerance(case):
    return {"rel": 1e-5 if case.get("dtype") == "fp32" else KINDS[case["kind"]][4]}


def exact(case, seed):
    return KINDS[case["kind"]][2](case, *_inputs(case, seed))
