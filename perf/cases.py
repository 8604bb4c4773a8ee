"""The workloads this framework's speed is measured on.

The framework trains and evaluates decoder layers: a user's program brings a model built from the
package's blocks (``models.llama``, ``models.gpt``) or calls its layers one by one
(``ops.functional``).  The cases below are those calls on one GPU: blocks forward (evaluation) and
forward + backward (training), the layers whose cost is not a matrix product (attention, the norms),
the head with its loss, and one whole model.  Sizes are the presets of the two model modules, the
shapes of ``benchmarks/`` and the ragged lengths of ``tests/``.

Training cases accumulate parameter gradients into one flat buffer that is zeroed at the start of the
pass, which is how the engine hands gradients to a block.

Kinds of a case (``kind``):

``gpt`` / ``llama``   one block, ``[batch, seq, hidden]`` in and out
``attention``         ``causal_attention`` over separate q, k, v (grouped-query when ``kv`` < ``heads``)
``rmsnorm``           residual add + RMSNorm (``add_rmsnorm``), as between the two halves of a block
``layernorm``         LayerNorm with gain and bias
``head``              ``linear_cross_entropy``: projection to the vocabulary and mean token loss
``model``             a whole GPT: embedding, blocks, final norm, tied head, loss, all gradients
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as tnf
from torch.utils.checkpoint import checkpoint

from flextrain_b200.models import gpt, llama
from flextrain_b200.ops import functional as F

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
EPS = 1e-5
LEAVES = ("x", "r", "q", "k", "v")            # activations that a training case differentiates


# ----------------------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest block the tests and the smoke run train: launches and latency
        dict(name="gpt_tiny_train", kind="gpt", batch=2, seq=128, hidden=256, heads=4, ffn=1024,
             dtype="bf16", train=True),
        # a GPT-2 small layer at its full context, two sequences per micro-batch
        dict(name="gpt2_small_train", kind="gpt", batch=2, seq=1024, hidden=768, heads=12, ffn=3072,
             dtype="fp16", train=True),
        # validation pass of a GPT-2 XL layer over texts of a length that is no multiple of any tile
        dict(name="gpt2_xl_eval_ragged", kind="gpt", batch=3, seq=1000, hidden=1600, heads=25, ffn=6400,
             dtype="bf16", train=False),
        # the ordinary Llama training layer: one full-context sequence per micro-batch
        dict(name="llama_7b_train", kind="llama", batch=1, seq=4096, hidden=4096, heads=32, kv=32,
             ffn=11008, dtype="bf16", train=True),
        # the forward half of the headline benchmark's layer, half its micro-batch (also what the
        # checkpointed recompute and an evaluation pass run)
        dict(name="llama_13b_eval", kind="llama", batch=4, seq=4096, hidden=5120, heads=40, kv=40,
             ffn=13824, dtype="bf16", train=False),
        # the largest layer: grouped-query attention, the widest projections
        dict(name="llama_70b_train", kind="llama", batch=1, seq=2048, hidden=8192, heads=64, kv=8,
             ffn=28672, dtype="bf16", train=True),
        # attention alone: the grouped-query shape of the attention benchmark
        dict(name="attention_gqa_train", kind="attention", batch=2, seq=4096, heads=64, kv=8, head_dim=128,
             dtype="bf16", train=True),
        # attention alone: short odd sequences with 64-wide heads
        dict(name="attention_ragged_train", kind="attention", batch=3, seq=1000, heads=16, kv=16,
             head_dim=64, dtype="fp16", train=True),
        # the residual add and norm of the headline layer, its whole micro-batch
        dict(name="rmsnorm_13b_train", kind="rmsnorm", batch=8, seq=4096, hidden=5120, dtype="bf16",
             train=True),
        # the LayerNorm of a GPT-2 XL layer, an odd number of rows
        dict(name="layernorm_xl_train", kind="layernorm", batch=3, seq=1365, hidden=1600, dtype="fp16",
             train=True),
        # the Llama head on one sequence whose first token has no prediction
        dict(name="head_7b_train", kind="head", batch=1, seq=4095, hidden=4096, vocab=32000, dtype="bf16",
             train=True),
        # one whole call: loss and every gradient of a GPT-2 small
        dict(name="gpt2_small_model_train", kind="model", batch=2, seq=512, hidden=768, heads=12, ffn=3072,
             layers=12, vocab=50304, dtype="bf16", train=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_any(rng):
    kind = rng.choice(["gpt", "llama", "attention", "rmsnorm", "layernorm", "head"])
    c = dict(kind=kind, batch=rng.choice([1, 1, 2, 3, 4]), dtype=rng.choice(["bf16", "bf16", "fp16"]),
             train=rng.random() < 0.7)
    if kind == "gpt":
        heads, d = _log(rng, 4, 40), rng.choice([64, 128])
        return dict(c, seq=_log(rng, 64, 2048), hidden=d * heads, heads=heads, ffn=4 * d * heads)
    if kind in ("rmsnorm", "layernorm"):
        return dict(c, seq=_log(rng, 64, 8192), hidden=64 * _log(rng, 4, 128))
    if kind == "head":
        return dict(c, seq=_log(rng, 64, 4096), hidden=64 * _log(rng, 4, 128),
                    vocab=rng.choice([1024, 32000, 50304]), train=True)
    heads = _log(rng, 2, 64)
    c.update(seq=_log(rng, 64, 4096), heads=heads, kv=rng.choice([k for k in (1, 2, 4, 8, heads) if heads % k == 0]))
    if kind == "attention":
        return dict(c, head_dim=rng.choice([64, 128]))
    hidden = 128 * heads
    return dict(c, hidden=hidden, ffn=8 * _log(rng, hidden // 4, hidden * 7 // 16))


def draw(rng):
    """A case of the same ranges: 64- and 128-wide heads, hidden 256 to 8192, 64 to 16384 tokens of any
    length, both 16-bit types, with and without a backward pass; nothing heavier than what is listed."""
    def cost(case):
        w = work(case)
        return w["flops"] / 1.5e15 + w["bytes"] / 6.5e12

    most = max(cost(c) for c in listed())
    while True:
        case = _draw_any(rng)
        if cost(case) <= 0.9 * most:
            return case


# ----------------------------------------------------------------------------- inputs
def _inputs(case, seed):
    """Every tensor of the case, in the case's type, from the seed alone: ``(activations, parameters)``,
    both dicts.  Parameter names are those of the block or model."""
    dev = torch.device("cuda")
    dt = DTYPES[case["dtype"]]
    gen = torch.Generator(device=dev).manual_seed(seed)

    def rand(*shape, std=1.0, mean=0.0):
        t = torch.empty(*shape, dtype=dt, device=dev)
        return t.normal_(mean, std, generator=gen)

    def tokens(vocab):
        return torch.randint(0, vocab, (case["batch"], case["seq"]), generator=gen, device=dev)

    def masked(labels):                                   # padding positions carry no loss
        drop = torch.rand(labels.shape, generator=gen, device=dev) < 0.05
        return labels.masked_fill(drop, -100)

    b, s, kind = case["batch"], case["seq"], case["kind"]
    if kind == "attention":
        q, k, d = case["heads"], case["kv"], case["head_dim"]
        return dict(q=rand(b, s, q, d), k=rand(b, s, k, d), v=rand(b, s, k, d), dy=rand(b, s, q, d)), {}
    h = case["hidden"]
    std = 0.02

    def gain(n):
        return rand(n, std=0.1, mean=1.0)

    def gpt_block(prefix=""):
        f, out_std = case["ffn"], std / math.sqrt(2.0 * case.get("layers", 12))
        return {prefix + k: v for k, v in dict(
            ln1_w=gain(h), ln1_b=rand(h, std=std), wqkv=rand(3 * h, h, std=std), bqkv=rand(3 * h, std=std),
            wo=rand(h, h, std=out_std), bo=rand(h, std=std), ln2_w=gain(h), ln2_b=rand(h, std=std),
            w_fc=rand(f, h, std=std), b_fc=rand(f, std=std), w_proj=rand(h, f, std=out_std),
            b_proj=rand(h, std=std)).items()}

    if kind == "rmsnorm":
        return dict(x=rand(b, s, h), r=rand(b, s, h), ds=rand(b, s, h), dy=rand(b, s, h)), dict(w=gain(h))
    if kind == "layernorm":
        return dict(x=rand(b, s, h), dy=rand(b, s, h)), dict(w=gain(h), b=rand(h, std=std))
    if kind == "head":
        return (dict(x=rand(b * s, h), labels=masked(tokens(case["vocab"])).reshape(-1)),
                dict(w=rand(case["vocab"], h, std=std)))
    if kind == "model":
        params = dict(wte=rand(case["vocab"], h, std=std), wpe=rand(s, h, std=std))
        for i in range(case["layers"]):
            params.update(gpt_block(f"blocks.{i}."))
        params.update(lnf_w=gain(h), lnf_b=rand(h, std=std))
        return dict(tokens=tokens(case["vocab"]), labels=masked(tokens(case["vocab"]))), params
    acts = dict(x=rand(b, s, h), dy=rand(b, s, h))
    if kind == "gpt":
        return acts, gpt_block()
    f, d = case["ffn"], h // case["heads"]
    return acts, dict(attn_norm=gain(h), wqkv=rand(h + 2 * case["kv"] * d, h, std=std), wo=rand(h, h, std=std),
                      ffn_norm=gain(h), w_gate_up=rand(2 * f, h, std=std), w_down=rand(h, f, std=std))


def _module(case, dtype):
    if case["kind"] == "llama":
        return llama.LlamaBlock(llama.LlamaConfig(
            num_layers=1, hidden=case["hidden"], num_heads=case["heads"], num_kv_heads=case["kv"],
            ffn=case["ffn"], seq_len=case["seq"], eps=EPS, init_std=0.0), dtype=dtype)
    cfg = gpt.GPTConfig(num_layers=case.get("layers", 1), hidden=case["hidden"], num_heads=case["heads"],
                        ffn=case["ffn"], vocab=case.get("vocab", 1024), seq_len=case["seq"], eps=EPS, init_std=0.0)
    return gpt.GPTModel(cfg, dtype=dtype) if case["kind"] == "model" else gpt.GPTBlock(cfg, dtype=dtype)


def prepare(case, seed):
    acts, params = _inputs(case, seed)
    train = case["train"]
    st = dict(case=case, **acts)
    if case["kind"] in ("gpt", "llama", "model"):
        with torch.device("meta"):
            mod = _module(case, DTYPES[case["dtype"]])
        mod.load_state_dict(params, assign=True)
        mod.requires_grad_(train)
        st["module"] = mod
        names = [n for n, _ in mod.named_parameters()]
        weights = [p for _, p in mod.named_parameters()]
    else:
        names = list(params)
        weights = [torch.nn.Parameter(p, requires_grad=train) for p in params.values()]
        st.update(zip(names, weights))
    if case["kind"] == "llama":
        st["cos"], st["sin"] = F.rope_tables(case["seq"], case["hidden"] // case["heads"], 10000.0,
                                             device=torch.device("cuda"))
    st["grads"] = {}
    if train:
        # gradients of all parameters in one buffer, each starting on a 16-byte boundary
        sizes = [(p.numel() + 7) // 8 * 8 for p in weights]
        st["flat"] = torch.zeros(sum(sizes), dtype=DTYPES[case["dtype"]], device="cuda")
        lo, spans = 0, {}
        for n, p, size in zip(names, weights, sizes):
            p.grad = st["flat"][lo:lo + p.numel()].view_as(p)
            if n.startswith("blocks."):              # reported block by block: "blocks.<i>"
                n = n.rsplit(".", 1)[0]
                spans[n] = (spans.get(n, (lo,))[0], lo + p.numel())
            else:
                st["grads"][n] = p.grad
            lo += size
        st["grads"].update({n: st["flat"][a:b] for n, (a, b) in spans.items()})
        st["leaves"] = {n: st[n].requires_grad_(True) for n in LEAVES if n in acts}
    return st


def _forward(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "gpt":
        return st["module"](st["x"])
    if kind == "llama":
        return st["module"](st["x"], st["cos"], st["sin"])
    if kind == "attention":
        return F.causal_attention(st["q"], st["k"], st["v"])
    if kind == "rmsnorm":
        return F.add_rmsnorm(st["x"], st["r"], st["w"], EPS)
    if kind == "layernorm":
        return F.layernorm(st["x"], st["w"], st["b"], EPS)
    if kind == "head":
        return F.linear_cross_entropy(st["x"], st["w"], st["labels"])
    return st["module"](st["tokens"], st["labels"])


def _named(case, out):
    return dict(zip(("sum", "out") if case["kind"] == "rmsnorm" else ("out",), out if isinstance(out, tuple) else (out,)))


def run(state):
    case = state["case"]
    if not case["train"]:
        with torch.no_grad():
            return _named(case, _forward(state))
    if state["grads"]:
        state["flat"].zero_()
    for t in state["leaves"].values():
        t.grad = None
    out = _forward(state)
    if case["kind"] in ("head", "model"):
        out.backward()
    elif case["kind"] == "rmsnorm":
        torch.autograd.backward(out, (state["ds"], state["dy"]))
    else:
        out.backward(state["dy"])
    res = {n: t.detach() for n, t in _named(case, out).items()}
    res.update({"d_" + n: t.grad for n, t in state["leaves"].items()})
    res.update({"d_" + n: g for n, g in state["grads"].items()})
    return res


# ----------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    b, s, train = case["batch"], case["seq"], case["train"]
    t = b * s
    kind = case["kind"]

    def attention_flops(heads, d):
        return 4.0 * b * heads * d * s * (s + 1) / 2 * (3.5 if train else 1.0)

    if kind == "attention":
        q, k = t * case["heads"] * case["head_dim"], t * case["kv"] * case["head_dim"]
        n = 2 * q + 2 * k + ((2 * q + 2 * k) if train else 0)          # + dy and dq, dk, dv
        return dict(bytes=2 * n, flops=attention_flops(case["heads"], case["head_dim"]))
    h = case["hidden"]
    if kind == "rmsnorm":                                              # x, r -> s, y; ds, dy -> dx and dr alike
        return dict(bytes=2 * (t * h * (7 if train else 4) + h * (2 if train else 1)), flops=0)
    if kind == "layernorm":
        return dict(bytes=2 * (t * h * (4 if train else 2) + h * (4 if train else 2)), flops=0)
    if kind == "head":
        n = t * h + case["vocab"] * h
        return dict(bytes=2 * n * (2 if train else 1) + 8 * t, flops=2.0 * t * h * case["vocab"] * (3 if train else 1))
    if kind == "llama":
        d = h // case["heads"]
        mats = h * (h + 2 * case["kv"] * d) + h * h + 3 * h * case["ffn"]
        vecs = 2 * h
    else:
        mats = 4 * h * h + 2 * h * case["ffn"]
        vecs = 9 * h + case["ffn"]
        d = h // case["heads"]
    layers = case.get("layers", 1)
    flops = layers * (2.0 * t * mats * (3 if train else 1) + attention_flops(case["heads"], d))
    if kind == "model":
        emb = case["vocab"] * h
        n = layers * (mats + vecs) + emb + s * h + 2 * h
        return dict(bytes=2 * 2 * n + 16 * t, flops=flops + 6.0 * t * emb)
    n = mats + vecs + 2 * t * h                                        # parameters, x and y
    return dict(bytes=2 * n * (2 if train else 1), flops=flops)


def tolerance(case):
    """About four times the distance from the 64-bit result that the kernels show: one rounding to the
    16-bit type per stored intermediate, which in bf16 leaves 0.0025 after a norm or attention, 0.005
    after a GPT block, 0.010 to 0.015 after a Llama block (unnormalised SwiGLU products, wider sums).
    fp16 has three more bits of mantissa."""
    rel = {"rmsnorm": 0.01, "layernorm": 0.01, "attention": 0.01, "head": 0.01, "gpt": 0.02, "llama": 0.04,
           "model": 0.05}[case["kind"]]
    return {"rel": rel / 6 if case["dtype"] == "fp16" else rel}


# ----------------------------------------------------------------------------- 64-bit results
def _attention64(q, k, v):
    """Causal attention of [b, s, heads, d] in 64 bits, one (sequence, key head) at a time and
    recomputed in the backward pass, so that no score matrix is kept."""
    s, d, rep = q.shape[1], q.shape[3], q.shape[2] // k.shape[2]
    mask = torch.ones(s, s, dtype=torch.bool, device=q.device).triu(1)

    def one(qh, kh, vh):                                               # [rep, s, d], [s, d], [s, d]
        p = (qh @ kh.T).mul(1.0 / math.sqrt(d)).masked_fill(mask, float("-inf"))
        return p.softmax(-1) @ vh

    rows = []
    for i in range(q.shape[0]):
        heads = [checkpoint(one, q[i, :, j * rep:(j + 1) * rep].transpose(0, 1), k[i, :, j], v[i, :, j],
                            use_reentrant=False) for j in range(k.shape[2])]
        rows.append(torch.cat(heads, 0).transpose(0, 1))
    return torch.stack(rows)


def _rms64(x, w):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + EPS) * w


def _gpt64(x, p, heads, prefix=""):
    w = lambda n: p[prefix + n]                                        # noqa: E731
    b, s, h = x.shape
    a = tnf.layer_norm(x, (h,), w("ln1_w"), w("ln1_b"), EPS) @ w("wqkv").T + w("bqkv")
    q, k, v = (t.unflatten(-1, (heads, h // heads)) for t in a.split(h, -1))
    x = x + _attention64(q, k, v).reshape(b, s, h) @ w("wo").T + w("bo")
    a = tnf.layer_norm(x, (h,), w("ln2_w"), w("ln2_b"), EPS) @ w("w_fc").T + w("b_fc")
    return x + tnf.gelu(a, approximate="tanh") @ w("w_proj").T + w("b_proj")


def _llama64(x, p, case):
    b, s, h = x.shape
    d, heads, kv = h // case["heads"], case["heads"], case["kv"]
    inv = 10000.0 ** (-torch.arange(0, d, 2, dtype=torch.float64, device=x.device) / d)
    ang = torch.arange(s, dtype=torch.float64, device=x.device)[:, None] * inv
    cos, sin = torch.cos(ang).repeat(1, 2)[:, None], torch.sin(ang).repeat(1, 2)[:, None]

    def rot(t):
        lo, hi = t.chunk(2, -1)
        return t * cos + torch.cat((-hi, lo), -1) * sin

    a = _rms64(x, p["attn_norm"]) @ p["wqkv"].T
    q, k, v = (t.unflatten(-1, (-1, d)) for t in a.split([heads * d, kv * d, kv * d], -1))
    x = x + _attention64(rot(q), rot(k), v).reshape(b, s, h) @ p["wo"].T
    g, u = (_rms64(x, p["ffn_norm"]) @ p["w_gate_up"].T).chunk(2, -1)
    return x + (tnf.silu(g) * u) @ p["w_down"].T


def exact(case, seed):
    acts, params = _inputs(case, seed)
    train, kind = case["train"], case["kind"]
    a = {n: t.double() if t.is_floating_point() else t for n, t in acts.items()}
    p = {n: t.double().requires_grad_(train) for n, t in params.items()}
    del acts, params
    leaves = {n: a[n].requires_grad_(train) for n in LEAVES if n in a}
    with torch.set_grad_enabled(train):
        if kind == "gpt":
            out = _gpt64(a["x"], p, case["heads"])
        elif kind == "llama":
            out = _llama64(a["x"], p, case)
        elif kind == "attention":
            out = _attention64(a["q"], a["k"], a["v"])
        elif kind == "rmsnorm":
            s = a["x"] + a["r"]
            out = (s, _rms64(s, p["w"]))
        elif kind == "layernorm":
            out = tnf.layer_norm(a["x"], (case["hidden"],), p["w"], p["b"], EPS)
        elif kind == "head":
            out = tnf.cross_entropy(a["x"] @ p["w"].T, a["labels"])
        else:
            x = p["wte"][a["tokens"]] + p["wpe"]
            for i in range(case["layers"]):
                x = _gpt64(x, p, case["heads"], f"blocks.{i}.")
            x = tnf.layer_norm(x, (case["hidden"],), p["lnf_w"], p["lnf_b"], EPS)
            out = tnf.cross_entropy((x @ p["wte"].T).flatten(0, 1), a["labels"].flatten())
        if not train:
            return _named(case, out)
        if kind == "rmsnorm":
            torch.autograd.backward(out, (a["ds"], a["dy"]))
        else:
            out.backward(a.get("dy"))
    res = {n: t.detach() for n, t in _named(case, out).items()}
    res.update({"d_" + n: t.grad for n, t in leaves.items()})
    blocks = {}
    for n, t in p.items():
        if n.startswith("blocks."):
            blocks.setdefault(n.rsplit(".", 1)[0], []).append(t.grad.reshape(-1))
        else:
            res["d_" + n] = t.grad
    res.update({"d_" + n: torch.cat(parts) for n, parts in blocks.items()})
    return res
