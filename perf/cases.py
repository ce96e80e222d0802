"""Performance cases of the library: what its users run on one GPU, through its public entry points.

Most cases are one MoE layer (``MoELayer``: inference forward, CUDA-graph replay, training forward + backward with and
without the optimizer in the weight-gradient epilogue) over the shapes of the library's own configurations:

    512 -> 2048, 768 -> 3072          the Transformer-XL and the BERT / GPT-2-small sized example models
    1024 -> 4096                      the layer benchmark of the evaluation scripts (4 to 64 experts, 8192 tokens)
    2048 -> 8192, 64 experts          the GPT-MoE benchmark model (8 sequences of 1024 tokens, GELU, top-2)
    4096 -> 14336, 8 experts          the SwiGLU layer (16384 tokens, capacity factor 1.2; 128 / 512 / 2048 tokens in fp16)

The rest are the parts around it that a training step calls: ``LayerNorm``, ``FusedSGD`` and a whole GPT-MoE forward.
"""
import math

import torch

from ccfuser_b200 import MoEConfig, MoELayer
from ccfuser_b200.models.gpt_moe import GPTMoE, GPTMoEConfig
from ccfuser_b200.ops.fused import GraphedForward
from ccfuser_b200.ops.norm import LayerNorm
from ccfuser_b200.ops.optim import FusedSGD

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
# learning rate of the in-place update: of the order of half a unit in the last place of a weight per pass, so that
# weights change and stay in the range of a freshly initialised layer over many passes
SGD_LR = 4e-6
STEP_LR, STEP_WD = 1e-2, 0.01


def _layer(name, mode, tokens, d, f, experts, *, top_k=2, act="gelu", dtype="bf16", cf=0.0, zipf=0.0):
    c = {"kind": "layer", "mode": mode, "tokens": tokens, "d": d, "f": f, "experts": experts, "top_k": top_k, "act": act,
         "dtype": dtype, "cf": cf, "zipf": zipf}
    return {"name": name, **c} if name else c


def listed():
    return [
        # decode of a small model, eager: a handful of tokens, launches and latency decide
        _layer("decode_16", "infer", 16, 1024, 4096, 16),
        # latency-bound serving replayed from a CUDA graph: 128 tokens, large SwiGLU experts in fp16, weights stream once
        _layer("graph_128", "graph", 128, 4096, 14336, 8, act="swiglu", dtype="fp16"),
        # a ragged serving batch on the GPT-MoE layer: about 24 rows for each of 64 experts
        _layer("infer_777", "infer", 777, 2048, 8192, 64),
        # prefill with skewed expert popularity and a capacity that drops rows
        _layer("prefill_zipf", "infer", 8192, 4096, 14336, 8, act="swiglu", cf=2.0, zipf=1.2),
        # training, evaluation-script layer: few experts with many rows each, and many experts with few
        _layer("train_4_experts", "train", 8192, 1024, 4096, 4),
        _layer("train_64_experts", "train", 8192, 1024, 4096, 64),
        # training, small example model in fp16 with an odd token count, ReLU experts and top-1 routing
        _layer("train_odd", "train", 3001, 768, 3072, 16, top_k=1, act="relu", dtype="fp16"),
        # training, one layer of the GPT-MoE benchmark with the expert SGD applied in the backward pass
        _layer("train_gpt_sgd", "train_sgd", 8192, 2048, 8192, 64),
        # training, the large SwiGLU layer
        _layer("train_swiglu", "train", 16384, 4096, 14336, 8, act="swiglu", cf=1.2),
        # the normalisation in front of every attention and FFN block of that model, forward and backward
        {"name": "layernorm", "kind": "norm", "rows": 8192, "d": 2048, "dtype": "bf16"},
        # the optimizer over the dense parameters of three transformer blocks (matrices, biases, norm weights)
        {"name": "sgd_blocks", "kind": "sgd", "blocks": 3, "d": 2048, "f": 8192, "dtype": "bf16"},
        # a whole call: token ids to logits through a two-block GPT-MoE (one dense and one MoE block)
        {"name": "gpt_logits", "kind": "gpt", "batch": 2, "seq": 1024, "d": 2048, "f": 8192, "experts": 64, "vocab": 50257},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# (d_model, d_ffn, expert counts, activations)
_SHAPES = [(512, 2048, (8, 16, 64), ("gelu", "relu")), (768, 3072, (8, 16, 32), ("gelu", "relu")),
           (1024, 4096, (4, 8, 16, 32, 64), ("gelu", "swiglu")), (2048, 8192, (8, 16, 64), ("gelu",)),
           (4096, 14336, (8,), ("swiglu",))]


def draw(rng):
    kind = rng.choice(["infer", "infer", "graph", "train", "train", "train", "train_sgd", "norm", "sgd"])
    dtype = rng.choice(["bf16", "bf16", "fp16"])
    if kind == "norm":
        return {"kind": "norm", "rows": _log_int(rng, 64, 16384), "d": rng.choice([512, 768, 1024, 2048]), "dtype": dtype}
    if kind == "sgd":
        d = rng.choice([512, 768, 1024, 2048])
        return {"kind": "sgd", "blocks": rng.choice([1, 2, 3]), "d": d, "f": 4 * d, "dtype": dtype}
    d, f, counts, acts = rng.choice(_SHAPES)
    experts, act = rng.choice(counts), rng.choice(acts)
    lo, hi = {"infer": (1, 8192), "graph": (8, 2048), "train": (128, 16384), "train_sgd": (1024, 16384)}[kind]
    if d >= 2048:
        hi = min(hi, 8192)
    top_k = rng.choice([1, 2, 2, 2])
    cf = rng.choice([0.0, 0.0, 1.2, 2.0])
    zipf = 1.2 if cf == 2.0 else 0.0
    return _layer(None, kind, _log_int(rng, lo, hi), d, f, experts, top_k=top_k, act=act, dtype=dtype, cf=cf, zipf=zipf)


# ---- inputs, from the seed alone -----------------------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _layer_inputs(case, seed):
    """Parameters N(0, 0.02^2), tokens and upstream gradient N(0, 1): what the layer benchmark uses. Tokens whose choice of
    experts is a near tie (k-th and next logit within 1e-3) are left out: it may go either way in another correct sum."""
    g = _generator(seed)
    dt, t, d, f, e, k = DTYPES[case["dtype"]], case["tokens"], case["d"], case["f"], case["experts"], case["top_k"]

    def normal(*shape, std=0.02):
        return torch.empty(*shape, dtype=dt, device="cuda").normal_(0.0, std, generator=g)

    p = {"gate.weight": normal(e, d), "gate.bias": normal(e), "w1": normal(e, f, d), "b1": normal(e, f),
         "w2": normal(e, d, f), "b2": normal(e, d)}
    if case["act"] == "swiglu":
        p["wg"], p["bg"] = normal(e, f, d), normal(e, f)
    if case["zipf"]:
        popularity = torch.arange(1, e + 1, dtype=torch.float64, device="cuda").pow(-case["zipf"])
        popularity = (popularity / popularity.sum()).log()
        p["gate.bias"] = popularity[torch.randperm(e, generator=g, device="cuda")].to(dt)
    pool = normal(t + t // 8 + 64, d, std=1.0)
    if k < e:
        top = (pool.float() @ p["gate.weight"].float().t() + p["gate.bias"].float()).topk(k + 1, dim=1).values
        near = top[:, k - 1] - top[:, k] < 1e-3
        pool = pool[torch.argsort(near.to(torch.int32), stable=True)[:t].sort().values]
    p["x"] = pool[:t].contiguous()
    p["dy"] = normal(t, d, std=1.0)
    return p


def _norm_inputs(case, seed):
    g = _generator(seed)
    dt, rows, d = DTYPES[case["dtype"]], case["rows"], case["d"]
    make = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    return {"x": (make(rows, d) * 2.0 + 0.25).to(dt), "dy": make(rows, d).to(dt), "w": (1.0 + 0.1 * make(d)).to(dt),
            "b": (0.1 * make(d)).to(dt)}


def _sgd_inputs(case, seed):
    g = _generator(seed)
    dt, d, f = DTYPES[case["dtype"]], case["d"], case["f"]
    shapes = []
    for _ in range(case["blocks"]):
        shapes += [(d, d), (d,)] * 4 + [(f, d), (f,), (d, f), (d,)] + [(d,)] * 4
    ps = [torch.empty(s, dtype=dt, device="cuda").normal_(0.0, 0.02, generator=g) for s in shapes]
    gs = [torch.empty(s, dtype=dt, device="cuda").normal_(0.0, 0.01, generator=g) for s in shapes]
    return ps, gs


class _State:
    """What a program holds between calls; gives the layer's symmetric buffers back when it is dropped."""

    def __init__(self, case, **kw):
        self.case = case
        self.__dict__.update(kw)

    def __del__(self):
        layers = [self.layer] if hasattr(self, "layer") else self.model.moe_layers() if hasattr(self, "model") else []
        self.__dict__.pop("graph", None)
        if layers:
            torch.cuda.synchronize()
            for m in layers:
                m.release()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "norm":
        v = _norm_inputs(case, seed)
        norm = LayerNorm(case["d"], device="cuda", dtype=DTYPES[case["dtype"]])
        with torch.no_grad():
            norm.weight.copy_(v["w"])
            norm.bias.copy_(v["b"])
        return _State(case, norm=norm, x=v["x"].requires_grad_(), dy=v["dy"])
    if kind == "sgd":
        ps, gs = _sgd_inputs(case, seed)
        params = [torch.nn.Parameter(p) for p in ps]
        for p, g in zip(params, gs):
            p.grad = g
        return _State(case, params=params, opt=FusedSGD(params, lr=STEP_LR, weight_decay=STEP_WD))
    if kind == "gpt":
        c = GPTMoEConfig(vocab_size=case["vocab"], n_layer=2, n_head=16, d_model=case["d"], d_ffn=case["f"],
                         seq_len=case["seq"], num_experts=case["experts"], backend="fused",
                         max_tokens=case["batch"] * case["seq"])
        torch.manual_seed(seed)
        torch.cuda.manual_seed(seed)
        model = GPTMoE(c, device="cuda")
        ids = torch.randint(0, case["vocab"], (case["batch"], case["seq"]), device="cuda", generator=_generator(seed))
        with torch.no_grad():
            model(ids[:1, :8])          # a first call sets the layer's buffers up
        return _State(case, model=model, ids=ids)
    v = _layer_inputs(case, seed)
    cfg = MoEConfig(d_model=case["d"], d_ffn=case["f"], num_experts=case["experts"], top_k=case["top_k"],
                    capacity_factor=case["cf"] or None, activation=case["act"], dtype=DTYPES[case["dtype"]],
                    backend="fused", max_tokens=case["tokens"])
    layer = MoELayer(cfg, device="cuda")
    with torch.no_grad():
        for name, p in _parameters(layer, case).items():
            p.copy_(v[name])
    mode = case["mode"]
    if mode == "graph":
        return _State(case, layer=layer, graph=GraphedForward(layer, case["tokens"]), x=v["x"])
    if mode == "train_sgd":
        layer.fuse_sgd(SGD_LR)
    with torch.no_grad():
        layer(v["x"][:1])               # a first call sets the layer's buffers up
    return _State(case, layer=layer, x=v["x"].requires_grad_(mode != "infer"), dy=v["dy"])


def _parameters(layer, case):
    ex = layer.experts
    p = {"gate.weight": layer.gate.gate.weight, "gate.bias": layer.gate.gate.bias, "w1": ex.htoh4.weight, "b1": ex.htoh4.bias,
         "w2": ex.h4toh.weight, "b2": ex.h4toh.bias}
    if case["act"] == "swiglu":
        p["wg"], p["bg"] = ex.htoh4_gate.weight, ex.htoh4_gate.bias
    return p


# ---- one pass --------------------------------------------------------------------------------------------------------
def run(state):
    case = state.case
    kind = case["kind"]
    if kind == "norm":
        state.x.grad = state.norm.weight.grad = state.norm.bias.grad = None
        y = state.norm(state.x)
        y.backward(state.dy)
        return {"y": y.detach(), "dx": state.x.grad, "dw": state.norm.weight.grad, "db": state.norm.bias.grad}
    if kind == "sgd":
        state.opt.step()
        return [p.detach() for p in state.params]
    if kind == "gpt":
        with torch.no_grad():
            return state.model(state.ids)
    if case["mode"] == "graph":
        return state.graph(state.x)
    if case["mode"] == "infer":
        with torch.no_grad():
            return state.layer(state.x)
    params = _parameters(state.layer, case)
    state.x.grad = None
    for p in params.values():
        p.grad = None
    y = state.layer(state.x)
    y.backward(state.dy)
    out = {"y": y.detach(), "dx": state.x.grad}
    for name, p in params.items():
        if p.grad is not None:
            out["d" + name] = p.grad
        else:
            out[name] = p.detach()      # updated in place by the backward pass
    return out


# ---- what a pass cannot do without -----------------------------------------------------------------------------------
def _kept_rows(case):
    slots, e = case["tokens"] * case["top_k"], case["experts"]
    if not case["cf"]:
        return slots
    cap = min(slots, math.ceil(case["cf"] * slots / e))
    if not case["zipf"]:
        return min(slots, e * cap)
    share = [r ** -case["zipf"] for r in range(1, e + 1)]
    return sum(min(cap, case["tokens"], slots * s / sum(share)) for s in share)


def work(case):
    kind = case["kind"]
    if kind == "norm":
        n = case["rows"] * case["d"]
        return {"bytes": 8 * n + 16 * case["d"], "flops": 20 * n}          # x, dy in; y, dx out
    if kind == "sgd":
        n = case["blocks"] * (4 * case["d"] ** 2 + 2 * case["d"] * case["f"] + 9 * case["d"] + case["f"])
        return {"bytes": 6 * n, "flops": 4 * n}
    if kind == "gpt":
        t, d, f, e = case["batch"] * case["seq"], case["d"], case["f"], case["experts"]
        vocab = (case["vocab"] + 127) // 128 * 128
        flops = t * (2 * (8 * d * d + 4 * case["seq"] * d // 2) + 4 * d * f + 2 * 4 * d * f + 2 * d * e + 2 * d * vocab)
        params = 2 * 4 * d * d + 2 * d * f + e * 2 * d * f + e * d + vocab * d
        return {"bytes": 2 * (params + t * vocab) + 8 * t, "flops": flops}
    t, d, f, e = case["tokens"], case["d"], case["f"], case["experts"]
    mats = 3 if case["act"] == "swiglu" else 2
    rows = _kept_rows(case)
    used = e * (1 - (1 - 1 / e) ** rows)                                    # experts that receive a row at all
    weights = 2 * used * mats * d * f + 2 * e * d
    flops = 2 * mats * d * f * rows + 2 * t * d * e
    if case["mode"] in ("infer", "graph"):
        return {"bytes": weights + 4 * t * d, "flops": flops}
    # x, dy in; y, dx out; weights read once, their gradients (or their new values) written once
    return {"bytes": 8 * t * d + weights + 2 * e * mats * d * f, "flops": 3 * flops}


def tolerance(case):
    """About four times what these outputs differ by from the same sums in 64 bits: operands, stored activations and
    results carry 8 (bf16) or 11 (fp16) bits of mantissa, sums are in fp32."""
    kind, bf16 = case["kind"], case.get("dtype", "bf16") == "bf16"
    if kind in ("norm", "sgd"):
        return {"rel": 7e-3 if bf16 else 1e-3}
    if kind == "gpt":
        return {"rel": 2e-2, "max": 0.5}
    return {"rel": 1.5e-2 if bf16 else 2e-3, "max": 0.5 if bf16 else 0.08}


# ---- the same in 64 bits, plain torch --------------------------------------------------------------------------------
def exact(case, seed):
    kind = case["kind"]
    if kind == "gpt":
        return None
    if kind == "norm":
        v = {k: t.double() for k, t in _norm_inputs(case, seed).items()}
        x, w, b = v["x"].requires_grad_(), v["w"].requires_grad_(), v["b"].requires_grad_()
        y = torch.nn.functional.layer_norm(x, (case["d"],), w, b, 1e-5)
        dx, dw, db = torch.autograd.grad(y, (x, w, b), v["dy"])
        return {"y": y.detach(), "dx": dx, "dw": dw, "db": db}
    if kind == "sgd":
        ps, gs = _sgd_inputs(case, seed)
        return [p.double() - STEP_LR * (g.double() + STEP_WD * p.double()) for p, g in zip(ps, gs)]
    return _exact_layer(case, seed)


def _exact_layer(case, seed):
    v = _layer_inputs(case, seed)
    t, k, e, act = case["tokens"], case["top_k"], case["experts"], case["act"]
    train = case["mode"] in ("train", "train_sgd")
    x = v["x"].double()
    gw, gb = v["gate.weight"].double().requires_grad_(train), v["gate.bias"].double().requires_grad_(train)
    xr = x.clone().requires_grad_(train)
    top, idx = (xr @ gw.t() + gb).topk(k, dim=1)
    score = torch.softmax(top, dim=1)
    slots = t * k
    cap = min(slots, math.ceil(case["cf"] * slots / e)) if case["cf"] else slots
    # rows beyond an expert's capacity, counted in token-major slot order, are dropped
    onehot = torch.nn.functional.one_hot(idx.reshape(-1), e)
    keep = ((onehot.cumsum(0) - 1).gather(1, idx.reshape(-1, 1)).squeeze(1) < cap).view(t, k)
    del onehot
    y = torch.zeros_like(x)
    dx = torch.zeros_like(x)
    dscore = torch.zeros(t, k, dtype=torch.float64, device="cuda")
    names = [n for n in ("w1", "b1", "wg", "bg", "w2", "b2") if n in v]
    sgd = case["mode"] == "train_sgd"
    grads = {n: torch.empty_like(v[n], dtype=torch.float64 if v[n].dim() < 3 or v[n].numel() < 1 << 28 else torch.float32)
             for n in names} if train else {}
    for i in range(e):
        tok, slot = ((idx == i) & keep).nonzero(as_tuple=True)
        p = {n: v[n][i].double().requires_grad_(train) for n in names}
        xe = x[tok].requires_grad_(train)
        s = score.detach()[tok, slot].requires_grad_(train)
        h = xe @ p["w1"].t() + p["b1"]
        if act == "swiglu":
            h = torch.nn.functional.silu(xe @ p["wg"].t() + p["bg"]) * h
        else:
            h = torch.nn.functional.gelu(h) if act == "gelu" else torch.relu(h)
        o = (h @ p["w2"].t() + p["b2"]) * s.unsqueeze(1)
        y.index_add_(0, tok, o.detach())
        if train:
            got = torch.autograd.grad(o, [xe, s] + [p[n] for n in names], v["dy"][tok].double())
            dx.index_add_(0, tok, got[0])
            dscore[tok, slot] = got[1]
            for n, gr in zip(names, got[2:]):
                grads[n][i] = p[n].detach() - SGD_LR * gr if sgd and n[0] == "w" else gr
        del p, h, o
    if not train:
        return y
    dxr, dgw, dgb = torch.autograd.grad(score, (xr, gw, gb), dscore)
    out = {"y": y, "dx": dx + dxr, "dgate.weight": dgw, "dgate.bias": dgb}
    for n in names:
        out[n if sgd and n[0] == "w" else "d" + n] = grads[n]
    return out
