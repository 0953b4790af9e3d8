"""Performance cases of the framework: what a user's program has it do, through `lf.*`.

`listed()` holds the named workloads, `draw(rng)` gives another one of the same ranges.  A case
is a dict of plain values; `prepare(case, seed)` builds what such a program keeps between calls
(model, optimizer, captured step, inputs), `run(state)` is one call, `work(case)` the bytes and
operations that call cannot do without, `tolerance(case)` how far two correct implementations
at the same precision may be apart.

Kinds:
  xor       XOR network step on the GPU: four samples, MSE, Adam.  Pure latency.
  mlp       classifier step: Linear-ReLU-Dropout-Linear, cross entropy, Adam; `bf16` trains
            through DDP (bf16 compute, fp32 master), otherwise the plain fp32 loop of a program
            that only moved its model to the GPU.
  conv      three-layer convolution net step under DDP, SGD with momentum.
  gpt       GPT training step under DDP, AdamW, `graph` replays it as one captured graph.
  block     transformer block forward + backward (the unit of the larger models).
  attention multi-head attention module forward + backward, lengths off the tile grid.
  score     GPT forward without gradients over whole prompts (prefill, evaluation): all logits.
  generate  GPT sampling, one token after another (decode).
  matmul    Tensor.matmul of two matrices, fp32 or bf16, any size.
  rows      the Tensor ops of a hand-written layer over [rows, cols]: layer norm, GELU + bias,
            softmax, product, column sum.
"""
from __future__ import annotations

import math

import torch

import luatorch_b200 as lf

VOCAB = 50257          # the vocabulary of the GPT configurations


def listed():
    return [
        # tools/xor_benchmark on the GPU: the smallest training step there is
        {"name": "xor_step", "kind": "xor", "hidden": 16, "batch": 4, "graph": False},
        # train/mlp: the quick-start classifier, data-parallel engine, eager launches
        {"name": "mlp_step_bf16", "kind": "mlp", "batch": 256, "inputs": 784, "hidden": 256,
         "classes": 10, "dropout": 0.2, "bf16": True, "graph": False},
        # the same classifier in a plain fp32 loop (model.cuda(), Adam), as a first program has it
        {"name": "mlp_step_fp32", "kind": "mlp", "batch": 256, "inputs": 784, "hidden": 256,
         "classes": 10, "dropout": 0.0, "bf16": False, "graph": False},
        # train/convnet: 3x32x32 images, batch 128, SGD momentum, replayed as a graph
        {"name": "convnet_step", "kind": "conv", "batch": 128, "graph": True},
        # train/gpt preset "small" (character level), eager launches
        {"name": "gpt_small_step", "kind": "gpt", "vocab": 256, "embed": 384, "heads": 6, "layers": 6,
         "seq": 128, "batch": 4, "graph": False},
        # bench.py's configuration: the headline training step
        {"name": "gpt124m_step", "kind": "gpt", "vocab": VOCAB, "embed": 768, "heads": 12, "layers": 12,
         "seq": 1024, "batch": 8, "graph": True},
        # one of the 24 blocks of the 1.3B configuration (head dim 128)
        {"name": "block_e2048_s2048", "kind": "block", "embed": 2048, "heads": 16, "seq": 2048, "batch": 4},
        # attention over sequences whose length is no multiple of a tile
        {"name": "attention_s1000", "kind": "attention", "embed": 768, "heads": 12, "seq": 1000, "batch": 4,
         "causal": True},
        # scoring a few prompts of odd length with the 124M configuration
        {"name": "gpt124m_score_s777", "kind": "score", "vocab": VOCAB, "embed": 768, "heads": 12,
         "layers": 12, "seq": 777, "batch": 3},
        # sampling a reply with the 124M configuration: temperature and top-k of train/gpt
        {"name": "gpt124m_generate", "kind": "generate", "vocab": VOCAB, "embed": 768, "heads": 12,
         "layers": 12, "prompt": 100, "tokens": 24},
        # fp32 matrices of generic odd sizes: the Tensor front end's default type
        {"name": "matmul_fp32_odd", "kind": "matmul", "m": 1021, "n": 1333, "k": 777, "bf16": False},
        # hand-written layer over fp32 rows
        {"name": "row_ops_fp32", "kind": "rows", "rows": 4096, "cols": 1000, "bf16": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["xor", "mlp", "mlp", "conv", "gpt", "gpt", "block", "attention", "attention",
                       "score", "generate", "matmul", "matmul", "rows", "rows"])
    if kind == "xor":
        return {"kind": kind, "hidden": _log_int(rng, 4, 256), "batch": _log_int(rng, 4, 64),
                "graph": rng.random() < 0.3}
    if kind == "mlp":
        bf16 = rng.random() < 0.6
        return {"kind": kind, "batch": _log_int(rng, 16, 4096), "inputs": _log_int(rng, 30, 2000),
                "hidden": _log_int(rng, 32, 2048), "classes": _log_int(rng, 2, 1000),
                "dropout": rng.choice([0.0, 0.2, 0.5]), "bf16": bf16, "graph": bf16 and rng.random() < 0.3}
    if kind == "conv":
        return {"kind": kind, "batch": _log_int(rng, 8, 512), "graph": rng.random() < 0.5}
    if kind == "gpt":
        heads = rng.randint(2, 12)
        return {"kind": kind, "vocab": _log_int(rng, 100, VOCAB), "embed": 64 * heads, "heads": heads,
                "layers": rng.randint(2, 8), "seq": _log_int(rng, 32, 1024), "batch": rng.randint(1, 8),
                "graph": rng.random() < 0.5}
    if kind == "block":
        dim = rng.choice([64, 128])
        heads = _log_int(rng, 2, 2048 // dim)
        return {"kind": kind, "embed": dim * heads, "heads": heads, "seq": _log_int(rng, 64, 2048),
                "batch": rng.randint(1, 4)}
    if kind == "attention":
        dim = rng.choice([64, 64, 128])
        heads = rng.randint(2, 1536 // dim)
        return {"kind": kind, "embed": dim * heads, "heads": heads, "seq": _log_int(rng, 33, 2048),
                "batch": rng.randint(1, 8), "causal": rng.random() < 0.7}
    if kind in ("score", "generate"):
        heads = rng.randint(4, 12)
        case = {"kind": kind, "vocab": _log_int(rng, 100, VOCAB), "embed": 64 * heads, "heads": heads,
                "layers": rng.randint(2, 12)}
        if kind == "score":
            case.update(seq=_log_int(rng, 10, 1024), batch=rng.randint(1, 8))
        else:
            case.update(prompt=_log_int(rng, 4, 700), tokens=rng.randint(4, 40))
        return case
    if kind == "matmul":
        return {"kind": kind, "m": _log_int(rng, 16, 4096), "n": _log_int(rng, 16, 4096),
                "k": _log_int(rng, 16, 4096), "bf16": rng.random() < 0.5}
    return {"kind": "rows", "rows": _log_int(rng, 16, 16384), "cols": _log_int(rng, 32, 4096),
            "bf16": rng.random() < 0.5}


# ------------------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _normal(g, *shape, dtype=torch.float32, scale=1.0):
    return (torch.randn(*shape, generator=g, device="cuda") * scale).to(dtype)


def _labels(g, n, classes):
    return torch.randint(0, classes, (n,), generator=g, device="cuda")


class _ConvNet(lf.nn.Module):
    """Conv2d(3,32,3,1,1)-ReLU-Conv2d(32,64,3,2,1)-ReLU-Conv2d(64,128,3,2,1)-ReLU-Linear(8192,10)."""

    def __init__(self):
        nn = lf.nn
        self.c1, self.c2, self.c3 = nn.Conv2d(3, 32, 3, 1, 1), nn.Conv2d(32, 64, 3, 2, 1), nn.Conv2d(64, 128, 3, 2, 1)
        self.fc = nn.Linear(8192, 10, pad_out=True)

    def children(self):
        return [self.c1, self.c2, self.c3, self.fc]

    def parameters(self):
        return [p for c in self.children() for p in c.parameters()]

    def forward(self, x, batch):
        nn, ag = lf.nn, lf.autograd
        h, oh, ow = self.c1(x, batch, 32, 32, act="relu")
        h = nn.to_nchw(h, batch, 32, oh * ow)
        h, oh, ow = self.c2(h, batch, oh, ow, act="relu")
        h = nn.to_nchw(h, batch, 64, oh * ow)
        h, oh, ow = self.c3(h, batch, oh, ow, act="relu")
        h = nn.to_nchw(h, batch, 128, oh * ow)
        flat = lf.Tensor.wrap(h._t.reshape(batch, 8192))
        ag.record("flatten", [h], flat, lambda g: ag.acc_grad(h, g._t.reshape(h._t.shape)))
        return self.fc(flat)


class _Attention(lf.nn.Module):
    """A model that holds one attention layer."""

    def __init__(self, embed, heads, causal):
        self.attn = lf.nn.FlashMultiHeadAttention(embed, heads, causal)

    def children(self):
        return [self.attn]

    def parameters(self):
        return self.attn.parameters()

    def forward(self, x, seq_len):
        return self.attn(x, seq_len=seq_len)


def _train_state(case, forward, crit, opt, x, y, zero_grad, sync=None, pinned=None):
    """One training step over static inputs, eager or captured."""

    def step(xt=x, yt=y):
        lf.autograd.zero_graph()
        zero_grad()
        loss = crit(forward(xt), yt)
        lf.autograd.backward(loss)
        if sync is not None:
            sync()
        opt.step()
        return loss

    state = {"step": step, "opt": opt, "pinned": pinned}
    if case["graph"]:
        state["step"] = lf.cuda.GraphedStep(step, opt, inputs=(x, y), warmup=2)
    return state


def _arena_outputs(loss, opt):
    """The loss, and every parameter, gradient and optimizer moment as the step left them."""
    a = opt.arena
    out = {"loss": loss._t, "master": a.master, "grad": a.grad}
    for name in ("m_flat", "v_flat"):
        if hasattr(opt, name):
            out[name] = getattr(opt, name)
    return out


def prepare(case, seed):
    kind = case["kind"]
    lf.manual_seed(seed)
    g = _gen(seed)
    nn, T = lf.nn, lf.Tensor
    if kind == "xor":
        h, b = case["hidden"], case["batch"]
        model = nn.Sequential(nn.Linear(2, h), nn.Tanh(), nn.Linear(h, 1), nn.Sigmoid())
        arena = lf.cuda.amp.autocast_bf16(model)
        opt = lf.optim.Adam(model.parameters(), 0.05)
        bits = torch.randint(0, 2, (b, 2), generator=g, device="cuda")
        x, y = T.wrap(bits.float()), T.wrap((bits[:, :1] ^ bits[:, 1:]).float())
        return {**_train_state(case, model, nn.MSELoss(), opt, x, y, arena.zero_grad), "kind": kind}
    if kind == "mlp":
        model = nn.Sequential(nn.Linear(case["inputs"], case["hidden"]), nn.ReLU(), nn.Dropout(case["dropout"]),
                              nn.Linear(case["hidden"], case["classes"]))
        x = T.wrap(torch.rand(case["batch"], case["inputs"], generator=g, device="cuda"))
        y = T.wrap(_labels(g, case["batch"], case["classes"]).float())
        crit = nn.CrossEntropyLoss()
        if not case["bf16"]:
            model.cuda()
            opt = lf.optim.Adam(model.parameters(), 1e-3)
            return {**_train_state(case, model, crit, opt, x, y, model.zero_grad), "kind": kind, "model": model}
        ddp = lf.distributed.DDP(model, mode="auto")
        opt = lf.optim.Adam(ddp.parameters(), 1e-3)
        ddp.attach(opt)
        return {**_train_state(case, ddp, crit, opt, x, y, ddp.zero_grad, ddp.sync_gradients), "kind": kind}
    if kind == "conv":
        b = case["batch"]
        model = _ConvNet()
        ddp = lf.distributed.DDP(model, mode="auto")
        opt = lf.optim.SGD(ddp.parameters(), 0.01, 0.9)
        ddp.attach(opt)
        x = T.wrap(_normal(g, b * 3 * 32 * 32))
        y = T.wrap(_labels(g, b, 10).float())
        return {**_train_state(case, lambda xt: model.forward(xt, b), nn.CrossEntropyLoss(), opt, x, y,
                               ddp.zero_grad, ddp.sync_gradients), "kind": kind}
    if kind == "gpt":
        v, b, s = case["vocab"], case["batch"], case["seq"]
        model = lf.models.GPT(v, case["embed"], case["heads"], case["layers"], s, 0.0, pos="learned")
        ddp = lf.distributed.DDP(model)
        opt = lf.optim.AdamW(ddp.parameters(), 6e-4, 0.9, 0.95, 1e-8, 0.1, model.no_decay_params())
        ddp.attach(opt)
        # the batch waits in pinned host memory, as a data loader leaves it
        tok = torch.randint(0, v, (b, s + 1), generator=g, device="cuda").to(torch.int32).cpu()
        x, y = tok[:, :-1].contiguous().pin_memory(), tok[:, 1:].reshape(-1).contiguous().pin_memory()
        return {**_train_state(case, ddp, nn.CrossEntropyLoss(v, inplace_backward=True), opt, T.wrap(x.cuda()),
                               T.wrap(y.cuda()), ddp.zero_grad, ddp.sync_gradients, pinned=(x, y)), "kind": kind}
    if kind in ("block", "attention"):
        e, s, b = case["embed"], case["seq"], case["batch"]
        if kind == "block":
            model = nn.TransformerBlock(e, case["heads"], 0.0)
        else:
            model = _Attention(e, case["heads"], case["causal"])
        ddp = lf.distributed.DDP(model)
        x = lf.autograd.watch(T.wrap(_normal(g, b * s, e, dtype=torch.bfloat16)))
        dy = T.wrap(_normal(g, b * s, e, dtype=torch.bfloat16, scale=0.01))
        return {"kind": kind, "ddp": ddp, "x": x, "dy": dy, "seq": s}
    if kind in ("score", "generate"):
        v = case["vocab"]
        model = lf.models.GPT(v, case["embed"], case["heads"], case["layers"], 1024, 0.0, pos="learned")
        _as_if_trained(model)
        lf.cuda.amp.autocast_bf16(model)
        model.eval()
        if kind == "score":
            ids = torch.randint(0, v, (case["batch"], case["seq"]), generator=g, device="cuda").to(torch.int32)
            return {"kind": kind, "model": model, "ids": T.wrap(ids)}
        ids = torch.randint(0, v, (case["prompt"],), generator=g, device="cuda").float().cpu()
        return {"kind": kind, "model": model, "ids": T.wrap(ids), "tokens": case["tokens"],
                "top_k": min(40, v - 1), "seed": seed}
    dt = torch.bfloat16 if case["bf16"] else torch.float32
    if kind == "matmul":
        return {"kind": kind, "a": T.wrap(_normal(g, case["m"], case["k"], dtype=dt)),
                "b": T.wrap(_normal(g, case["k"], case["n"], dtype=dt))}
    r, c = case["rows"], case["cols"]
    return {"kind": kind, "x": T.wrap(_normal(g, r, c, dtype=dt)),
            "gamma": T.wrap(1 + _normal(g, c, dtype=dt, scale=0.1)), "beta": T.wrap(_normal(g, c, dtype=dt, scale=0.1)),
            "bias": T.wrap(_normal(g, c, dtype=dt))}


def _as_if_trained(model):
    """Random weights with the two traits of a trained language model that matter here: residual
    branches that add to the stream instead of drowning it, and a next-token distribution with
    a clear favourite (the head's column of a token resembles the embedding of the token before
    it), so that a sampled text does not hang on the last bit of a logit."""
    n = len(model.blocks)
    for blk in model.blocks:
        for lin in (blk.attn.out_proj, blk.ffn2):
            lin.weight._t.mul_((2 * n) ** -0.5)
    emb = model.token_emb.weight._t
    emb.mul_(50.0)
    model.head.weight._t.copy_(emb.roll(1, 0).t() * (23.0 / emb.shape[1]))


# ------------------------------------------------------------------------------ one pass
def run(state):
    kind = state["kind"]
    T = lf.Tensor
    if kind in ("xor", "mlp", "conv"):
        loss = state["step"]()
        if state["opt"].arena is not None:
            return _arena_outputs(loss, state["opt"])
        params = state["model"].parameters()
        return {"loss": loss._t, "params": [p._t for p in params], "grads": [p.grad._t for p in params],
                "m": state["opt"].m, "v": state["opt"].v}
    if kind == "gpt":
        x, y = state["pinned"]
        if not isinstance(state["step"], lf.cuda.GraphedStep):
            x, y = (T.wrap(t.to("cuda", non_blocking=True)) for t in (x, y))
        return _arena_outputs(state["step"](x, y), state["opt"])
    if kind in ("block", "attention"):
        ddp, x = state["ddp"], state["x"]
        lf.autograd.zero_graph()
        ddp.zero_grad()
        x.grad = None
        out = ddp(x, state["seq"])
        lf.autograd.backward(out, state["dy"])
        return {"out": out._t, "dx": x.grad._t, "grad": ddp.arena.grad}
    if kind == "score":
        with lf.autograd.no_grad():
            return state["model"](state["ids"])._t
    if kind == "generate":
        lf.manual_seed(state["seed"])
        return state["model"].generate(state["ids"], state["tokens"], 0.8, state["top_k"])._t
    if kind == "matmul":
        return T.matmul(state["a"], state["b"])._t
    x = state["x"]
    y = T.fused_layernorm(x, state["gamma"], state["beta"])
    z = T.fused_gelu_bias(y, state["bias"])
    p = T.softmax(z)
    q = T.mul(p, x)
    return {"norm": y._t, "act": z._t, "soft": p._t, "prod": q._t, "colsum": T.add_broadcast_backward(q)._t}


# ------------------------------------------------------------------------------ work and tolerance
def _gpt_params(case, positions):
    e = case["embed"]
    per_block = 12 * e * e + 10 * e
    return case["layers"] * per_block, case["vocab"] * e, positions * e + 2 * e


def work(case):
    kind = case["kind"]
    if kind == "xor":
        h, b = case["hidden"], case["batch"]
        n = 4 * h + 1
        return {"bytes": 28.0 * n + 12.0 * b, "flops": 6.0 * b * 3 * h}
    if kind == "mlp":
        b, i, h, c = case["batch"], case["inputs"], case["hidden"], case["classes"]
        n = i * h + h + h * c + c
        # fp32: parameter, both moments in and out, gradient out; bf16 adds the shadow weights
        return {"bytes": (28.0 + 2.0 * case["bf16"]) * n + 4.0 * b * (i + 1),
                "flops": 2.0 * b * (2 * i * h + 3 * h * c)}
    if kind == "conv":
        b = case["batch"]
        n = 27 * 32 + 32 + 288 * 64 + 64 + 576 * 128 + 128 + 81920 + 10
        macs = 1024 * 27 * 32 * 2 + 256 * 288 * 64 * 3 + 64 * 576 * 128 * 3 + 81920 * 3
        return {"bytes": 22.0 * n + 4.0 * b * (3072 + 1), "flops": 2.0 * b * macs}
    if kind == "gpt":
        t = case["batch"] * case["seq"]
        blocks, table, rest = _gpt_params(case, case["seq"])
        n = blocks + 2 * table + rest
        attn = 7.0 * t * case["seq"] * case["embed"] * case["layers"]
        return {"bytes": 28.0 * n + 8.0 * t, "flops": 6.0 * t * (blocks + table) + attn}
    if kind in ("block", "attention"):
        e, t = case["embed"], case["batch"] * case["seq"]
        n = (12 if kind == "block" else 4) * e * e
        attn = 7.0 * t * case["seq"] * e * (1 if case.get("causal", True) else 2)
        return {"bytes": 4.0 * n + 8.0 * t * e, "flops": 6.0 * t * n + attn}
    if kind == "score":
        t = case["batch"] * case["seq"]
        blocks, table, _ = _gpt_params(case, 1024)
        return {"bytes": 2.0 * (blocks + table) + 2.0 * t * (case["vocab"] + case["embed"]),
                "flops": 2.0 * t * (blocks + table) + 2.0 * t * case["seq"] * case["embed"] * case["layers"]}
    if kind == "generate":
        blocks, table, _ = _gpt_params(case, 1024)
        new, p = case["tokens"], case["prompt"]
        # every token needs one pass over the weights; logits only of the last position
        return {"bytes": new * 2.0 * (blocks + table),
                "flops": 2.0 * (p + new) * blocks + 2.0 * new * table + 2.0 * (p + new) ** 2 * case["embed"] * case["layers"]}
    if kind == "matmul":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": (2.0 if case["bf16"] else 4.0) * (m * k + k * n + m * n), "flops": 2.0 * m * n * k}
    r, c = case["rows"], case["cols"]
    return {"bytes": (2.0 if case["bf16"] else 4.0) * (5.0 * r * c + 4 * c), "flops": 30.0 * r * c}


def tolerance(case):
    kind = case["kind"]
    if kind == "generate":
        return "exact"                     # token ids
    if kind == "matmul":
        # fp32 products come from bf16 hi + lo parts: about 16 bits of each operand
        return {"rel": 4e-3} if case["bf16"] else {"rel": 3e-5}
    if kind == "rows":
        return {"rel": 1e-2} if case["bf16"] else {"rel": 1e-5, "max": 1e-3}
    if kind == "mlp" and not case["bf16"]:
        # 16-bit operand parts again; a unit whose pre-activation is nearly zero may switch side
        return {"rel": 5e-3, "max": 0.3}
    # bf16 activations and gradients through several layers, and Adam's normalised update
    return {"rel": 2e-2}
