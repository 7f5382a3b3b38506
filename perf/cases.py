"""Workloads of the framework as a user's program runs them, through the public entry points, for timing and comparison.

listed() names the representative ones, draw() takes more from the same ranges.  prepare() makes what a program has in hand
before the call (weights, models, inputs), run() is one pass, work() what a pass cannot do without, exact() the same results in
64-bit torch arithmetic without this library's code.

Kinds:
  gpt        a small fp32 GPT-2-style stack composed of C-ABI calls (the reference's own use: a few kilobytes per matrix, where
             launches and latencies count), a prompt or one token against cached keys
  expr       one expression node with a reduction, a norm or a softmax over fp32 matrices
  attention  prefill attention over token-major q, k, v (bf16 on the tensor cores, f32 on the CUDA cores), causal or not,
             grouped-query or not
  kv_decode  one query token per sequence against a paged bf16 cache of ragged context lengths
  decode     the LLaMA-shape decoder: steps of a batch against a filled cache, token ids in, tokens and last logits out
  prefill    the LLaMA-shape decoder: one prompt into the paged cache
  prompt     a layer-list decoder (Zugolorn, Vagonex): one prompt, logits of a few positions as a trace replay asks for them
  serve      a layer-list decoder: a batch of short prompts in one step, then one token per sequence and step
"""
import math

import numpy as np
import torch

import jasmine_b200 as jb
from jasmine_b200.decoder import vagonex_model, zugolorn_model
from jasmine_b200.model import Llama

DEV = "cuda"
EPS = 1e-5
BF16, F32 = torch.bfloat16, torch.float32
LEAF0, LEAF1 = (jb.OP_LEAF, 0), (jb.OP_LEAF, 1)
AXPB = [LEAF0, (jb.OP_IMM, 0.125), (jb.OP_MUL,), LEAF1, (jb.OP_ADD,)]


def listed():
    return [
        # the reference's own scale: a 64-token prompt through two layers of width 128
        {"name": "gpt_small", "kind": "gpt", "layers": 2, "width": 128, "heads": 4, "vocab": 256, "tokens": 64, "past": 0},
        # fused attention-score softmax of a 4096 x 4096 expression
        {"name": "softmax_rows", "kind": "expr", "op": "softmax", "rows": 4096, "cols": 4096},
        # long prompts, 32 heads of 128
        {"name": "flash_4096", "kind": "attention", "dtype": "bf16", "batch": 4, "tokens": 4096, "heads": 32, "kv_heads": 32, "dim": 128, "causal": True},
        # grouped-query decode attention of 64 sequences with contexts from 512 to 8192
        {"name": "kv_decode_64", "kind": "kv_decode", "batch": 64, "heads": 32, "kv_heads": 8, "low": 512, "high": 8192},
        # interactive generation: one sequence, the shape of a 7B model with eight of its layers
        {"name": "llama_decode_1", "kind": "decode", "layers": 8, "width": 4096, "heads": 32, "kv_heads": 32, "vocab": 32000, "batch": 1, "context": 512, "steps": 8},
        # a small batch of the same model: the headline workload
        {"name": "llama_decode_8", "kind": "decode", "layers": 8, "width": 4096, "heads": 32, "kv_heads": 32, "vocab": 32000, "batch": 8, "context": 512, "steps": 8},
        # a 512-token prompt of the same model
        {"name": "llama_prefill_512", "kind": "prefill", "layers": 8, "width": 4096, "heads": 32, "kv_heads": 32, "vocab": 32000, "tokens": 512},
        # a long prompt: latent attention with feed-forward, selective scan
        {"name": "zugolorn_prompt_2048", "kind": "prompt", "design": "zugolorn", "dtype": "bfloat16", "layers": 2, "width": 4096, "vocab": 32000, "tokens": 2048},
        # eight conversations at a time
        {"name": "zugolorn_serve_8", "kind": "serve", "design": "zugolorn", "dtype": "bfloat16", "layers": 4, "width": 2048, "vocab": 32000, "batch": 8, "tokens": 96, "steps": 48},
        # a long prompt: delta rule, decayed sum, chunked attention, each with feed-forward
        {"name": "vagonex_prompt_2048", "kind": "prompt", "design": "vagonex", "dtype": "bfloat16", "layers": 4, "width": 2048, "vocab": 32000, "tokens": 2048},
        # a full batch
        {"name": "vagonex_serve_64", "kind": "serve", "design": "vagonex", "dtype": "bfloat16", "layers": 4, "width": 2048, "vocab": 32000, "batch": 64, "tokens": 32, "steps": 24},
        # an f32 model of ragged sizes, as a trace is replayed for reference logits
        {"name": "vagonex_f32_300", "kind": "prompt", "design": "vagonex", "dtype": "float32", "layers": 4, "width": 1024, "vocab": 8000, "tokens": 300},
    ]


def _log(rng, low, high):
    """A whole number between low and high, spread over its logarithm."""
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choice(["gpt", "expr", "attention", "kv_decode", "decode", "prefill", "prompt", "prompt", "serve"])
    if kind == "gpt":
        width = rng.choice([64, 128, 256, 512])
        past = rng.choice([0, _log(rng, 1, 200)])
        return {"kind": kind, "layers": rng.randint(1, 4), "width": width, "heads": rng.choice([2, 4, 8]), "vocab": rng.choice([101, 256, 1000]),
                "tokens": 1 if past else _log(rng, 2, 256), "past": past}
    if kind == "expr":
        return {"kind": kind, "op": rng.choice(["softmax", "layernorm", "rmsnorm", "sum", "elementwise", "layernorm_columns"]),
                "rows": _log(rng, 16, 4096), "cols": _log(rng, 16, 4096)}
    if kind == "attention":
        if rng.random() < 0.3:
            return {"kind": kind, "dtype": "f32", "batch": rng.randint(1, 4), "tokens": _log(rng, 8, 700), "heads": 4, "kv_heads": rng.choice([1, 2, 4]),
                    "dim": rng.choice([16, 32, 64, 80, 128]), "causal": rng.random() < 0.8}
        heads = rng.choice([8, 16, 32])
        return {"kind": kind, "dtype": "bf16", "batch": rng.randint(1, 4), "tokens": _log(rng, 128, 4096), "heads": heads,
                "kv_heads": heads // rng.choice([1, 4]), "dim": 128, "causal": rng.random() < 0.8}
    if kind == "kv_decode":
        heads = rng.choice([16, 32])
        low = _log(rng, 16, 2000)
        return {"kind": kind, "batch": _log(rng, 1, 64), "heads": heads, "kv_heads": heads // rng.choice([1, 2, 4, 8]), "low": low, "high": min(8192, low * rng.randint(1, 16))}
    if kind in ("decode", "prefill"):
        width = rng.choice([1024, 2048, 4096])
        c = {"kind": kind, "layers": rng.randint(1, 4), "width": width, "heads": width // 128, "kv_heads": width // 128 // rng.choice([1, 4]), "vocab": rng.choice([8000, 32000])}
        if kind == "prefill":
            return {**c, "tokens": _log(rng, 24, 512)}
        return {**c, "batch": _log(rng, 1, 64), "context": _log(rng, 16, 512), "steps": rng.randint(4, 8)}
    design = rng.choice(["zugolorn", "vagonex"])
    dtype = "float32" if rng.random() < 0.25 else "bfloat16"
    c = {"kind": kind, "design": design, "dtype": dtype, "layers": rng.randint(2, 4), "width": rng.choice([512, 1024] if dtype == "float32" else [1024, 1536, 2048]),
         "vocab": rng.choice([8000, 32000]) if dtype == "bfloat16" else 8000}
    if kind == "prompt":
        return {**c, "tokens": _log(rng, 8, 300 if dtype == "float32" else 2048)}
    return {**c, "batch": _log(rng, 1, 64 if dtype == "bfloat16" else 8), "tokens": _log(rng, 4, 128 if dtype == "bfloat16" else 32), "steps": rng.randint(8, 24)}


# ---- inputs -----------------------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(1000003 * (int(seed) + 1))


def _randn(g, shape, std=1.0, mean=0.0, dtype=F32):
    return (torch.randn(shape, generator=g, device=DEV) * std + mean).to(dtype)


def _ids(g, shape, vocab):
    return torch.randint(0, vocab, shape, generator=g, device=DEV, dtype=torch.int32)


def _ffn(width):
    return width * 43 // 16


def _model_config(case):
    """A layer-list configuration with the proportions of a real model: heads of 128, feed-forward 43/16 of the width."""
    w, heads = case["width"], max(2, case["width"] // 128)
    base = {"width": w, "vocab": case["vocab"], "norm": {"eps": EPS}}
    if case["design"] == "zugolorn":
        attn = {"type": "latent_attention",
                "mixer": {"heads": heads, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": min(512, w // 4), "mask": {"size": 1024},
                          "rot": {"base": 10000.0, "dims": 64}, "scale": 192 ** -0.5},
                "mlp": {"kind": "dense", "ff": _ffn(w), "limit": 7.0}}
        scan = {"type": "mamba1", "mixer": {"inner": 2 * w, "state": 16, "dt_rank": w // 16, "conv": 4}, "mlp": None}
        return {**base, "architecture": "Zugolorn", "logit_softcap": 30.0, "layers": ([attn, scan] * 4)[:case["layers"]]}
    ff = {"kind": "dense", "ff": _ffn(w)}
    delta = {"type": "delta", "mixer": {"heads": heads, "kv_heads": heads // 2, "dim": 128, "vdim": 128, "conv": 4}, "mlp": ff}
    light = {"type": "lightning", "mixer": {"heads": heads, "dim": 128, "vdim": 128, "decay": [1.0 - 2.0 ** (-3 - 7 * h / heads) for h in range(heads)]}, "mlp": ff}
    attn = {"type": "attention",
            "mixer": {"heads": heads, "kv_heads": max(1, heads // 4), "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 1024},
                      "rot": {"base": 10000.0, "dims": 64, "scaling": {"factor": 4.0, "fast": 32.0, "slow": 1.0, "original": 4096}}}, "mlp": ff}
    return {**base, "architecture": "Vagonex", "postln_alpha": 2.0, "embedding": {"scale": 1.0}, "layers": ([delta, light, attn] + [delta] * 8)[:case["layers"]]}


def _decoder_weights(cfg, g):
    """(name, bf16 tensor) of every tensor of a layer-list model."""
    d = cfg["width"]

    def mat(rows, cols, gain=1.0):
        return _randn(g, (rows, cols), gain * cols ** -0.5, dtype=BF16)

    def vec(n, std, mean=0.0):
        return _randn(g, (n,), std, mean, BF16)

    yield "embed", _randn(g, (cfg["vocab"], d), 1.0, dtype=BF16)
    yield "final.norm", vec(d, 0.1, 1.0)
    for i, e in enumerate(cfg["layers"]):
        p, x, m = f"l{i}.", f"l{i}.mix.", e["mixer"]
        yield p + "norm1", vec(d, 0.05, 0.4)
        if e["type"] == "latent_attention":
            H, r = m["heads"], m["kv_rank"]
            yield x + "q", mat(H * (m["dim"] + m["rot_dim"]), d)
            yield x + "dkv", mat(r + m["rot_dim"], d)
            yield x + "dkv.norm", vec(r, 0.1, 1.0)
            yield x + "uk", mat(H * m["dim"], r)
            yield x + "uv", mat(H * m["vdim"], r)
            yield x + "o", mat(d, H * m["vdim"])
        elif e["type"] == "mamba1":
            c, n, R = m["inner"], m["state"], m["dt_rank"]
            yield x + "in", mat(2 * c, d)
            yield x + "conv", _randn(g, (c, m["conv"]), 0.5, dtype=BF16)
            yield x + "conv.b", vec(c, 0.1)
            yield x + "x", mat(R + 2 * n, c)
            yield x + "dt", mat(c, R)
            yield x + "dt.b", vec(c, 0.5, -4.0)
            yield x + "A_log", _randn(g, (c, n), 0.5, dtype=BF16)
            yield x + "D", vec(c, 0.1, 1.0)
            yield x + "o", mat(d, c)
        else:
            H, n, v = m["heads"], m["dim"], m["vdim"]
            G = m.get("kv_heads", H)
            yield x + "q", mat((G if e["type"] == "delta" else H) * n, d)
            yield x + "k", mat(G * n, d)
            yield x + "v", mat((G if e["type"] == "attention" else H) * v, d)
            yield x + "g", mat(H if e["type"] == "attention" else H * v, d)
            if e["type"] == "attention":
                yield x + "q.b", vec(H * n, 0.1)
                yield x + "q.norm", vec(n, 0.1, 1.0)
                yield x + "k.b", vec(G * n, 0.1)
                yield x + "k.norm", vec(n, 0.1, 1.0)
                yield x + "v.b", vec(G * v, 0.1)
                yield x + "sink", vec(H, 0.5)
            elif e["type"] == "lightning":
                yield x + "norm", vec(H * v, 0.1, 1.0)
            else:
                for s, rows in (("q", G * n), ("k", G * n), ("v", H * v)):
                    yield x + s + ".conv", _randn(g, (rows, m["conv"]), 0.5, dtype=BF16)
                yield x + "b", mat(H, d)
                yield x + "a", mat(H, d)
                yield x + "A_log", vec(H, 0.5)
                yield x + "dt_bias", vec(H, 0.5, -3.0)
                yield x + "norm", vec(v, 0.1, 1.0)
            yield x + "o", mat(d, H * v)
        if e["mlp"] is not None:
            f = e["mlp"]["ff"]
            yield p + "norm2", vec(d, 0.05, 0.4)
            yield p + "mlp.gate", mat(f, d)
            yield p + "mlp.up", mat(f, d)
            yield p + "mlp.down", mat(d, f)


def _decoder(case, seed):
    """The model, its token ids [batch, tokens + steps], prompt lengths and the generator's tensors."""
    cfg, g = _model_config(case), _gen(seed)
    batch, total = case.get("batch", 1), case["tokens"] + case.get("steps", 0)
    ids = _ids(g, (batch, total), case["vocab"]).cpu().numpy()
    # ragged prompts: from half of the length to all of it
    lens = [case["tokens"] - (case["tokens"] // 2 * b) // batch for b in range(batch)]
    make = zugolorn_model if case["design"] == "zugolorn" else vagonex_model
    m = make(cfg, dtype=case["dtype"], max_batch=batch, max_context=max(total, 64), max_step_tokens=2048)
    for name, t in _decoder_weights(cfg, g):
        m.set_weight(name, t.view(torch.int16).cpu().numpy().view(np.uint16))
    return m.finalize(), ids, lens


def _llama_tensors(case, g):
    d, f, hq, hkv = case["width"], _ffn(case["width"]), case["heads"] * 128, case["kv_heads"] * 128
    yield "emb", _randn(g, (case["vocab"], d), 1.0, dtype=BF16)
    yield "gf", _randn(g, (d,), 0.1, 1.0)
    yield "lm_head", _randn(g, (case["vocab"], d), d ** -0.5, dtype=BF16)
    for l in range(case["layers"]):
        yield f"layers.{l}.g1", _randn(g, (d,), 0.1, 1.0)
        yield f"layers.{l}.g2", _randn(g, (d,), 0.1, 1.0)
        yield f"layers.{l}.wqkv", _randn(g, (hq + 2 * hkv, d), d ** -0.5, dtype=BF16)
        yield f"layers.{l}.wo", _randn(g, (d, hq), 0.5 * hq ** -0.5, dtype=BF16)
        yield f"layers.{l}.wgu", _randn(g, (2 * f, d), d ** -0.5, dtype=BF16)
        yield f"layers.{l}.wdown", _randn(g, (d, f), 0.5 * f ** -0.5, dtype=BF16)


def _gpt_weights(case, g):
    d, f, n = case["width"], 4 * case["width"], case["past"] + case["tokens"]
    lin = lambda o, i: (_randn(g, (o, i), i ** -0.5), _randn(g, (1, o), 0.1))  # noqa: E731
    norm = lambda: (_randn(g, (d,), 0.1, 1.0), _randn(g, (d,), 0.1))  # noqa: E731
    return {"tok": _randn(g, (case["vocab"], d)), "pos": _randn(g, (n, d), 0.1), "lnf": norm(), "head": lin(case["vocab"], d),
            "layers": [{"ln1": norm(), "ln2": norm(), "q": lin(d, d), "k": lin(d, d), "v": lin(d, d), "o": lin(d, d), "w1": lin(f, d), "w2": lin(d, f),
                        "kc": _randn(g, (n, d)), "vc": _randn(g, (n, d))} for _ in range(case["layers"])]}


def prepare(case, seed):
    kind, g = case["kind"], _gen(seed)
    if kind == "gpt":
        w = _gpt_weights(case, g)
        T, past = case["tokens"], case["past"]
        return {"case": case, "w": w, "ids": _ids(g, (T,), case["vocab"]), "at": torch.arange(past, past + T, dtype=torch.int32, device=DEV)}
    if kind == "expr":
        R, C, op = case["rows"], case["cols"], case["op"]
        n = C if op != "layernorm_columns" else R
        s = {"case": case, "a": _randn(g, (R, C)), "b": _randn(g, (R, C)), "gain": _randn(g, (n,), 0.1, 1.0), "bias": _randn(g, (n,), 0.1)}
        return {**s, "out": torch.empty((R, 1) if op == "sum" else (R, C), device=DEV)}
    if kind == "attention":
        dt, rows, D = BF16 if case["dtype"] == "bf16" else F32, case["batch"] * case["tokens"], case["dim"]
        q = _randn(g, (rows, case["heads"] * D), dtype=dt)
        k, v = (_randn(g, (rows, case["kv_heads"] * D), dtype=dt) for _ in "kv")
        return {"case": case, "q": q, "k": k, "v": v, "out": torch.empty_like(q)}
    if kind == "kv_decode":
        n, Hq, Hkv = case["batch"], case["heads"], case["kv_heads"]
        lens = torch.randint(case["low"], case["high"] + 1, (n,), generator=g, device=DEV, dtype=torch.int32)
        pages = [-(-x // 64) for x in lens.tolist()]
        total, most = sum(pages), -(-case["high"] // 64)
        order = torch.randperm(total, generator=g, device=DEV).to(torch.int32)  # a pool in use hands its pages out in any order
        table, at = torch.zeros(n, most, dtype=torch.int32, device=DEV), 0
        for b, p in enumerate(pages):
            table[b, :p] = order[at:at + p]
            at += p
        pool = torch.empty(total, 2, Hkv, 64, 128, dtype=BF16, device=DEV)
        for p0 in range(0, total, 512):
            pool[p0:p0 + 512] = _randn(g, pool[p0:p0 + 512].shape, dtype=BF16)
        scratch = torch.empty(jb.lib().jsm_attn_decode_scratch_bytes(n, Hq, 128, case["high"]) // 4 + 4, device=DEV)
        q = _randn(g, (n, Hq * 128), dtype=BF16)
        return {"case": case, "q": q, "pool": pool, "table": table, "lens": lens, "scratch": scratch, "out": torch.empty_like(q)}
    if kind in ("decode", "prefill"):
        paged = kind == "prefill"
        batch, ctx, steps = case.get("batch", 1), case.get("context", 0), case.get("steps", 0)
        m = Llama(case["layers"], case["width"], case["heads"], case["kv_heads"], _ffn(case["width"]), case["vocab"], max_batch=batch, max_context=1024,
                  norm_eps=EPS, pool_pages=16 if paged else 0)
        for name, t in _llama_tensors(case, g):
            m.set_weight(name, t)
        stream = torch.cuda.Stream()
        torch.cuda.synchronize()
        logits = torch.empty(batch, case["vocab"]).pin_memory()
        if paged:
            return {"case": case, "m": m, "ids": _ids(g, (case["tokens"],), case["vocab"]).cpu(), "logits": logits, "stream": stream}
        ids = _ids(g, (batch, ctx + steps), case["vocab"])
        with torch.cuda.stream(stream):
            for b in range(batch):
                m.prefill(ids[b, :ctx].contiguous(), b)
        torch.cuda.synchronize()
        return {"case": case, "m": m, "ids": ids[:, ctx:].t().contiguous().cpu().pin_memory(), "next": torch.empty(batch, dtype=torch.int32).pin_memory(),
                "logits": logits, "stream": stream}
    m, ids, lens = _decoder(case, seed)
    rows = len(_wanted(case)) if kind == "prompt" else case["batch"]
    return {"case": case, "m": m, "ids": ids, "lens": lens, "next": np.empty(rows, np.int32), "logits": torch.empty(rows, case["vocab"]).pin_memory()}


def _wanted(case):
    """Places of a prompt whose logits are asked for: eight spread over it, the last among them."""
    T = case["tokens"]
    return sorted({T * (i + 1) // 8 - 1 for i in range(8)} - {-1})


# ---- one pass ---------------------------------------------------------------------------------------------------------
def _gpt_linear(x, wb, epilogue=0, residual=None, out=None):
    out = torch.empty(x.shape[0], wb[0].shape[0], device=DEV) if out is None else out
    return jb.dot_f32(x, wb[0].t(), out, bias=wb[1], epilogue=epilogue, residual=residual)


def _gpt_norm(x, gb):
    return jb.eval_rows(jb.ROWS_LAYERNORM, 1, [LEAF0], [x], torch.empty_like(x), gain=gb[0], bias=gb[1], eps=EPS)


def _run_gpt(s):
    c, w = s["case"], s["w"]
    H, d, p0, p1 = c["heads"], c["width"], c["past"], c["past"] + c["tokens"]
    x = jb.embedding(w["tok"], s["ids"], w["pos"], s["at"])
    for l in w["layers"]:
        n = _gpt_norm(x, l["ln1"])
        q = _gpt_linear(n, l["q"])
        _gpt_linear(n, l["k"], out=l["kc"][p0:p1])
        _gpt_linear(n, l["v"], out=l["vc"][p0:p1])
        a = jb.attn_prefill(q, l["kc"], l["vc"], 1, H, H, d // H)
        x = _gpt_linear(a, l["o"], 3, x)
        x = _gpt_linear(_gpt_linear(_gpt_norm(x, l["ln2"]), l["w1"], 2), l["w2"], 3, x)
    return _gpt_linear(_gpt_norm(x, w["lnf"]), w["head"])


def _run_expr(s):
    op, a, b, out = s["case"]["op"], s["a"], s["b"], s["out"]
    if op == "softmax":
        return jb.eval_rows(jb.ROWS_SOFTMAX, 1, AXPB, [a, b], out)
    if op == "layernorm":
        return jb.eval_rows(jb.ROWS_LAYERNORM, 1, [LEAF0, LEAF1, (jb.OP_ADD,)], [a, b], out, gain=s["gain"], bias=s["bias"], eps=EPS)
    if op == "layernorm_columns":
        return jb.eval_rows(jb.ROWS_LAYERNORM, 0, [LEAF0], [a], out, gain=s["gain"], bias=s["bias"], eps=EPS)
    if op == "rmsnorm":
        return jb.eval_rows(jb.ROWS_RMSNORM, 1, [LEAF0], [a], out, gain=s["gain"], eps=EPS)
    if op == "sum":
        return jb.eval_rows(jb.ROWS_SUM, 1, [LEAF0], [a], out)
    return jb.eval_elementwise(AXPB, [a, b], out)


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "gpt":
        return _run_gpt(s)
    if kind == "expr":
        return _run_expr(s)
    if kind == "attention":
        return jb.attn_prefill(s["q"], s["k"], s["v"], c["batch"], c["heads"], c["kv_heads"], c["dim"], causal=c["causal"], out=s["out"])
    if kind == "kv_decode":
        return jb.attn_decode(s["q"], s["pool"], s["table"], s["lens"], c["heads"], c["kv_heads"], 128, c["high"], scratch=s["scratch"], out=s["out"])
    m = s["m"]
    if kind == "prefill":
        with torch.cuda.stream(s["stream"]):
            row, _ = m.admit(s["ids"], s["logits"])
            m.retire(row)
        return s["logits"]
    if kind == "decode":
        with torch.cuda.stream(s["stream"]):
            for b in range(c["batch"]):
                m.set_context(b, c["context"])  # the sequences are rewound to the end of their prompts
            for k in range(c["steps"]):
                m.decode_step_host(s["ids"][k], s["next"], s["logits"] if k + 1 == c["steps"] else None)
        return s["logits"]
    if kind == "prompt":
        row = m.open()
        m.step([(row, s["ids"][0])], _wanted(c), s["next"], s["logits"])
        m.retire(row)
        return s["logits"]
    ids, lens = s["ids"], s["lens"]
    rows = [m.open() for _ in lens]
    ends = np.cumsum(lens) - 1
    m.step([(r, ids[r, :lens[r]]) for r in rows], ends, s["next"], logits=False)
    for k in range(c["steps"]):
        m.step_active(np.ascontiguousarray(ids[:, c["tokens"] + k]), s["next"], s["logits"] if k + 1 == c["steps"] else None)
    for r in reversed(rows):
        m.retire(r)
    return s["logits"]


# ---- what a pass cannot do without ------------------------------------------------------------------------------------
def _decoder_params(cfg):
    """Weights of the layers without the vocabulary, and multiply-adds of attention per token and visible key."""
    params, per_key, state = 0, 0, 0
    d = cfg["width"]
    for e in cfg["layers"]:
        m = e["mixer"]
        if e["type"] == "latent_attention":
            H, r = m["heads"], m["kv_rank"]
            params += d * (H * (m["dim"] + m["rot_dim"]) + r + m["rot_dim"] + H * m["vdim"]) + H * (m["dim"] + m["vdim"]) * r
            per_key += H * (m["dim"] + m["rot_dim"] + m["vdim"])
        elif e["type"] == "mamba1":
            c, n, R = m["inner"], m["state"], m["dt_rank"]
            params += 3 * c * d + c * (R + 2 * n) + c * R
            state += 3 * c * n
        else:
            H, n, v, G = m["heads"], m["dim"], m["vdim"], m.get("kv_heads", m["heads"])
            if e["type"] == "attention":
                params += d * (H * n + H + G * (n + v) + H * v)
                per_key += H * (n + v)
            else:
                params += d * ((2 * G * n if e["type"] == "delta" else 2 * H * n) + 3 * H * v)
                state += 3 * H * n * v
        if e["mlp"]:
            params += 3 * d * e["mlp"]["ff"]
    return params, per_key, state


def work(case):
    kind = case["kind"]
    if kind == "gpt":
        d, T, n = case["width"], case["tokens"], case["past"] + case["tokens"]
        params = case["layers"] * 12 * d * d + case["vocab"] * d
        return {"bytes": 4 * (params + case["layers"] * 2 * n * d + T * (d + case["vocab"])), "flops": 2 * T * params + case["layers"] * 4 * T * n * d // 2}
    if kind == "expr":
        n = 4 * case["rows"] * case["cols"]
        moved = {"softmax": 3 * n, "layernorm": 3 * n, "elementwise": 3 * n, "rmsnorm": 2 * n, "layernorm_columns": 2 * n, "sum": n}[case["op"]]
        return {"bytes": moved, "flops": 0}
    if kind == "attention":
        T, D, es = case["tokens"], case["dim"], 2 if case["dtype"] == "bf16" else 4
        return {"bytes": es * case["batch"] * T * D * 2 * (case["heads"] + case["kv_heads"]), "flops": 4 * case["batch"] * case["heads"] * T * T * D // (2 if case["causal"] else 1)}
    if kind == "kv_decode":
        keys = case["batch"] * (case["low"] + case["high"]) // 2
        return {"bytes": keys * case["kv_heads"] * 512 + 4 * case["batch"] * case["heads"] * 128, "flops": 4 * keys * case["heads"] * 128}
    if kind in ("decode", "prefill"):
        d, f, hq, hkv = case["width"], _ffn(case["width"]), case["heads"] * 128, case["kv_heads"] * 128
        layer, head = d * (2 * hq + 2 * hkv) + 3 * d * f, case["vocab"] * d
        if kind == "prefill":
            T = case["tokens"]
            return {"bytes": 2 * (case["layers"] * (layer + 2 * T * hkv) + head), "flops": 2 * case["layers"] * T * (layer + T * hq) + 2 * head}
        B, keys = case["batch"], case["context"] + case["steps"] // 2
        return {"bytes": 2 * case["steps"] * (case["layers"] * (layer + B * keys * 2 * hkv) + head),
                "flops": 2 * case["steps"] * B * (case["layers"] * (layer + 2 * keys * hq) + head)}
    cfg, es = _model_config(case), 2 if case["dtype"] == "bfloat16" else 4
    params, per_key, state = _decoder_params(cfg)
    head = cfg["vocab"] * cfg["width"]
    T = case["tokens"]
    flops = lambda tokens, keys, heads: 2 * tokens * (params + per_key * keys + state) + 2 * heads * head  # noqa: E731
    if kind == "prompt":
        return {"bytes": es * (params + head), "flops": flops(T, T / 2, len(_wanted(case)))}
    B, S = case["batch"], case["steps"]
    return {"bytes": (S + 1) * es * (params + head) + S * B * 8 * state / 3, "flops": flops(B * T * 3 // 4, T / 2, B) + flops(S * B, T, S * B)}


def tolerance(case):
    """About four times the distance from exact() that was measured for each kind."""
    kind = case["kind"]
    if kind in ("gpt", "expr"):
        return {"rel": 4e-6}
    if kind in ("attention", "kv_decode"):
        return {"rel": 2e-6} if case.get("dtype") == "f32" else {"rel": 1e-2, "max": 0.2}
    if kind in ("decode", "prefill"):
        return {"rel": 0.03, "max": 0.3}
    return {"rel": 0.02, "max": 0.2} if case["dtype"] == "bfloat16" else {"rel": 4e-6}


# ---- the same in 64 bits ----------------------------------------------------------------------------------------------
def _rms(x, w):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS) * w


def _layer_norm(x, gain, bias):
    c = x - x.mean(-1, keepdim=True)
    return c / torch.sqrt((c * c).mean(-1, keepdim=True) + EPS) * gain + bias


def _attend(q, k, v, scale, seen, sink=None):
    """q [T, H, n], k [S, G, n], v [S, G, m]; seen [T, S] or None; sink [H] joins the denominator."""
    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    out = torch.empty(T, H, v.shape[2], dtype=q.dtype, device=q.device)
    for h in range(H):
        s = q[:, h] @ k[:, h * G // H].t() * scale
        if seen is not None:
            s = s.masked_fill(~seen, -math.inf)
        top = s.max(1, keepdim=True).values
        if sink is not None:
            top = top.clamp(min=float(sink[h]))
        e = torch.exp(s - top)
        z = e.sum(1, keepdim=True)
        if sink is not None:
            z = z + torch.exp(sink[h] - top)
        out[:, h] = (e @ v[:, h * G // H]) / z
    return out


def _seen(T, window=0, chunk=0):
    i, j = torch.arange(T, device=DEV)[:, None], torch.arange(T, device=DEV)[None, :]
    m = j <= i
    if window:
        m &= i - j < window
    if chunk:
        m &= i // chunk == j // chunk
    return m


def _rotate(x, freq, half, magnitude=1.0):
    """Rotates the first 2 len(freq) components of [T, H, n]: pairs (i, i + len(freq)) if half, else (2i, 2i + 1)."""
    P = len(freq)
    a = torch.arange(x.shape[0], device=DEV, dtype=torch.float64)[:, None, None] * freq
    c, s = torch.cos(a) * magnitude, torch.sin(a) * magnitude
    out = x.clone()
    u, v = (slice(0, P), slice(P, 2 * P)) if half else (slice(0, 2 * P, 2), slice(1, 2 * P, 2))
    out[..., u] = x[..., u] * c - x[..., v] * s
    out[..., v] = x[..., u] * s + x[..., v] * c
    return out


def _freqs(n, base):
    return torch.tensor([float(base) ** (-2.0 * i / n) for i in range(n // 2)], device=DEV, dtype=torch.float64)


def _yarn(rot):
    n, base, sc = rot["dims"], rot["base"], rot["scaling"]
    turns = lambda t: n * math.log(sc["original"] / (2.0 * math.pi * t)) / (2.0 * math.log(base))  # noqa: E731
    lo, hi = max(math.floor(turns(sc["fast"])), 0), min(math.ceil(turns(sc["slow"])), n - 1)
    ramp = ((torch.arange(n // 2, device=DEV, dtype=torch.float64) - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
    f = _freqs(n, base)
    return f / sc["factor"] * ramp + f * (1.0 - ramp), 0.1 * math.log(sc["factor"]) + 1.0


def _silu(x):
    return x * torch.sigmoid(x)


def _conv(x, w, b=None):
    taps, T = w.shape[1], x.shape[0]
    p = torch.cat([torch.zeros(taps - 1, x.shape[1], device=DEV, dtype=x.dtype), x])
    out = sum(p[k:k + T] * w[:, k] for k in range(taps))
    return _silu(out if b is None else out + b)


def _mix_latent(x, w, m):
    T, H, n, r = x.shape[0], m["heads"], m["dim"], m["rot_dim"]
    f = _freqs(r, m["rot"]["base"])
    q = (x @ w["q"].t()).view(T, H, n + r)
    q = torch.cat([q[..., :n], _rotate(q[..., n:], f, True)], -1)
    down = x @ w["dkv"].t()
    c = _rms(down[:, :m["kv_rank"]], w["dkv.norm"])
    kr = _rotate(down[:, None, m["kv_rank"]:], f, True).expand(T, H, r)
    k = torch.cat([(c @ w["uk"].t()).view(T, H, n), kr], -1)
    v = (c @ w["uv"].t()).view(T, H, m["vdim"])
    return _attend(q, k, v, m["scale"], _seen(T, window=m["mask"]["size"])).reshape(T, -1) @ w["o"].t()


def _mix_scan(x, w, m):
    c, n, R = m["inner"], m["state"], m["dt_rank"]
    xz = x @ w["in"].t()
    u = _conv(xz[:, :c], w["conv"], w["conv.b"])
    p = u @ w["x"].t()
    dt = torch.nn.functional.softplus(p[:, :R] @ w["dt"].t() + w["dt.b"], threshold=1e9)
    A, S, y = -torch.exp(w["A_log"]), torch.zeros(c, n, device=DEV, dtype=x.dtype), torch.empty_like(u)
    for t in range(x.shape[0]):
        S = torch.exp(dt[t][:, None] * A) * S + (dt[t] * u[t])[:, None] * p[t, R:R + n]
        y[t] = S @ p[t, R + n:]
    return ((y + w["D"] * u) * _silu(xz[:, c:])) @ w["o"].t()


def _mix_attention(x, w, m):
    T, H, G, n = x.shape[0], m["heads"], m["kv_heads"], m["dim"]
    f, mag = _yarn(m["rot"])
    q = _rotate(_rms((x @ w["q"].t() + w["q.b"]).view(T, H, n), w["q.norm"]), f, False, mag)
    k = _rotate(_rms((x @ w["k"].t() + w["k.b"]).view(T, G, n), w["k.norm"]), f, False, mag)
    v = (x @ w["v"].t() + w["v.b"]).view(T, G, m["vdim"])
    o = _attend(q, k, v, m["scale"], _seen(T, chunk=m["mask"]["size"]), w["sink"]) * torch.sigmoid(x @ w["g"].t())[:, :, None]
    return o.reshape(T, -1) @ w["o"].t()


def _mix_recurrence(x, w, m, delta):
    T, H, n, v, G = x.shape[0], m["heads"], m["dim"], m["vdim"], m.get("kv_heads", m["heads"])
    if delta:
        unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
        q, k, u = (_conv(x @ w[s].t(), w[s + ".conv"]) for s in "qkv")
        q, k = (unit(t.view(T, G, n)).repeat_interleave(H // G, 1) for t in (q, k))
        q = q * n ** -0.5
        beta = torch.sigmoid(x @ w["b"].t())
        decay = torch.exp(-torch.exp(w["A_log"]) * torch.nn.functional.softplus(x @ w["a"].t() + w["dt_bias"], threshold=1e9))
    else:
        q, k, u = (_silu(x @ w[s].t()) for s in "qkv")
        q, k = q.view(T, H, n), k.view(T, H, n)
        decay = torch.tensor(m["decay"], device=DEV, dtype=F32).double().expand(T, H)
    u, S, o = u.view(T, H, v), torch.zeros(H, n, v, device=DEV, dtype=x.dtype), torch.empty(T, H, v, device=DEV, dtype=x.dtype)
    for t in range(T):
        S = S * decay[t][:, None, None]
        b = u[t]
        if delta:
            b = beta[t][:, None] * (b - torch.matmul(k[t][:, None], S)[:, 0])
        S = S + k[t][:, :, None] * b[:, None]
        o[t] = torch.matmul(q[t][:, None], S)[:, 0]
    z = x @ w["g"].t()
    if delta:
        o = _rms(o, w["norm"]).reshape(T, -1) * _silu(z)
    else:
        o = _rms(o.reshape(T, -1), w["norm"]) * torch.sigmoid(z)
    return o @ w["o"].t()


def _decoder_hidden(cfg, weights, ids):
    """Residual stream of a layer-list model behind its last layer."""
    vagonex = cfg["architecture"] == "Vagonex"
    alpha = cfg.get("postln_alpha")
    x = weights["embed"][torch.as_tensor(ids, device=DEV, dtype=torch.long)].double()
    join = (lambda x, y, w: _rms(alpha * x + y, w)) if vagonex else (lambda x, y, w: x + _rms(y, w))
    for i, e in enumerate(cfg["layers"]):
        w = {k[len(f"l{i}."):]: t.double() for k, t in weights.items() if k.startswith(f"l{i}.")}
        mix = {k[4:]: t for k, t in w.items() if k.startswith("mix.")}
        fn = {"latent_attention": _mix_latent, "mamba1": _mix_scan, "attention": _mix_attention}.get(e["type"])
        y = fn(x, mix, e["mixer"]) if fn else _mix_recurrence(x, mix, e["mixer"], e["type"] == "delta")
        x = join(x, y, w["norm1"])
        if e["mlp"]:
            gate, up = x @ w["mlp.gate"].t(), x @ w["mlp.up"].t()
            if vagonex:
                a = torch.nn.functional.gelu(gate, approximate="tanh") * up
            else:
                lim = e["mlp"]["limit"]
                gate = gate.clamp(max=lim)
                a = gate * torch.sigmoid(1.702 * gate) * (up.clamp(-lim, lim) + 1.0)
            x = join(x, a @ w["mlp.down"].t(), w["norm2"])
    return x


def _exact_decoder(case, seed):
    cfg, g = _model_config(case), _gen(seed)
    batch, total = case.get("batch", 1), case["tokens"] + case.get("steps", 0)
    ids = _ids(g, (batch, total), case["vocab"])
    lens = [case["tokens"] - (case["tokens"] // 2 * b) // batch for b in range(batch)]
    w = dict(_decoder_weights(cfg, g))
    last = []
    for b in range(batch):
        x = _decoder_hidden(cfg, w, torch.cat([ids[b, :lens[b]], ids[b, case["tokens"]:]]))
        last.append(x[_wanted(case)] if case["kind"] == "prompt" else x[-1:])
    y = _rms(torch.cat(last), w["final.norm"].double()) @ w["embed"].double().t()
    cap = cfg.get("logit_softcap")
    return cap * torch.tanh(y / cap) if cap else y


def _exact_llama(case, seed):
    g = _gen(seed)
    w = dict(_llama_tensors(case, g))
    d, f, Hq, Hkv = case["width"], _ffn(case["width"]), case["heads"], case["kv_heads"]
    if case["kind"] == "prefill":
        ids = _ids(g, (case["tokens"],), case["vocab"])[None]
    else:
        ids = _ids(g, (case["batch"], case["context"] + case["steps"]), case["vocab"])
    B, T = ids.shape
    freq, seen = _freqs(128, 10000.0), _seen(T)
    x = w["emb"][ids.long()].double()
    for l in range(case["layers"]):
        L = {k: w[f"layers.{l}.{k}"].double() for k in ("g1", "g2", "wqkv", "wo", "wgu", "wdown")}
        qkv = (_rms(x, L["g1"]) @ L["wqkv"].t()).view(B, T, Hq + 2 * Hkv, 128)
        a = torch.stack([_attend(_rotate(s[:, :Hq], freq, False), _rotate(s[:, Hq:Hq + Hkv], freq, False), s[:, Hq + Hkv:], 128 ** -0.5, seen) for s in qkv])
        x = x + a.reshape(B, T, -1) @ L["wo"].t()
        gu = _rms(x, L["g2"]) @ L["wgu"].t()
        x = x + (_silu(gu[..., :f]) * gu[..., f:]) @ L["wdown"].t()
    return (_rms(x[:, -1], w["gf"].double()) @ w["lm_head"].double().t())


def exact(case, seed):
    kind = case["kind"]
    if kind in ("prompt", "serve"):
        return _exact_decoder(case, seed)
    if kind in ("decode", "prefill"):
        return _exact_llama(case, seed)
    s = {k: v.double() if isinstance(v, torch.Tensor) and v.is_floating_point() else v for k, v in prepare(case, seed).items()}
    if kind == "expr":
        op, a, b, gain, bias = case["op"], s["a"], s["b"], s["gain"], s["bias"]
        if op == "softmax":
            return torch.softmax(a * 0.125 + b, 1)
        if op == "layernorm":
            return _layer_norm(a + b, gain, bias)
        if op == "layernorm_columns":
            return _layer_norm(a.t(), gain, bias).t().contiguous()
        if op == "rmsnorm":
            return _rms(a, gain)
        return a.sum(1, keepdim=True) if op == "sum" else a * 0.125 + b
    if kind == "attention":
        B, T, D = case["batch"], case["tokens"], case["dim"]
        q, k, v = (s[n].view(B, T, -1, D) for n in "qkv")
        seen = _seen(T) if case["causal"] else None
        return torch.stack([_attend(q[b], k[b], v[b], D ** -0.5, seen) for b in range(B)]).reshape(B * T, -1)
    if kind == "kv_decode":
        out = []
        for b, n in enumerate(s["lens"].tolist()):
            pages = s["pool"][s["table"][b, :-(-n // 64)].long()]  # [pages, 2, kv heads, 64, 128]
            k, v = (pages[:, i].transpose(1, 2).reshape(-1, case["kv_heads"], 128)[:n] for i in (0, 1))
            out.append(_attend(s["q"][b].view(1, -1, 128), k, v, 128 ** -0.5, None).reshape(-1))
        return torch.stack(out)
    up = lambda v: v.double() if isinstance(v, torch.Tensor) else {k: up(x) for k, x in v.items()} if isinstance(v, dict) else type(v)(up(x) for x in v)  # noqa: E731
    w, T, p0, H = up(s["w"]), case["tokens"], case["past"], case["heads"]
    lin = lambda x, wb: x @ wb[0].t() + wb[1]  # noqa: E731
    x = w["tok"][s["ids"].long()] + w["pos"][p0:p0 + T]
    seen = _seen(p0 + T)[p0:]
    for l in w["layers"]:
        n = _layer_norm(x, *l["ln1"])
        k, v = (torch.cat([l[c][:p0], lin(n, l[p])]).view(p0 + T, H, -1) for c, p in (("kc", "k"), ("vc", "v")))
        a = _attend(lin(n, l["q"]).view(T, H, -1), k, v, (case["width"] // H) ** -0.5, seen)
        x = x + lin(a.reshape(T, -1), l["o"])
        x = x + lin(torch.nn.functional.gelu(lin(_layer_norm(x, *l["ln2"]), l["w1"])), l["w2"])
    return lin(_layer_norm(x, *w["lnf"]), w["head"])
