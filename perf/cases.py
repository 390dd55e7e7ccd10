"""What this framework's users have it do, as cases that can be timed on one GPU.

A case is a dict of plain values; its ``kind`` names the public entry point that the pass goes through:

* ``graph_mlp``   ``TaskGraph``: SwiGLU MLP (two ``linear`` nodes), with ``block`` also the pre-norm and the residual add
                  around it; 16-bit, one row (a decode step of one sequence) to thousands (prefill, training forward)
* ``graph_fp32``  ``TaskGraph``: a chain of two fp32 ``linear`` nodes (the README's smallest graph)
* ``decode``      ``Qwen3DecodeLayer``: one decode step of a decoder layer over a filled KV cache
* ``moe``         ``MoEEPLayer``: routing, dispatch, experts, combine
* ``train``       ``DPMLPStackBackward``: forward and backward of a stack of linear + GELU layers
* ``attention``   ``ops.attention_decode``: over a cache that is exactly full (with ``out=``), or over the filled part of
                  a longer cache (a strided view, no ``out=``)
* ``rows``        row-wise and point-wise operators of ``ops``

``draw`` gives more cases of the same ranges. Weights of the model classes come from their own seeded constructors
(host generators), so their sizes are one GPU's share of a tensor- or expert-parallel layer rather than a whole one.
"""
from __future__ import annotations

import math

import torch

import maco_b200 as maco
from maco_b200 import ops

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def listed():
    return [
        # Smallest graph: two fp32 layers on 32 rows, the chain every first program of the API builds. Launches and
        # host work count here.
        dict(name="graph_fp32_chain_32", kind="graph_fp32", rows=32, d_in=512, d_mid=1024, d_out=512),
        # The benchmark's layer: prefill / training forward of an 8192-token SwiGLU MLP.
        dict(name="graph_mlp_8192", kind="graph_mlp", dtype="bf16", rows=8192, hidden=4096, ffn=14336, block=False),
        # The same layer in a decode step: 64 sequences, one token each; the weights stream through once.
        dict(name="graph_mlp_decode_64", kind="graph_mlp", dtype="bf16", rows=64, hidden=4096, ffn=14336, block=False),
        # A whole MLP block (norm, MLP, residual) on a ragged prompt of a smaller model, fp16.
        dict(name="graph_block_ragged_1003", kind="graph_mlp", dtype="fp16", rows=1003, hidden=2048, ffn=5504, block=True),
        # Decoder layer, decode step: one GPU's share (of four) of the benchmark's layer, batch 64 over 4096 cached keys.
        dict(name="decode_layer_b64", kind="decode", hidden=5120, q_heads=16, kv_heads=2, ffn=6400, batch=64, kv_len=4096),
        # The same step when few users are on: batch 3, a short ragged cache, a smaller layer.
        dict(name="decode_layer_b3", kind="decode", hidden=2048, q_heads=16, kv_heads=4, ffn=6144, batch=3, kv_len=701),
        # MoE layer at prefill: 4096 tokens, 64 experts, top-8.
        dict(name="moe_4096tok_64e", kind="moe", hidden=2048, experts=64, top_k=8, inter=768, tokens=4096),
        # MoE layer with few tokens per expert (small batches): bound by the experts' weights.
        dict(name="moe_256tok_32e", kind="moe", hidden=1024, experts=32, top_k=4, inter=512, tokens=256),
        # Training step of the data-parallel benchmark's stack (four of its layers): forward, then backward.
        dict(name="train_stack_4x4096", kind="train", layers=4, hidden=4096, tokens=8192),
        # Decode attention over full caches, grouped-query heads, 16 sequences of 8192 keys.
        dict(name="attention_b16_8192", kind="attention", dtype="bf16", batch=16, kv_heads=8, group=4, keys=8192, capacity=8192),
        # Decode attention over the filled, ragged part of a preallocated cache.
        dict(name="attention_view_1357", kind="attention", dtype="fp16", batch=4, kv_heads=4, group=8, keys=1357, capacity=4096),
        # Norm of a prompt's hidden states.
        dict(name="rmsnorm_8192x5120", kind="rows", op="rmsnorm", dtype="bf16", rows=8192, cols=5120),
    ]


def _log(rng, lo, hi, step=1):
    """An integer of [lo, hi], spread over the logarithm, a multiple of ``step``."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def draw(rng):
    kind = rng.choice(["graph_mlp", "graph_mlp", "graph_fp32", "decode", "moe", "train", "attention", "attention", "rows", "rows"])
    if kind == "graph_fp32":
        return dict(kind=kind, rows=_log(rng, 1, 512), d_in=_log(rng, 64, 2048), d_mid=_log(rng, 64, 2048), d_out=_log(rng, 64, 2048))
    if kind == "graph_mlp":
        return dict(kind=kind, dtype=rng.choice(["bf16", "fp16"]), rows=_log(rng, 1, 8192), hidden=_log(rng, 512, 4096, 128),
                    ffn=_log(rng, 1024, 14336, 128), block=rng.random() < 0.5)
    if kind == "decode":
        kv_heads = rng.choice([1, 2, 4])
        batch = _log(rng, 1, 64)
        most = min(8192, (64 * 2 * 4096) // (batch * kv_heads))          # the listed share's cache at most
        return dict(kind=kind, hidden=_log(rng, 1024, 5120, 256), q_heads=kv_heads * rng.choice([2, 4]) if kv_heads > 1 else 8,
                    kv_heads=kv_heads, ffn=_log(rng, 1024, 6400, 128), batch=batch, kv_len=_log(rng, 64, most))
    if kind == "moe":
        return dict(kind=kind, hidden=_log(rng, 512, 2048, 256), experts=rng.choice([8, 16, 32, 64]), top_k=rng.choice([2, 4, 6, 8]),
                    inter=_log(rng, 256, 768, 128), tokens=_log(rng, 128, 4096, 128))
    if kind == "train":
        return dict(kind=kind, layers=rng.randint(2, 4), hidden=_log(rng, 512, 4096, 256), tokens=_log(rng, 256, 8192, 128))
    if kind == "attention":
        batch, kv_heads = _log(rng, 1, 64), rng.choice([1, 2, 4, 8])
        keys = _log(rng, 16, min(32768, 16 * 8 * 8192 // (batch * kv_heads)))
        view = rng.random() < 0.4
        return dict(kind=kind, dtype=rng.choice(["bf16", "fp16"]), batch=batch, kv_heads=kv_heads, group=rng.choice([1, 4, 8]),
                    keys=keys, capacity=keys + _log(rng, 1, 4096) if view else keys)
    op = rng.choice(["rmsnorm", "layernorm", "softmax", "gelu", "silu_gate", "add"])
    return dict(kind="rows", op=op, dtype=rng.choice(["bf16", "fp16", "fp32"]), rows=_log(rng, 1, 16384),
                cols=_log(rng, 64, 8192, rng.choice([1, 8, 128])))


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _normal(g, *shape, dtype=torch.bfloat16, std=1.0):
    return (torch.randn(*shape, generator=g, device="cuda", dtype=torch.float32) * std).to(dtype)


def prepare(case, seed):
    kind = case["kind"]
    g = _generator(seed)
    st = {"kind": kind}
    if kind == "graph_fp32":
        x = _normal(g, case["rows"], case["d_in"], dtype=torch.float32)
        w1 = _normal(g, case["d_mid"], case["d_in"], dtype=torch.float32, std=case["d_in"] ** -0.5)
        w2 = _normal(g, case["d_out"], case["d_mid"], dtype=torch.float32, std=case["d_mid"] ** -0.5)
        graph = maco.TaskGraph()
        a = graph.linear(x, w1)
        b = graph.linear(a.output, w2)
        graph.compile()
        st.update(graph=graph, outputs=[a.output, b.output], keep=[x, w1, w2])
    elif kind == "graph_mlp":
        dt = DTYPES[case["dtype"]]
        hidden, ffn = case["hidden"], case["ffn"]
        x = _normal(g, case["rows"], hidden, dtype=dt)
        w_in = ops.interleave_gate_up(_normal(g, ffn, hidden, dtype=dt, std=0.02), _normal(g, ffn, hidden, dtype=dt, std=0.02))
        w_out = _normal(g, hidden, ffn, dtype=dt, std=0.02)
        graph = maco.TaskGraph()
        h, outputs = x, []
        if case["block"]:
            w_norm = (1.0 + 0.1 * torch.randn(hidden, generator=g, device="cuda")).to(dt)
            h = graph.rmsnorm(x, w_norm).output
        y = graph.linear(graph.linear(h, w_in, activation="swiglu").output, w_out)
        outputs.append(y.output)
        if case["block"]:
            outputs.append(graph.add(y.output, x).output)
        graph.compile()
        st.update(graph=graph, outputs=outputs, keep=[x, w_in, w_out])
    elif kind == "decode":
        from maco_b200.models.qwen3_layer import Qwen3DecodeLayer
        sizes = {k: case[k] for k in ("hidden", "q_heads", "kv_heads", "ffn", "batch", "kv_len")}
        st.update(layer=Qwen3DecodeLayer(**sizes, seed=int(seed) % 100003), x=_normal(g, case["batch"], case["hidden"]))
    elif kind == "moe":
        from maco_b200.models.moe_layer import MoEEPLayer
        sizes = {k: case[k] for k in ("hidden", "experts", "top_k", "inter", "tokens")}
        # twice the mean load is the layer's default capacity; small batches spread more than that
        layer = MoEEPLayer(**sizes, seed=int(seed) % 100003, capacity_factor=2.0 if case["tokens"] >= 2048 else 4.0, on_drop="raise")
        st.update(layer=layer, x=_normal(g, case["tokens"], case["hidden"]))
    elif kind == "train":
        from maco_b200.models.dp_mlp_stack import DPMLPStackBackward
        st.update(model=DPMLPStackBackward(case["layers"], case["hidden"], case["tokens"], seed=int(seed) % 100003))
    elif kind == "attention":
        dt = DTYPES[case["dtype"]]
        batch, heads, keys = case["batch"], case["kv_heads"], case["keys"]
        q = _normal(g, batch, heads * case["group"], 128, dtype=dt)
        k = _normal(g, batch, heads, case["capacity"], 128, dtype=dt)
        v = _normal(g, batch, heads, case["capacity"], 128, dtype=dt)
        st.update(q=q, k=k[:, :, :keys], v=v[:, :, :keys], out=torch.empty_like(q) if case["capacity"] == keys else None)
    else:
        dt = DTYPES[case["dtype"]]
        x = _normal(g, case["rows"], case["cols"], dtype=dt)
        w = (1.0 + 0.1 * torch.randn(case["cols"], generator=g, device="cuda")).to(dt)
        y = _normal(g, case["rows"], case["cols"], dtype=dt) if case["op"] in ("silu_gate", "add") else None
        b = _normal(g, case["cols"], dtype=dt, std=0.1) if case["op"] == "layernorm" else None
        st.update(op=case["op"], x=x, w=w, b=b, y=y)
    return st


def run(st):
    kind = st["kind"]
    if kind in ("graph_fp32", "graph_mlp"):
        st["graph"].execute()
        return st["outputs"]
    if kind == "decode":
        layer = st["layer"]
        return {"out": layer.forward(st["x"]), "k_cache": layer.k_cache, "v_cache": layer.v_cache}
    if kind == "moe":
        return st["layer"].forward(st["x"])
    if kind == "train":
        model = st["model"]
        return {"activations": model.forward(), "grads": model.backward()}
    if kind == "attention":
        return ops.attention_decode(st["q"], st["k"], st["v"], out=st["out"])
    op = st["op"]
    if op == "rmsnorm":
        return ops.rmsnorm(st["x"], st["w"], 1e-6)
    if op == "layernorm":
        return ops.layernorm(st["x"], st["w"], st["b"], 1e-5)
    if op == "softmax":
        return ops.softmax(st["x"])
    if op == "gelu":
        return ops.gelu(st["x"])
    if op == "silu_gate":
        return ops.silu_gate(st["x"], st["y"])
    return ops.add(st["x"], st["y"])


def work(case):
    c, kind = case, case["kind"]
    if kind == "graph_fp32":
        weights = c["d_in"] * c["d_mid"] + c["d_mid"] * c["d_out"]
        return {"bytes": 4 * (weights + c["rows"] * (c["d_in"] + c["d_mid"] + c["d_out"])), "flops": 2 * c["rows"] * weights}
    if kind == "graph_mlp":
        weights = 3 * c["hidden"] * c["ffn"]
        acts = c["rows"] * c["hidden"] * (3 if c["block"] else 2)
        return {"bytes": 2 * (weights + acts), "flops": 2 * c["rows"] * weights}
    if kind == "decode":
        weights = c["hidden"] * 128 * (2 * c["q_heads"] + 2 * c["kv_heads"]) + 3 * c["hidden"] * c["ffn"]
        cache = 2 * c["batch"] * c["kv_heads"] * 128 * (c["kv_len"] + 1)
        return {"bytes": 2 * (weights + cache + 2 * c["batch"] * c["hidden"]),
                "flops": 2 * c["batch"] * weights + 4 * c["batch"] * c["q_heads"] * 128 * (c["kv_len"] + 1)}
    if kind == "moe":
        expert = 3 * c["hidden"] * c["inter"]
        return {"bytes": 2 * (c["experts"] * (expert + c["hidden"]) + 2 * c["tokens"] * c["hidden"]),
                "flops": 2 * c["tokens"] * (c["top_k"] * expert + c["experts"] * c["hidden"])}
    if kind == "train":
        square, acts = c["hidden"] ** 2, c["tokens"] * c["hidden"]
        return {"bytes": 2 * (c["layers"] * square + 3 * acts) + 4 * c["layers"] * square,
                "flops": 2 * acts * c["hidden"] * (3 * c["layers"] - 1)}
    if kind == "attention":
        pairs = c["batch"] * c["kv_heads"]
        return {"bytes": 2 * 128 * pairs * (2 * c["keys"] + 2 * c["group"]), "flops": 4 * 128 * pairs * c["group"] * c["keys"]}
    n, size = c["rows"] * c["cols"], 4 if c["dtype"] == "fp32" else 2
    extra = {"rmsnorm": c["cols"], "layernorm": 2 * c["cols"], "silu_gate": n, "add": n}.get(c["op"], 0)
    return {"bytes": size * (2 * n + extra), "flops": 4 * n}


def tolerance(case):
    kind = case["kind"]
    if kind == "graph_fp32":
        return {"rel": 1e-5}                      # fp32 sums of up to 2048 terms
    if kind == "moe":
        # 16-bit activations; and a token whose router logits tie after rounding may take another expert
        return {"rel": 2e-2, "max": 0.99}
    if kind in ("decode", "train"):
        return {"rel": 1e-2}                      # bf16 activations between the operators (the gradients are sums of bf16 products)
    if kind == "rows" and case["dtype"] == "fp32":
        return {"rel": 1e-5}
    return {"rel": 1e-2 if case["dtype"] == "bf16" else 2e-3}
