"""Performance cases of the q4f16 path: what a program that uses this package asks of it.

A case is a dict of plain values; its ``kind`` says which entry point it goes through:

``call``        one eager ``ops.q4f16_matmul`` (a host that launches operator by operator)
``chain``       ``sets`` matmuls over distinct weights, captured once as a CUDA graph and replayed (what a compiled
                module does with the C ABI; also the benchmark's default workload)
``host``        ``b200_q4f16_matmul_host``: activation and result in pinned host memory
``dequantize``  ``ops.q4f16_dequantize``: the decode stage alone
``decode``      one decode step of ``DecodeEngine`` (one replay of its graph) with the KV cache filled up to ``pos``

Weights, scales and activations have the distributions of :mod:`relax_b200.synth`.
"""
from __future__ import annotations

import torch

from relax_b200 import _lib, decoder, ops, synth

SIZES_7B = dict(hidden=4096, heads=32, inter=11008, vocab=32000)


def listed():
    return [
        # one token through one projection of a 4096-wide model, operator by operator: launch latency counts
        dict(name="call_m1", kind="call", m=1, n=4096, k=4096, layout="reference"),
        # a narrow model whose width is a multiple of the group size but not of 256, a few rows
        dict(name="call_m3_k3200", kind="call", m=3, n=8640, k=3200, layout="reference"),
        # a served batch through the widest projection (gate|up) of the 7B shape
        dict(name="call_m64_gate_up", kind="call", m=64, n=22016, k=4096, layout="reference"),
        # a prompt of 2048 tokens: gate (or up) of the 7B shape
        dict(name="prefill_m2048", kind="call", m=2048, n=11008, k=4096, layout="reference"),
        # a short prompt of odd length on one eighth of a K=8192 model, weights repacked when they were bound
        dict(name="prefill_m777_shard", kind="call", m=777, n=3584, k=8192, layout="paired"),
        # batch-1 matmuls back to back over more weights than the L2 holds
        dict(name="chain_m1", kind="chain", m=1, n=4096, k=4096, sets=40),
        # the same matmul for a caller whose activations live in host memory
        dict(name="host_m1", kind="host", m=1, n=4096, k=4096),
        # decode as a kernel of its own (weights expanded once for a library matmul)
        dict(name="dequantize", kind="dequantize", n=11008, k=4096),
        # one token of one sequence, 7B shape, nearly full context
        dict(name="decode_b1", kind="decode", batch=1, pos=2011, layers=32, **SIZES_7B),
        # the same at the largest batch of the skinny kernels
        dict(name="decode_b16", kind="decode", batch=16, pos=2011, layers=32, **SIZES_7B),
        # a served batch of 64 at half the context
        dict(name="decode_b64", kind="decode", batch=64, pos=1001, layers=32, **SIZES_7B),
        # a small model, a few sequences, short odd context
        dict(name="decode_small_b5", kind="decode", batch=5, pos=333, layers=8, hidden=2048, heads=16, inter=5632, vocab=32000),
    ]


def _log(rng, lo, hi):
    """Spread over the logarithm of lo..hi, odd values among them."""
    return int(min(hi, max(lo, round(lo * (hi / lo) ** rng.random()))))


def _width(rng, lo, hi):
    """A reduction length: mostly whole 256-blocks as models have them, sometimes only whole scale groups."""
    step = 256 if rng.random() < 0.8 else 32
    return max(step, _log(rng, lo, hi) // step * step)


def draw(rng):
    kind = rng.choice(("call", "call", "call", "chain", "host", "dequantize", "decode", "decode", "decode"))
    if kind == "call":
        return dict(kind=kind, m=_log(rng, 1, 2048), n=_log(rng, 512, 28672), k=_width(rng, 1024, 11008),
                    layout=rng.choice(("reference", "reference", "paired")))
    if kind == "chain":
        return dict(kind=kind, m=_log(rng, 1, 128), n=_log(rng, 1024, 22016), k=_width(rng, 1024, 11008), sets=rng.randint(8, 40))
    if kind == "host":
        return dict(kind=kind, m=_log(rng, 1, 512), n=_log(rng, 1024, 22016), k=_width(rng, 1024, 11008))
    if kind == "dequantize":
        return dict(kind=kind, n=_log(rng, 512, 28672), k=_width(rng, 1024, 11008))
    batch = _log(rng, 1, 64)
    heads = rng.choice((8, 16, 20, 32, 40))
    hidden = heads * 128
    return dict(kind=kind, batch=batch, pos=_log(rng, 16, min(2040, 64 * 1001 // batch)), layers=rng.randint(2, 20), hidden=hidden,
                heads=heads, inter=int(hidden * rng.uniform(2.5, 3.5)) // 256 * 256, vocab=32000)


# ---------------------------------------------------------------------------------------------- states
def _generator(seed, stream):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 1000 + stream)
    return g


def _activations(m, k, seed):
    return torch.randn((m, k), dtype=torch.float16, device="cuda", generator=_generator(seed, 1))


def _check(rc):
    if rc:
        raise _lib.B200Error(rc, _lib.last_error())


def _prepare_chain(case, seed):
    m, n, k = case["m"], case["n"], case["k"]
    x = _activations(m, k, seed)
    weights = [synth.make_weights_torch(n, k, seed * 64 + i, "cuda") for i in range(case["sets"])]
    ys = [torch.empty((m, n), dtype=torch.float16, device="cuda") for _ in weights]
    matmul = _lib.lib().b200_q4f16_matmul

    def once(stream):
        for (wq, s), y in zip(weights, ys):
            _check(matmul(x.data_ptr(), wq.data_ptr(), s.data_ptr(), y.data_ptr(), m, n, k, stream.cuda_stream))

    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        once(stream)
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            once(stream)
    return dict(kind="chain", x=x, weights=weights, ys=ys, graph=graph)


def _prepare_decode(case, seed):
    cfg = decoder.DecoderConfig(hidden=case["hidden"], heads=case["heads"], inter=case["inter"], layers=case["layers"],
                                vocab=case["vocab"])
    layers = []
    for i in range(cfg.layers):
        layer = decoder.synth_layer_torch(cfg, seed * 64 + i, "cuda")
        for name in ("qkv", "o", "gu", "down"):
            # weights of a trained model's size (standard deviation near 0.006): the residual stream stays inside fp16
            layer[name] = (layer[name][0], layer[name][1] * 0.1)
        layer["inter_local"] = cfg.inter
        layers.append(layer)
    embed = torch.randn((cfg.vocab, cfg.hidden), dtype=torch.float16, device="cuda", generator=_generator(seed, 2)) * 0.02
    norm = torch.ones(cfg.hidden, dtype=torch.float16, device="cuda")
    pos, batch = case["pos"], case["batch"]
    engine = decoder.DecodeEngine(cfg, layers, embed, norm, embed, batch, (pos + 1 + 63) // 64 * 64, "cuda")
    g = _generator(seed, 3)
    for cache in engine.kc + engine.vc:
        cache.normal_(generator=g)
    tokens = torch.randint(0, cfg.vocab, (batch,), dtype=torch.int32, device="cuda", generator=g)
    engine.tokens.copy_(tokens)
    engine.set_position(pos)
    engine.capture(torch.cuda.Stream())
    return dict(kind="decode", engine=engine, tokens=tokens, pos=pos)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "chain":
        return _prepare_chain(case, seed)
    if kind == "decode":
        return _prepare_decode(case, seed)
    n, k = case["n"], case["k"]
    wq, scales = synth.make_weights_torch(n, k, seed, "cuda")
    state = dict(kind=kind, wq=wq, scales=scales)
    if kind == "dequantize":
        state["out"] = torch.empty((n, k), dtype=torch.float16, device="cuda")
        return state
    m = case["m"]
    x = _activations(m, k, seed)
    y = torch.empty((m, n), dtype=torch.float16, device="cuda")
    if kind == "host":
        state.update(m=m, n=n, k=k, x_dev=x, y_dev=y, x_host=x.cpu().pin_memory(),
                     y_host=torch.empty((m, n), dtype=torch.float16).pin_memory())
        return state
    if case["layout"] != "reference":
        state["wq"] = ops.q4f16_repack(wq, case["layout"])
    state.update(x=x, out=y, layout=None if case["layout"] == "reference" else case["layout"])
    return state


def run(state):
    kind = state["kind"]
    if kind == "call":
        return ops.q4f16_matmul(state["x"], state["wq"], state["scales"], out=state["out"], layout=state["layout"])
    if kind == "chain":
        state["graph"].replay()
        return state["ys"]
    if kind == "host":
        s = state
        _check(_lib.lib().b200_q4f16_matmul_host(
            s["x_host"].data_ptr(), s["x_dev"].data_ptr(), s["wq"].data_ptr(), s["scales"].data_ptr(), s["y_dev"].data_ptr(),
            s["y_host"].data_ptr(), s["m"], s["n"], s["k"], torch.cuda.current_stream().cuda_stream))
        return s["y_host"]
    if kind == "dequantize":
        return ops.q4f16_dequantize(state["wq"], state["scales"], out=state["out"])
    # decode: the host feeds the tokens and the position, the graph runs the step; it returns the logits and the
    # cache entries that the step appended in the last layer (which depend on every layer before it)
    engine, pos = state["engine"], state["pos"]
    engine.tokens.copy_(state["tokens"])
    engine.set_position(pos)
    engine.graph.replay()
    return {"logits": engine.logits, "k": engine.kc[-1][:, pos], "v": engine.vc[-1][:, pos]}


# ---------------------------------------------------------------------------------------------- what a pass must do
def _weight_bytes(n, k):
    return n * k // 2 + n * (k // 32) * 2


def work(case):
    kind = case["kind"]
    if kind == "decode":
        h, i, b, pos = case["hidden"], case["inter"], case["batch"], case["pos"]
        shapes = ((3 * h, h), (h, h), (2 * i, h), (h, i))
        per_layer = sum(_weight_bytes(n, k) for n, k in shapes) + 4 * h + b * (pos + 1) * h * 2 * 2
        flops = sum(2 * b * n * k for n, k in shapes) + 4 * b * (pos + 1) * h
        return {"bytes": case["layers"] * per_layer + case["vocab"] * h * 2 + b * case["vocab"] * 2,
                "flops": case["layers"] * flops + 2 * b * case["vocab"] * h}
    n, k = case["n"], case["k"]
    if kind == "dequantize":
        return {"bytes": _weight_bytes(n, k) + 2 * n * k, "flops": n * k}
    m, sets = case["m"], case.get("sets", 1)
    return {"bytes": sets * (_weight_bytes(n, k) + 2 * m * n) + 2 * m * k, "flops": sets * 2 * m * n * k}


def tolerance(case):
    """About four times what another form of the same arithmetic was seen to differ by: a matmul against its product
    in 64 bits over the dequantised weights by 2.8e-4 (one fp16 rounding of the result, at batch 1 also of the
    weights), one value by 8e-4; a decode step against the engine's other kernels (separate or fused, the weights
    rounded to fp16 or not) by up to 1.4e-3, one value by 6e-3."""
    if case["kind"] == "dequantize":
        return "exact"
    if case["kind"] == "decode":
        return {"rel": 5e-3, "max": 2.5e-2}
    return {"rel": 1.1e-3, "max": 3.2e-3}


# ---------------------------------------------------------------------------------------------- the same in 64 bits
def _expand(wq, scales):
    """The weights in 64 bits with the values that the decode stage gives them: (q - 7) * s rounded once to fp16."""
    n, words = wq.shape
    shifts = torch.arange(0, 32, 4, dtype=torch.int32, device="cuda")
    q = (wq.view(torch.int32).unsqueeze(-1) >> shifts) & 15
    w = (q - 7).view(n, words // 4, 32).double() * scales.double().unsqueeze(-1)
    return w.to(torch.float16).double().view(n, words * 8)


def _rmsnorm(x, weight, eps):
    return x * torch.rsqrt((x * x).mean(dim=-1, keepdim=True) + eps) * weight.double()


def _rotate(v, cos, sin):
    a, b = v[..., :64], v[..., 64:]
    return torch.cat((a * cos - b * sin, b * cos + a * sin), dim=-1)


def _exact_decode(case, seed):
    cfg = decoder.DecoderConfig(hidden=case["hidden"], heads=case["heads"], inter=case["inter"], layers=case["layers"],
                                vocab=case["vocab"])
    h, pos, batch = cfg.hidden, case["pos"], case["batch"]
    embed = torch.randn((cfg.vocab, h), dtype=torch.float16, device="cuda", generator=_generator(seed, 2)) * 0.02
    g = _generator(seed, 3)
    shape = (batch, (pos + 1 + 63) // 64 * 64, cfg.heads, 128)
    kc, vc = ([torch.empty(shape, dtype=torch.float16, device="cuda").normal_(generator=g) for _ in range(cfg.layers)] for _ in "kv")
    tokens = torch.randint(0, cfg.vocab, (batch,), dtype=torch.int32, device="cuda", generator=g)
    angle = pos * cfg.theta ** (-torch.arange(64, dtype=torch.float64, device="cuda") * 2.0 / 128)
    cos, sin = torch.cos(angle), torch.sin(angle)
    x = embed[tokens.long()].double()
    for i in range(cfg.layers):
        layer = decoder.synth_layer_torch(cfg, seed * 64 + i, "cuda")
        w = {name: _expand(layer[name][0], layer[name][1] * 0.1) for name in ("qkv", "o", "gu", "down")}
        qkv = (_rmsnorm(x, layer["norm1"], cfg.eps) @ w["qkv"].t()).view(batch, 3, cfg.heads, 128)
        q, k, v = _rotate(qkv[:, 0], cos, sin), _rotate(qkv[:, 1], cos, sin), qkv[:, 2]
        attn = torch.empty((batch, cfg.heads, 128), dtype=torch.float64, device="cuda")
        for b in range(batch):
            keys = torch.cat((kc[i][b, :pos].double(), k[b:b + 1]))
            values = torch.cat((vc[i][b, :pos].double(), v[b:b + 1]))
            p = torch.softmax(torch.einsum("hd,thd->ht", q[b], keys) / 128 ** 0.5, dim=-1)
            attn[b] = torch.einsum("ht,thd->hd", p, values)
        x = x + attn.view(batch, h) @ w["o"].t()
        gate, up = (_rmsnorm(x, layer["norm2"], cfg.eps) @ w["gu"].t()).chunk(2, dim=1)
        x = x + (torch.nn.functional.silu(gate) * up) @ w["down"].t()
    ones = torch.ones(h, dtype=torch.float16, device="cuda")
    return {"logits": _rmsnorm(x, ones, cfg.eps) @ embed.double().t(), "k": k, "v": v}


def exact(case, seed):
    kind = case["kind"]
    if kind == "decode":
        return _exact_decode(case, seed)
    n, k = case["n"], case["k"]
    if kind == "dequantize":
        return _expand(*synth.make_weights_torch(n, k, seed, "cuda")).to(torch.float16)
    x = _activations(case["m"], k, seed).double()
    if kind == "chain":
        return [x @ _expand(*synth.make_weights_torch(n, k, seed * 64 + i, "cuda")).t() for i in range(case["sets"])]
    y = x @ _expand(*synth.make_weights_torch(n, k, seed, "cuda")).t()
    return y.cpu() if kind == "host" else y
