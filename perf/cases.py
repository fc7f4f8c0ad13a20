"""The calls a user of this package makes, with the sizes they make them at, as measurable cases.

A case is a dict of plain values.  ``kind`` says which entry points one pass goes through:

* ``fused``  -- ``attention.hogwild_fused`` on fragment tensors (one attention layer's call);
* ``split``  -- ``attention.hogwild_rope`` followed by ``attention.hogwild_sdpa`` (callers that rotate themselves);
* ``step``   -- the attention side of a model step over ``layers`` layers: ``FragmentCache.update`` and
  ``attention.hogwild_fused_planned`` per layer, eagerly or replayed from a CUDA graph (``graph``);
* ``layer``  -- ``module.HogwildAttention.forward`` over ``layers`` layers: projections, cache update, attention;
* ``paged``  -- ``attention.copy_to_blocks`` of the new tokens and ``attention.hogwild_paged_sdpa``;
* ``varlen`` -- ``attention.hogwild_varlen_paged_sdpa`` on packed queries: prompt chunks and single tokens mixed.

Sizes: ``W`` workers (sequences for the paged kinds), ``Hq`` / ``Hkv`` heads of size ``E``, ``S`` query tokens per
worker.  Fragment kinds: a shared prompt of ``prompt`` keys (0: none) and one fragment per worker of ``own`` keys,
``ragged`` fewer for each further worker, the ``S`` newest tokens included.  Paged kinds: ``own`` keys per sequence,
``ragged`` fewer for each further one, in blocks of ``block`` rows.
"""
from __future__ import annotations

import math

import torch

from inference_lib_b200 import attention as ops
from inference_lib_b200.cache import FragmentCache
from inference_lib_b200.module import HogwildAttention
from inference_lib_b200.workloads import hogwild_locations, rope_tables

DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
THETA = 5e5
DEVICE = "cuda"


def listed():
    return [
        # the smallest call there is: two workers of a small fp32 model a few hundred tokens in (launches and host path)
        dict(name="tiny_f32", kind="fused", dtype="f32", W=2, Hq=8, Hkv=2, E=64, S=1, prompt=256, own=64, ragged=0),
        # one attention call of an eager decode loop, an ordinary context
        dict(name="decode_8k", kind="fused", dtype="bf16", W=2, Hq=32, Hkv=8, E=128, S=1, prompt=4096, own=2048, ragged=0),
        # a serving loop's decode step: four workers, 16 K keys, cache update and attention of four layers in a CUDA graph
        dict(name="step_16k_graph", kind="step", dtype="bf16", W=4, Hq=32, Hkv=8, E=128, S=1, prompt=8192, own=2048,
             ragged=0, layers=4, graph=True),
        # decode through the attention layers themselves (what a model runs after model_surgery), five heads per kv head,
        # workers that have written different amounts
        dict(name="layer_decode", kind="layer", dtype="bf16", W=3, Hq=40, Hkv=8, E=128, S=1, prompt=5003, own=1501,
             ragged=211, layers=2, hidden=5120),
        # decode at the longest context
        dict(name="decode_131k", kind="fused", dtype="bf16", W=2, Hq=32, Hkv=8, E=128, S=1, prompt=131072, own=4096, ragged=0),
        # eight workers that advance by chunks of 16 tokens over a common prompt
        dict(name="chunk_16", kind="fused", dtype="bf16", W=8, Hq=64, Hkv=8, E=128, S=16, prompt=16384, own=1024, ragged=0),
        # prefill of a prompt, one sequence, causal
        dict(name="prompt_prefill", kind="fused", dtype="bf16", W=1, Hq=32, Hkv=8, E=128, S=4000, prompt=0, own=4000, ragged=0),
        # every worker reads a block of its own instructions behind the shared prompt; five heads per kv head, ragged
        # fragments, fp16
        dict(name="worker_prefill_f16", kind="fused", dtype="f16", W=3, Hq=40, Hkv=8, E=128, S=256, prompt=4099, own=901, ragged=100),
        # decode of a small model: heads of 64, seven per kv head, fp16, rotation and attention as separate calls
        dict(name="split_d64_f16", kind="split", dtype="f16", W=4, Hq=14, Hkv=2, E=64, S=1, prompt=6001, own=517, ragged=40),
        # paged decode of a batch of long sequences
        dict(name="paged_decode", kind="paged", dtype="bf16", W=8, Hq=32, Hkv=2, E=128, S=1, own=16384, ragged=0, block=16),
        # a continuous batch: two prompt chunks and six single tokens, all at their own lengths
        dict(name="paged_mixed", kind="varlen", dtype="bf16", W=8, Hq=32, Hkv=8, E=128, S=512, chunks=2, own=6000, ragged=411, block=16),
        # decode in fp32 (a checking run in full precision)
        dict(name="decode_f32", kind="fused", dtype="f32", W=2, Hq=32, Hkv=8, E=128, S=1, prompt=6000, own=701, ragged=1),
    ]


def draw(rng):
    """One more case: a kind, then its sizes, spread over the range between the smallest and the largest listed use."""
    def log(lo, hi):
        return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))

    while True:
        kind = rng.choice(["fused", "fused", "fused", "fused", "split", "step", "layer", "paged", "varlen"])
        hkv = rng.choice([1, 2, 4, 8])
        c = dict(kind=kind, dtype=rng.choice(["bf16", "bf16", "f16"]), W=rng.randint(1, 8), Hq=hkv * rng.choice([1, 4, 4, 5, 7, 8]),
                 Hkv=hkv, E=rng.choice([128, 128, 64]), S=1)
        if kind in ("fused", "split") and rng.random() < 0.2:
            c.update(dtype="f32", W=rng.randint(1, 3))
        if kind in ("paged", "varlen"):
            c.update(own=log(500, 16384), ragged=rng.randint(0, 50), block=rng.choice([16, 16, 32, 64]))
            c.update(S=rng.choice([1, 1, 4])) if kind == "paged" else c.update(S=log(16, 512), chunks=rng.randint(1, min(2, c["W"])))
        else:
            if c["dtype"] != "f32" and c["E"] == 128 and kind in ("fused", "split") and rng.random() < 0.6:
                c["S"] = _chunk(log(2, 4096), c["Hq"] // hkv)                          # chunks and prefill; decode otherwise
            c.update(prompt=0 if rng.random() < 0.15 else log(200, 131072 if c["S"] == 1 and c["dtype"] != "f32" else 16384),
                     own=c["S"] + log(64, 4096), ragged=rng.randint(0, 60))
            if kind in ("step", "layer"):
                c.update(layers=rng.randint(1, 3))
                c.update(graph=rng.random() < 0.5) if kind == "step" else c.update(hidden=c["Hq"] * c["E"])
        rows = c["W"] * c["S"] * c["Hq"] // hkv
        if kind in ("fused", "split") and c["S"] > 1 and 16 < rows < 128:
            continue                                                                   # (a block is not filled)
        # no dearer than the largest listed uses, and large enough for every worker to hold its new tokens
        w = work(c)
        shortest = c["own"] - c["ragged"] * (c["W"] - 1)
        if (shortest >= c["S"] and w["bytes"] <= 4e8 and w["flops"] <= (5e8 if c["dtype"] == "f32" else 9e10 if kind != "varlen" else 1.5e10)):
            return c


def _chunk(s, heads):
    """The chunk sizes schedulers cut prompts to: whole 128-row blocks of query rows per kv head, or powers of two below."""
    step = 128 // math.gcd(heads, 128)
    return s - s % step if s >= step else (1 << (s.bit_length() - 1) if 128 % heads == 0 else 1)


# ---- shapes ---------------------------------------------------------------------------------------------------------
def _owned(c):
    return [c["own"] - c["ragged"] * w for w in range(c["W"])]


def _fragments(c):
    """Fragment lengths and every worker's order of them: prompt, the other workers, its own."""
    p = 1 if c["prompt"] else 0
    lengths = ([c["prompt"]] if p else []) + _owned(c)
    orders = [list(range(p)) + [p + o for o in range(c["W"]) if o != w] + [p + w] for w in range(c["W"])]
    return lengths, orders


def _query_tokens(c):
    """Query tokens per sequence of a packed batch."""
    return [c["S"] if w < c["chunks"] else 1 for w in range(c["W"])]


def _causal(keys, s):
    """Keys seen by the `s` newest tokens of a run of `keys`, added up."""
    return s * keys - s * (s - 1) // 2


def work(case):
    c, size = case, 4 if case["dtype"] == "f32" else 2
    kv_row, q_row = 2 * c["Hkv"] * c["E"] * size, c["Hq"] * c["E"] * size
    if c["kind"] in ("paged", "varlen"):
        tokens = _query_tokens(c) if c["kind"] == "varlen" else [c["S"]] * c["W"]
        seen = sum(_causal(n, s) for n, s in zip(_owned(c), tokens))
        new = c["W"] * c["S"] if c["kind"] == "paged" else 0
        return {"bytes": sum(_owned(c)) * kv_row + 2 * sum(tokens) * q_row + new * kv_row, "flops": 4 * c["Hq"] * c["E"] * seen}
    lengths, _ = _fragments(c)
    seen = c["W"] * _causal(sum(lengths), c["S"])
    tokens = c["W"] * c["S"]
    one = sum(lengths) * kv_row + (2 + len(lengths)) * tokens * q_row              # keys, values, queries, output, rotated queries
    flops = 4 * c["Hq"] * c["E"] * seen
    if c["kind"] in ("step", "layer"):
        one += tokens * kv_row                                                     # the appended rows
    if c["kind"] == "layer":
        weights = c["hidden"] * (2 * c["Hq"] + 2 * c["Hkv"]) * c["E"]
        one += weights * size + 2 * tokens * c["hidden"] * size - 2 * tokens * q_row
        flops += 2 * tokens * weights
    layers = c.get("layers", 1)
    return {"bytes": layers * one, "flops": layers * flops}


def tolerance(case):
    """Four times what a pass differs by from the same call in 64 bits (2-norm; largest over root mean square): 3e-7 to 6e-7
    and 3e-6 in fp32, 3e-4 and 1.4e-3 in fp16, 2.4e-3 and 5e-2 (short rows of a causal prompt) in bf16."""
    return {"f32": {"rel": 2.5e-6, "max": 2e-5}, "f16": {"rel": 1.2e-3, "max": 1e-2}, "bf16": {"rel": 1e-2, "max": 0.2}}[case["dtype"]]


# ---- inputs -----------------------------------------------------------------------------------------------------------
def _randn(gen, *shape, dtype, scale=1.0):
    return (torch.randn(*shape, device=DEVICE, generator=gen) * scale).to(dtype)


def prepare(case, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    make = {"fused": _prepare_fragments, "split": _prepare_fragments, "step": _prepare_step, "layer": _prepare_step,
            "paged": _prepare_paged, "varlen": _prepare_paged}[case["kind"]]
    return dict(make(dict(case), gen), kind=case["kind"])


def _prepare_fragments(c, gen):
    # normally distributed queries, keys and values; a rotation leaves that distribution as it is, so keys need none
    dt, W, Hq, Hkv, E, S = DTYPES[c["dtype"]], c["W"], c["Hq"], c["Hkv"], c["E"], c["S"]
    lengths, orders = _fragments(c)
    loc = hogwild_locations(lengths, orders, S)
    cos, sin = (t.to(DEVICE) for t in rope_tables(loc, E, THETA))
    return dict(q=_randn(gen, W, Hq, S, E, dtype=dt), scale=E ** -0.5, loc=loc.to(DEVICE), cos=cos, sin=sin,
                keys=[_randn(gen, 1, Hkv, n, E, dtype=dt) for n in lengths], values=[_randn(gen, 1, Hkv, n, E, dtype=dt) for n in lengths],
                frags=torch.tensor(lengths, dtype=torch.int32, device=DEVICE),
                rq=torch.empty(len(lengths), W, Hq, S, E, dtype=dt, device=DEVICE), out=torch.empty(W, Hq, S, E, dtype=dt, device=DEVICE))


def _prepare_step(c, gen):
    dt, W, Hq, Hkv, E, S, L = DTYPES[c["dtype"]], c["W"], c["Hq"], c["Hkv"], c["E"], c["S"], c["layers"]
    lengths, orders = _fragments(c)
    p = len(lengths) - W
    inv_freq = 1.0 / (THETA ** (torch.arange(0, E, 2, dtype=torch.float32) / E))
    cache = FragmentCache(layers=L, capacities=lengths[:p] + [n + 64 for n in lengths[p:]], Hkv=Hkv, E=E, dtype=dt, device=DEVICE,
                          order=orders, inv_freq=inv_freq)
    start = [n - (S if f >= p else 0) for f, n in enumerate(lengths)]            # before this step's tokens
    for f, n in enumerate(start):
        cache.load_fragment(f, [_randn(gen, Hkv, n, E, dtype=dt) for _ in range(L)], [_randn(gen, Hkv, n, E, dtype=dt) for _ in range(L)])
    positions = torch.tensor([[start[p + w] + s for s in range(S)] for w in range(W)])
    cos, sin = (t.to(device=DEVICE, dtype=dt) for t in rope_tables(positions, E, THETA))
    s = dict(cache=cache, start=start, start_dev=[torch.tensor(start, dtype=torch.int32, device=DEVICE)] * L, scale=E ** -0.5,
             cos=cos, sin=sin, layers=L, first_own=p, position_ids=positions.to(DEVICE))
    if c["kind"] == "layer":
        s["modules"] = []
        for layer in range(L):
            m = HogwildAttention(c["hidden"], Hq, Hkv, E, layer, dtype=dt, device=DEVICE)
            for lin in (m.q_proj, m.k_proj, m.v_proj, m.o_proj):
                lin.weight.data.normal_(0.0, lin.in_features ** -0.5, generator=gen)
                if lin.bias is not None:
                    lin.bias.data.normal_(0.0, 0.1, generator=gen)
            s["modules"].append(m.requires_grad_(False))
        s["hidden"] = _randn(gen, W, S, c["hidden"], dtype=dt)
        return s
    # q / k / v as the transposed views of projection outputs that a layer hands over
    s["qkv"] = [tuple(_randn(gen, W, S, h, E, dtype=dt).transpose(1, 2) for h in (Hq, Hkv, Hkv)) for _ in range(L)]
    s["rq"] = [torch.empty(len(lengths), W, Hq, S, E, dtype=dt, device=DEVICE) for _ in range(L)]
    s["out"] = [torch.empty(W, Hq, S, E, dtype=dt, device=DEVICE) for _ in range(L)]
    if c["graph"]:
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _step(s)
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            s["result"] = _step(s)
        s["graph"] = graph
    return s


def _prepare_paged(c, gen):
    dt, W, Hq, Hkv, E, bs = DTYPES[c["dtype"]], c["W"], c["Hq"], c["Hkv"], c["E"], c["block"]
    lens = _owned(c)
    per_seq = (max(lens) + bs - 1) // bs
    blocks = W * per_seq
    s = dict(scale=E ** -0.5, kc=_randn(gen, blocks, Hkv, bs, E, dtype=dt), vc=_randn(gen, blocks, Hkv, bs, E, dtype=dt),
             table=torch.randperm(blocks, device=DEVICE, generator=gen).to(torch.int32).reshape(W, per_seq))
    if c["kind"] == "paged":
        S = c["S"]
        s.update(k=_randn(gen, W, Hkv, S, E, dtype=dt), v=_randn(gen, W, Hkv, S, E, dtype=dt), q=_randn(gen, 1, W, Hq, S, E, dtype=dt),
                 before=torch.tensor([n - S for n in lens], dtype=torch.int32, device=DEVICE),
                 loc=torch.tensor([[[n - S + t for t in range(S)] for n in lens]], dtype=torch.int32, device=DEVICE),
                 frags=torch.tensor([max(lens)], dtype=torch.int32, device=DEVICE), out=torch.empty(W, Hq, S, E, dtype=dt, device=DEVICE))
    else:
        tokens = _query_tokens(c)
        loc = [n - s_w + t for n, s_w in zip(lens, tokens) for t in range(s_w)]
        cu = [sum(tokens[:w]) for w in range(W + 1)]
        s.update(q=_randn(gen, 1, sum(tokens), Hq, E, dtype=dt), loc=torch.tensor([loc], dtype=torch.int32, device=DEVICE),
                 frags=torch.tensor([lens], dtype=torch.int32, device=DEVICE), cu=torch.tensor(cu, dtype=torch.int32, device=DEVICE),
                 out=torch.empty(sum(tokens), Hq, E, dtype=dt, device=DEVICE))
    return s


# ---- one pass ---------------------------------------------------------------------------------------------------------
def _roll_back(s):
    """Back to the lengths before the step, as a program does that drops the tokens of a rejected draft."""
    cache = s["cache"]
    torch._foreach_copy_([cache.frags(layer) for layer in range(s["layers"])], s["start_dev"])
    for layer in range(s["layers"]):
        cache.host_lengths[layer][:] = s["start"]


def _written(s):
    """The fragments that the step appended to."""
    cache = s["cache"]
    return [(cache.keys[layer][f], cache.values[layer][f]) for layer in range(s["layers"]) for f in range(s["first_own"], cache.F)]


def _step(s):
    _roll_back(s)
    for layer, (q, k, v) in enumerate(s["qkv"]):
        cs = s["cache"].update(k, v, layer, s["cos"], s["sin"])
        ops.hogwild_fused_planned(q, cs.loc, cs.keys, cs.values, s["scale"], cs.frags, cs.cos, cs.sin, rotated_queries=s["rq"][layer],
                                  out=s["out"][layer], host_lengths=cs.host_lengths, stable_fragments=cs.stable)
    return {"out": s["out"], "rq": s["rq"], "lengths": s["cache"].frags(0), "written": _written(s)}


@torch.no_grad()
def run(state):
    s = state
    if s["kind"] == "fused":
        out = ops.hogwild_fused(s["q"], s["loc"], s["keys"], s["values"], s["scale"], s["frags"], s["cos"], s["sin"],
                                rotated_queries=s["rq"], out=s["out"])
        return {"out": out, "rq": s["rq"]}
    if s["kind"] == "split":
        rq = ops.hogwild_rope(s["q"], s["cos"], s["sin"], out=s["rq"])
        return {"out": ops.hogwild_sdpa(rq, s["loc"], s["keys"], s["values"], s["scale"], s["frags"], out=s["out"]), "rq": rq}
    if s["kind"] == "step":
        if "graph" in s:
            s["graph"].replay()
            return s["result"]
        return _step(s)
    if s["kind"] == "layer":
        _roll_back(s)
        x = s["hidden"]
        for m in s["modules"]:
            x = x + m(x, (s["cos"], s["sin"]), past_key_values=s["cache"], position_ids=s["position_ids"])[0]
        return {"hidden": x, "lengths": s["cache"].frags(0), "written": _written(s)}
    if s["kind"] == "paged":
        ops.copy_to_blocks(s["k"], s["v"], s["kc"], s["vc"], s["table"], s["before"])
        out = ops.hogwild_paged_sdpa(s["q"], s["loc"], s["kc"], s["vc"], s["table"], s["scale"], s["frags"], out=s["out"])
        return {"out": out, "key_cache": s["kc"], "value_cache": s["vc"]}
    return ops.hogwild_varlen_paged_sdpa(s["q"], s["loc"], s["kc"], s["vc"], s["table"], s["scale"], s["frags"], s["cu"], out=s["out"])
