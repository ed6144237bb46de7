"""The work this package is measured on: decode steps, prefills and page selections as a long-context
serving program has them done, through the package's public classes.

A case is a dict of plain values; `path` says what kind of work it is:

  decode    one new token for `layers` attention layers (or, with `streams` > 0, for that many independent
            sequences dealt to `streams` CUDA streams), each with a KV prefix of its own in pinned host memory.
            `graph`: the token step is captured once and replayed, as a chat program does; otherwise every
            layer is called eagerly.  A prefix of at most `lru` tokens is fully resident.
  tokens    one generate call with several tokens (the tail of a prompt that arrives after its prefill)
  prefill   the prompt of one layer: dense causal attention, then the cache is built from its keys and values
  select    page scoring and top-k page selection alone

Values have the structure that matters to the path: N(0,1) keys and values with a few outlier channels, `needle`
pages whose keys lie along a shared direction, queries near that direction that drift a little per step.  A decode
state cycles through thousands of steps' inputs, one per pass, so that a steady step keeps missing a few pages per head.
"""

from __future__ import annotations

import math

import torch

from dram_attention_b200 import DRAMAttention
from dram_attention_b200.lru_cache import LRUCache
from dram_attention_b200.topk_selector import IPUpperboundTopKSelector

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
ELEMENT_BYTES = {"bf16": 2, "fp16": 2, "fp32": 4}
STEPS = 4096            # one-token inputs a state holds
OUTPUT = 256            # tokens its local window has room for (positions start over after that many)
DRIFT = 0.05            # change of a query channel per step


def _decode(name, dram, layers=1, hk=8, rep=4, d=128, page=16, lru=32768, local=4096, top_k=4096, dtype="bf16",
            graph=True, streams=0, redraw=0, tail=0):
    return {"name": name, "path": "decode", "dram": dram, "tail": tail, "layers": layers, "hk": hk, "rep": rep,
            "d": d, "page": page, "lru": lru, "local": local, "top_k": top_k, "dtype": dtype, "graph": graph,
            "streams": streams, "redraw": redraw}


def listed():
    return [
        # the smallest calls: a float32 toy layer driven step by step from Python (tests, notebooks)
        _decode("decode-4k-fp32-eager", 4096, hk=2, d=64, lru=2048, local=256, top_k=512, dtype="fp32", graph=False),
        # an ordinary layer called eagerly: evaluation harnesses that do not capture the step
        _decode("decode-64k-eager", 65536, graph=False),
        # the headline: Llama-3-8B-shaped layers at 128K, the token step of a stack in one graph
        _decode("decode-128k-4-layers", 131072, layers=4),
        # odd sizes, another GQA group, larger pages, float16: one tensor-parallel share of a bigger model
        _decode("decode-77k-odd-fp16", 77792, layers=3, hk=3, rep=8, page=32, lru=20000, local=1000, top_k=1056,
                dtype="fp16", tail=19),
        # a million tokens, all KV heads on one GPU
        _decode("decode-1m", 1048576, lru=65536, local=8192, top_k=8192),
        # a million tokens, one KV head of eight: a GPU's share when the heads are sharded
        _decode("decode-1m-one-head-8-layers", 1048576, layers=8, hk=1, lru=65536, local=8192, top_k=8192),
        # batched serving: eight sequences whose topic changes every 32 tokens
        _decode("decode-64k-8-sequences", 65536, layers=8, streams=4, redraw=32),
        # a short conversation: the prefix fits the cache
        _decode("decode-resident-13k", 13008, layers=4, tail=5),
        # five prompt tokens that come after the prefill
        {"name": "tokens-5-64k", "path": "tokens", "tokens": 5, "dram": 65536, "tail": 7, "hk": 8, "rep": 4, "d": 128,
         "page": 16, "lru": 32768, "local": 4096, "top_k": 1024, "dtype": "bf16"},
        # prompts: a short one of odd length, and a long one
        {"name": "prefill-2999", "path": "prefill", "prompt": 2999, "hk": 8, "rep": 4, "d": 128, "page": 16, "lru": 1024,
         "local": 512, "top_k": 256, "dtype": "bf16"},
        {"name": "prefill-32k", "path": "prefill", "prompt": 32768, "hk": 8, "rep": 4, "d": 128, "page": 16,
         "lru": 8192, "local": 4096, "top_k": 1024, "dtype": "bf16"},
        # scoring and selection over a million tokens' pages
        {"name": "select-64k-pages", "path": "select", "pages": 65536, "hk": 8, "rep": 4, "d": 128, "page": 16, "k": 256,
         "dtype": "bf16"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choices(["decode", "tokens", "prefill", "select"], [6, 1, 3, 2])[0]
    dtype = rng.choices(["bf16", "fp16", "fp32"], [7, 2, 1])[0]
    d = 128 if rng.random() < 0.85 else 64
    page = 16 if rng.random() < 0.8 else 32
    hk = rng.choice([1, 2, 3, 4, 5, 8, 8])
    rep = rng.choice([1, 2, 4, 4, 8])
    if path == "select":
        return {"path": "select", "pages": _log(rng, 512, 65536), "hk": hk, "rep": rep, "d": d, "page": page,
                "k": min(512, _log(rng, 16, 512)), "dtype": dtype}
    if path == "prefill":
        local = _log(rng, 256, 1024)
        # dense attention in 16-bit types; at most as much work as the longest listed prompt
        dtype = "fp16" if dtype == "fp32" else dtype
        prompt = _log(rng, 2048, 32768)
        if prompt > 12000:
            hk = min(hk, 4)
        lru = max(page * 16, min(_log(rng, 512, 16384), (prompt - local) // 2) // page * page)
        return {"path": "prefill", "prompt": prompt, "hk": hk, "rep": min(rep, 4), "d": 128, "page": page, "lru": lru,
                "local": local, "top_k": lru // 8 // page * page, "dtype": dtype}
    slots = _log(rng, 128, 4096)                      # slots per head
    dram_pages = _log(rng, slots // 2, 65536 if hk <= 2 else 16384)
    c = {"dram": dram_pages * page, "tail": rng.randrange(page), "hk": hk, "rep": rep, "d": d, "page": page,
         "lru": slots * page, "local": _log(rng, 200, 8192), "dtype": dtype}
    if path == "tokens":
        tokens = rng.randint(2, 8)
        c["dram"] = max(c["dram"], (slots + 16) * page)
        return {"path": "tokens", "tokens": tokens, **c, "top_k": max(1, min(256, slots // (tokens * rep))) * page}
    graph = rng.random() < 0.75
    layers = rng.randint(1, 4) if graph else 1
    return {"path": "decode", **c, "layers": layers, "graph": graph, "streams": rng.choice([0, 0, 0, 2]) if layers > 1 else 0,
            "redraw": 32 if rng.random() < 0.2 else 0, "top_k": max(1, min(512, slots // (2 * rep))) * page}


# ---- inputs --------------------------------------------------------------------------------------------

def _generator(seed, *more):
    for m in more:
        seed = (seed * 1000003 + m + 1) % (1 << 62)
    return torch.Generator(device="cuda").manual_seed(seed)


def _prefix(g, case, length):
    """Keys and values (1, length, hk, d) of a prompt, the needle direction and the outlier channels."""
    hk, d, dtype = case["hk"], case["d"], DTYPES[case["dtype"]]
    outliers = torch.randperm(d, generator=g, device="cuda")[:max(1, d // 16)]
    u = torch.randn(d, generator=g, device="cuda")
    u = u / u.norm() * d ** 0.5
    kv = []
    for _ in range(2):
        t = torch.empty(1, length, hk, d, dtype=dtype, device="cuda")
        for a in range(0, length, 131072):
            x = torch.randn(min(131072, length - a), hk, d, generator=g, device="cuda")
            x[..., outliers] *= 10.0
            t[0, a:a + 131072] = x
        kv.append(t)
    page = case["page"]
    n_needles = min(32, max(1, length // (page * 64)))
    at = torch.randperm(length // page, generator=g, device="cuda")[:n_needles]
    rows = (at[:, None] * page + torch.arange(page, device="cuda")[None]).reshape(-1)
    noise = torch.randn(rows.numel(), hk, d, generator=g, device="cuda")
    kv[0][0, rows] = (u + 0.3 * noise).to(dtype)
    return kv[0], kv[1], u, outliers


def _steps(g, case, u, outliers, steps, tokens=1, redraw=0):
    """(steps, 1, tokens, hq + 2 hk, d): per step the queries, the new keys and the new values side by side, as a
    fused projection leaves them.  A query is u plus N(0,1) noise that forgets itself slowly, DRIFT per token; every
    `redraw` steps it becomes N(0,1) altogether."""
    hk, d, dtype = case["hk"], case["d"], DTYPES[case["dtype"]]
    hq = hk * case["rep"]
    n = steps * tokens
    keep = 1.0 - DRIFT ** 2 / 2
    walk = (1.0 - keep ** 2) ** 0.5 * torch.randn(n, hq, d, generator=g, device="cuda")
    noise = torch.randn(hq, d, generator=g, device="cuda")
    for a in range(0, n, 512):        # noise[t] = keep * noise[t-1] + walk[t], a block at a time
        block = walk[a:a + 512]
        power = (keep ** torch.arange(1, block.shape[0] + 1, device="cuda", dtype=torch.float32)).view(-1, 1, 1)
        block.copy_(power * (noise + torch.cumsum(block / power, 0)))
        noise = block[-1]
    for i in range(redraw, steps, redraw) if redraw else ():
        walk[i * tokens:] += torch.randn(hq, d, generator=g, device="cuda") - u - walk[i * tokens]
    kv = torch.randn(n, 2 * hk, d, generator=g, device="cuda")
    kv[..., outliers] *= 10.0
    return torch.cat([(walk + u).to(dtype), kv.to(dtype)], 1).view(steps, 1, tokens, hq + 2 * hk, d)


def _operator(case, max_output):
    return DRAMAttention(max_output_length=max_output, lru_hbm_cache_size=case["lru"], local_cache_size=case["local"],
                         page_size=case["page"], top_k=case["top_k"], n_kv_heads=case["hk"], head_dim=case["d"],
                         device="cuda", dtype=DTYPES[case["dtype"]])


def _split(qkv, hk):
    hq = qkv.shape[2] - 2 * hk
    return qkv[:, :, :hq], qkv[:, :, hq:hq + hk], qkv[:, :, hq + hk:]


def _cache_state(op):
    """What a generate call leaves behind besides its output."""
    state = {"cache_k": op.cache_k, "cache_v": op.cache_v, "slots": op.lru_cache.hbm_kv_cache}
    if isinstance(op.lru_cache, LRUCache):
        state["slot_pages"] = op.lru_cache.hbm_page_to_dram_page_mapping
        state["slot_times"] = op.lru_cache.page_access_time
    return state


def _attached(case, seed, max_output, steps, tokens=1):
    """Operators with their prefixes attached, and the inputs of every step (steps, layers, 1, tokens, heads, d)."""
    length = case["dram"] + case["local"] - case["page"] + case["tail"]
    ops, inputs = [], []
    for layer in range(case.get("layers", 1)):
        g = _generator(seed, layer)
        k, v, u, outliers = _prefix(g, case, length)
        op = _operator(case, max_output)
        op.init_cache(k, v)
        ops.append(op)
        inputs.append(_steps(g, case, u, outliers, steps, tokens, case.get("redraw", 0)))
    return ops, torch.stack(inputs, 1), length


def _prepare_decode(case, seed):
    ops, inputs, length = _attached(case, seed, OUTPUT, STEPS)
    state = {"ops": ops, "inputs": inputs, "length": length, "step": 0}
    if not case["graph"]:
        return state
    hk = case["hk"]
    state["qkv"] = qkv = inputs[0].clone()
    state["positions"] = positions = torch.arange(length, length + OUTPUT, dtype=torch.int32, device="cuda").view(-1, 1)
    state["pos"] = pos = positions[0].clone()
    streams = [torch.cuda.Stream() for _ in range(case["streams"])]

    def token_step():
        outs = [None] * len(ops)
        main = torch.cuda.current_stream()
        for s in streams:
            s.wait_stream(main)
        for i, op in enumerate(ops):
            q, k, v = _split(qkv[i], hk)
            with torch.cuda.stream(streams[i % len(streams)] if streams else main):
                outs[i] = op(q, k, v, start_pos=pos, stage="generate")
        for s in streams:
            main.wait_stream(s)
        return outs

    token_step()                  # once eagerly: everything a step needs exists
    torch.cuda.synchronize()
    state["graph"] = graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        state["outs"] = token_step()
    return state


def _run_decode(case, state):
    i = state["step"] % STEPS
    state["step"] += 1
    if case["graph"]:
        state["qkv"].copy_(state["inputs"][i])
        state["pos"].copy_(state["positions"][i % OUTPUT])
        state["graph"].replay()
        outs = state["outs"]
    else:
        outs = []
        for layer, op in enumerate(state["ops"]):
            q, k, v = _split(state["inputs"][i][layer], case["hk"])
            outs.append(op(q, k, v, start_pos=state["length"] + i % OUTPUT, stage="generate"))
    return {"out": outs, "state": [_cache_state(op) for op in state["ops"]]}


def _prepare_tokens(case, seed):
    tokens = case["tokens"]
    ops, inputs, length = _attached(case, seed, OUTPUT, STEPS // tokens, tokens)
    calls = [tuple(t.contiguous() for t in _split(x[0], case["hk"])) for x in inputs]
    return {"ops": ops, "calls": calls, "length": length, "step": 0}


def _run_tokens(case, state):
    i = state["step"]
    state["step"] += 1
    q, k, v = state["calls"][i % len(state["calls"])]
    pos = state["length"] + i % (OUTPUT // case["tokens"]) * case["tokens"]
    out = state["ops"][0](q, k, v, start_pos=pos, stage="generate")
    return {"out": out, "state": _cache_state(state["ops"][0])}


def _prepare_prefill(case, seed):
    g = _generator(seed)
    k, v, u, _ = _prefix(g, case, case["prompt"])
    q = torch.randn(1, case["prompt"], case["hk"] * case["rep"], case["d"], generator=g, device="cuda")
    return {"op": _operator(case, 128), "q": (q + 0.5 * u).to(k.dtype), "k": k, "v": v}


def _run_prefill(case, state):
    op = state["op"]
    out = op(state["q"], state["k"], state["v"], start_pos=0, stage="prefill")
    result = {"out": out, **_cache_state(op)}
    if isinstance(op.lru_cache, LRUCache):
        result["pages"] = op.lru_cache.dram_kv_cache
        result["summaries"] = op.lru_cache.top_k_selector.chunk_min_max
    return result


def _prepare_select(case, seed):
    g = _generator(seed)
    hk, d, tokens = case["hk"], case["d"], case["pages"] * case["page"]
    keys = torch.empty(hk, tokens, d, dtype=DTYPES[case["dtype"]], device="cuda")
    for h in range(hk):
        keys[h] = torch.randn(tokens, d, generator=g, device="cuda")
    selector = IPUpperboundTopKSelector(keys, case["pages"], device="cuda")
    q = torch.randn(1, 1, hk * case["rep"], d, generator=g, device="cuda").to(keys.dtype)
    return {"selector": selector, "q": q, "k": min(case["k"], case["pages"])}


def _run_select(case, state):
    return state["selector"].top_k(state["q"], state["k"])


PATHS = {"decode": (_prepare_decode, _run_decode), "tokens": (_prepare_tokens, _run_tokens),
         "prefill": (_prepare_prefill, _run_prefill), "select": (_prepare_select, _run_select)}


def prepare(case, seed):
    state = PATHS[case["path"]][0](case, seed)
    state["case"] = case
    return state


def run(state):
    case = state["case"]
    return PATHS[case["path"]][1](case, state)


# ---- what a pass cannot do without -----------------------------------------------------------------------

def work(case):
    e, hk, rep, d = ELEMENT_BYTES[case["dtype"]], case["hk"], case["rep"], case["d"]
    hq = hk * rep
    if case["path"] == "select":
        n = case["pages"]
        return {"bytes": 2 * hk * n * d * e + hq * d * e + hq * case["k"] * 8, "flops": 4 * hq * n * d}
    if case["path"] == "prefill":
        s = case["prompt"]
        prefix = max(0, (s - case["local"] + case["page"]) // case["page"] * case["page"])
        built = 2 * prefix * hk * d * e          # pages in host memory, or the resident prefix
        if prefix > case["lru"]:
            built += 2 * case["lru"] * hk * d * e + 2 * (prefix // case["page"]) * hk * d * e
        return {"bytes": (2 * hq + 2 * hk) * s * d * e + built, "flops": 2 * hq * d * s * (s + 1)}
    tokens = case.get("tokens", 1)
    resident = case["dram"] <= case["lru"]
    prefix = case["dram"] if resident else case["lru"] // case["page"] * case["page"]
    local = case["local"] + case["tail"] - case["page"] + OUTPUT // 2
    n_pages = 0 if resident else case["dram"] // case["page"]
    # page summaries, slot table, local window, queries and outputs, new keys and values in and into the window
    size = (2 * hk * n_pages + 2 * hk * (prefix + local) + tokens * (2 * hq + 4 * hk)) * d * e
    flops = tokens * hq * d * (4 * n_pages + 4 * (prefix + local))
    layers = case.get("layers", 1)
    return {"bytes": size * layers, "flops": flops * layers}


def tolerance(case):
    # outputs carry the rounding of the element type and of P, which the tensor cores take in it; page lists and
    # slot tables may differ where two scores tie to the last bit of a float32 sum
    return {"rel": {"bf16": 1e-2, "fp16": 2e-3, "fp32": 1e-5}[case["dtype"]], "differ": 1e-3}
