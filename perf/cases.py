"""The work that a program using this package has it do, as measurable cases.

Five kinds, all through the entry points that stand in for the reference's Python surface:

* ``decode``   one token's wave-index attention: ``retroinfer_cache.decode_update_kv_cache`` followed by
               ``attn_hub.retroinfer_decode_attn``, layer after layer, index and KV in HBM;
* ``host``     the same two calls with the clustered KV in pinned host memory (``kv_on_host=True``);
* ``dense``    the full-attention comparator: ``flash_attn_cache`` with ``attn_hub.decode_full_flash_attn``;
* ``prefill``  ``attn_hub.retroinfer_prefill_attn`` over a prompt;
* ``index``    ``retroinfer_cache.prefill_update_kv_cache``: clustering and layout of one request's layer.

The caches advance their length at the model's last layer.  The decode kinds run the layers in front of it (the share of
one GPU of a model whose layers are split over several), so a pass can be repeated at the same length: it writes the same
row of the steady zone (or of the dense cache) again.
"""
import math

import torch

from retrievalattention_b200.attn_hub import (decode_full_flash_attn, prefill_full_flash_attn, retroinfer_decode_attn,
                                               retroinfer_prefill_attn)
from retrievalattention_b200.cache_hub import flash_attn_cache, retroinfer_cache
from retrievalattention_b200.config import generate_config
from retrievalattention_b200.synthetic import make_kv

DIM = 128
SINK, RECENT = 4, 64
BUDGET, ESTIMATE = 0.018, 0.232          # retrieval budget and estimation share of the benchmark configurations
ITERS = 10                               # Lloyd iterations of the index build
HOST_STEPS = 32                          # queries that a host-tier state steps through
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


def listed():
    return [
        # -- decode, wave index in HBM.  `pad`: left padding of the last request (prompts of different lengths)
        # a short context and one user: launches and host work count
        dict(name="decode-8k-b1", kind="decode", batch=1, kv_heads=8, group=4, context=8192, layers=4, dtype="bf16", pad=0),
        # an ordinary batch of uneven prompts, no size a power of two, GQA 7
        dict(name="decode-45k-b3-ragged", kind="decode", batch=3, kv_heads=4, group=7, context=45003, layers=4, dtype="fp16",
             pad=9001),
        # Llama-3-8B geometry, 128K context, batch 4: the benchmark's default workload
        dict(name="decode-128k-b4", kind="decode", batch=4, kv_heads=8, group=4, context=131072, layers=4, dtype="bf16",
             pad=0),
        # one KV head of Qwen2.5-72B geometry, as one GPU of eight holds it, batch 16
        dict(name="decode-128k-shard", kind="decode", batch=16, kv_heads=1, group=8, context=131072, layers=4, dtype="bf16",
             pad=0),
        # Qwen2.5-7B geometry at 256K, batch 8: 16384 centroids per head
        dict(name="decode-256k-b8", kind="decode", batch=8, kv_heads=4, group=7, context=262144, layers=2, dtype="bf16",
             pad=0),
        # -- the same with the clustered KV in pinned host memory and a page cache on the GPU; queries drift from token to token
        dict(name="host-64k-b4", kind="host", batch=4, kv_heads=4, group=7, context=65536, layers=2, dtype="bf16", pad=0),
        # -- full attention over the whole cache, batch of uneven prompts
        dict(name="dense-32k-b4", kind="dense", batch=4, kv_heads=8, group=4, context=32768, layers=4, dtype="bf16", pad=5000),
        # -- attention over the prompt: a question, an ordinary document of odd length, a long one
        dict(name="prefill-777", kind="prefill", batch=1, kv_heads=8, group=4, tokens=777, causal=True, dtype="bf16"),
        dict(name="prefill-5001-b2", kind="prefill", batch=2, kv_heads=4, group=7, tokens=5001, causal=True, dtype="fp16"),
        dict(name="prefill-32k", kind="prefill", batch=1, kv_heads=8, group=4, tokens=32768, causal=True, dtype="bf16"),
        # -- the index of one request's layer: the shortest context with a full-size index, and 128K
        dict(name="index-8k", kind="index", kv_heads=8, context=8192, dtype="bf16", pad=0),
        dict(name="index-128k", kind="index", kv_heads=8, context=131072, dtype="bf16", pad=0),
    ]


def _between(rng, low, high):
    """A whole number from low to high, spread over the logarithm."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(("decode", "decode", "decode", "prefill", "prefill", "index", "index", "dense", "host"))
    dtype = rng.choice(("bf16", "bf16", "fp16"))
    kv_heads, group = rng.choice(((8, 4), (4, 7), (1, 8), (2, 8), (8, 8), (4, 1), (2, 5), (8, 2)))
    if kind == "prefill":
        tokens = _between(rng, 200, 24000)
        batch = rng.randint(1, 4) if tokens < 4000 else 1
        return dict(kind=kind, batch=batch, kv_heads=kv_heads, group=group, tokens=tokens, causal=rng.random() < 0.85,
                    dtype=dtype)
    if kind == "index":
        context = _between(rng, 4096, 131072)
        return dict(kind=kind, kv_heads=kv_heads, context=context, dtype=dtype, pad=rng.choice((0, rng.randint(1, 999))))
    if kind == "host":
        context = _between(rng, 8192, 65536)
        batch = rng.randint(1, max(1, min(8, 16 // kv_heads)))
        return dict(kind=kind, batch=batch, kv_heads=kv_heads, group=group, context=context, layers=2, dtype=dtype, pad=0)
    context = _between(rng, 4096, 200000 if kind == "decode" else 50000)
    most = (1 << 22) if kind == "decode" else (1 << 20)                  # rows of K (and of V) a layer holds
    batch = rng.randint(1, max(1, min(16, most // (kv_heads * context))))
    pad = rng.choice((0, rng.randint(1, context // 4))) if batch > 1 else 0
    return dict(kind=kind, batch=batch, kv_heads=kv_heads, group=group, context=context, layers=rng.randint(2, 4), dtype=dtype,
                pad=pad)


def _starts(case):
    """First valid token of every request: left padding from none (first request) to `pad` (last one)."""
    b = case.get("batch", 1)
    return [case["pad"] if b == 1 else case["pad"] * i // (b - 1) for i in range(b)]


def _randn(shape, seed, dtype):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32).to(dtype)


def _wave_cache(case, layers, **more):
    batch, kv_heads, context = case.get("batch", 1), case["kv_heads"], case["context"]
    max_new = 64
    cfg = generate_config(context, BUDGET, ESTIMATE)
    return retroinfer_cache(_starts(case), layers, batch, context + max_new, kv_heads, kv_heads * case.get("group", 4), DIM,
                            DTYPES[case["dtype"]], {str(i): "cuda:0" for i in range(layers)}, max_new, num_gpus=1, model_size=8,
                            **cfg.as_kwargs(), **more)


def _step_inputs(case, seed, steps):
    """Queries, keys and values of a token for every layer that runs; with several steps the queries drift."""
    dtype, b, hk = DTYPES[case["dtype"]], case["batch"], case["kv_heads"]
    hq = hk * case["group"]
    q = [_randn((case["layers"], b, 1, hq, DIM), seed * 7919 + 1, torch.float32)]
    for i in range(1, steps):
        q.append(0.95 * q[-1] + 0.31 * _randn(q[0].shape, seed * 7919 + 10 + i, torch.float32))
    k = _randn((case["layers"], b, 1, hk, DIM), seed * 7919 + 2, dtype)
    v = _randn((case["layers"], b, 1, hk, DIM), seed * 7919 + 3, dtype)
    return [[x.to(dtype) for x in s.unbind(0)] for s in q], list(k.unbind(0)), list(v.unbind(0))


def prepare(case, seed):
    dtype, kind = DTYPES[case["dtype"]], case["kind"]
    state = dict(case=case)
    if kind == "prefill":
        b, s, hk = case["batch"], case["tokens"], case["kv_heads"]
        hq = hk * case["group"]
        kv = [make_kv(hk, s, DIM, seed=seed * 31 + i, device="cuda", dtype=dtype) for i in range(b)]
        state["q"] = _randn((b, s, hq, DIM), seed * 31 + 17, dtype)
        state["k"], state["v"] = (torch.cat([x[j] for x in kv], 0).contiguous() for j in (0, 1))
        return state
    if kind == "index":
        state["cache"] = _wave_cache(case, 1)
        state["k"], state["v"] = make_kv(case["kv_heads"], case["context"], DIM, seed=seed * 31, device="cuda", dtype=dtype)
        return state
    layers = case["layers"] + 1          # the last one is not run (see the top) and holds nothing
    if kind == "dense":
        cache = flash_attn_cache(_starts(case), layers, case["batch"], case["context"] + 64, case["kv_heads"],
                                 case["kv_heads"] * case["group"], DIM, dtype, {str(i): "cuda:0" for i in range(layers)}, 1, 8)
    else:
        cache = _wave_cache(case, layers, **(dict(kv_on_host=True) if kind == "host" else {}))
    for layer in range(case["layers"]):
        for b in range(case["batch"]):
            k, v = make_kv(case["kv_heads"], case["context"], DIM, seed=(seed * 31 + layer) * 31 + b, device="cuda", dtype=dtype)
            cache.prefill_update_kv_cache(None, k, v, layer, b)
            cache.sync(layer, b)
    if kind != "dense":
        cache.prepare_cache()
    state["cache"], state["step"] = cache, 0
    state["q"], state["k"], state["v"] = _step_inputs(case, seed, HOST_STEPS if kind == "host" else 1)
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "prefill":
        attend = retroinfer_prefill_attn if case["causal"] else prefill_full_flash_attn
        return attend(state["q"], state["k"], state["v"], case["causal"])
    cache = state["cache"]
    if kind == "index":
        cache.prefill_update_kv_cache(None, state["k"], state["v"], 0, 0)
        return [t[0] for t in (cache.centroids, cache.value_sum, cache.cluster_size, cache.cluster_count, cache.cluster_offset,
                               cache.list_keys, cache.list_values, cache.steady_zone_keys, cache.steady_zone_values)]
    queries = state["q"][state["step"] % len(state["q"])]
    state["step"] += 1
    outs = []
    for layer in range(case["layers"]):
        kept = cache.decode_update_kv_cache(state["k"][layer], state["v"][layer], layer)
        if kind == "dense":
            outs += [decode_full_flash_attn(queries[layer], kept[0], kept[1], layer, cache), *kept]
        else:
            outs += [retroinfer_decode_attn(queries[layer], None, None, layer, cache), cache.steady_zone_keys[layer],
                     cache.steady_zone_values[layer]]
    return outs


def work(case):
    kind, d = case["kind"], DIM
    hk, b = case["kv_heads"], case.get("batch", 1)
    if kind == "prefill":
        s, hq = case["tokens"], hk * case["group"]
        pairs = s * (s + 1) / 2 if case["causal"] else s * s
        return {"bytes": 2 * d * b * s * (2 * hq + 2 * hk), "flops": 4 * d * b * hq * pairs}
    rows = [case["context"] - start for start in _starts(case)]          # tokens of every request
    if kind == "dense":
        layers, hq = case["layers"], hk * case["group"]
        tokens = sum(n + 1 for n in rows)
        return {"bytes": layers * (2 * d * 2 * hk * tokens + 2 * d * 2 * b * hq), "flops": layers * 4 * d * hq * tokens}
    cfg = generate_config(case["context"], BUDGET, ESTIMATE)
    c = cfg.n_centroids
    if kind == "index":
        n = rows[0] - SINK - RECENT
        flops = 2 * d * hk * n * ((ITERS - 1) * c / cfg.n_segment + c)
        # K and V in and out once each; centroids, value sums, sizes, counts and offsets out
        return {"bytes": hk * (4 * 2 * d * n + c * (4 * d + 10)), "flops": flops}
    # a token and layer: every centroid, the estimation zone's value sums, K and V of the steady zone and of the retrieved
    # clusters.  Clusters near a query hold about 0.7 of the mean size on these inputs.
    g, gs, layers = b * hk, case["group"], case["layers"]
    est = cfg.max_compute_cluster_num - cfg.nprobe
    exact = SINK + RECENT + 1 + 0.7 * cfg.nprobe * sum(n - SINK - RECENT for n in rows) / (b * c)
    per_group = 2 * d * (c + est + 2 * exact) + 2 * c + 4 * d * gs
    flops = 2 * d * gs * (c + est + 2 * exact)
    return {"bytes": layers * g * per_group, "flops": layers * g * flops}


def tolerance(case):
    if case["kind"] == "index":
        # centroids and value sums are rounded to 16 bits from 32-bit sums; sizes, offsets and the row order are whole
        # numbers that a token between two equally near centroids may change
        return {"rel": 1e-2, "differ": 1e-3}
    # 16-bit results of 32-bit accumulation; probabilities are 16-bit operands of the second product
    return {"rel": 1e-2}
