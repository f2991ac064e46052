"""Workloads of the framework, through the entry points that a program uses: the cache classes
(``prefill_update_kv_cache`` / ``decode_update_kv_cache`` / ``compute``), the operator modules under ``cache_hub`` and
the dense one-token products of a decode step.

    listed()            the named cases
    draw(rng)           another case of the same ranges
    prepare(case, seed) inputs and the cache, weights or buffers that a program keeps
    run(state)          one pass
    work(case)          bytes and operations that a pass cannot do without
    tolerance(case)     how far two correct implementations may differ

Kinds of case
    decode    one decode token through the attention of `layers` layers: append the K/V row, retrieve, attend.  Called
              eagerly, as a model runtime calls the cache, or replayed as one captured graph, as a serving loop does.
    prefill   a prompt of every sample into the cache: key coding, cluster histograms, K/V rows into the store.
    ops       the retrieval chain from the stand-alone operators, on tensors that the caller keeps.
    dense     the projections, norms, rotary embedding and gated activation of one token through `layers` layers.
"""
import math

import torch

from pariskv_b200 import _lib, ops
from pariskv_b200.cache_hub import polar_cache_adaptivek_varlen, polar_cache_atten_value_indices_adaptive_k
from pariskv_b200.cache_hub.collision_fused.collison_interface import update_cache_cnt_cuda_interface
from pariskv_b200.cache_hub.gather_trans.trans_h2d import h2d_gather_kv
from pariskv_b200.cache_hub.polar_cache import TIER_RATIOS, polar_cache
from pariskv_b200.cache_hub.rerank.rerank import partial_rerank_cuda
from pariskv_b200.cache_hub.topk import bucket_topk

DEV = "cuda:0"
OUTLIERS = (7, 37, 71, 101)   # key channels with large values
POOL = 32                     # decode steps whose q / k / v rows are made ahead of time, used in turn
CLASSES = {"topk": polar_cache, "adaptive": polar_cache_adaptivek_varlen.polar_cache,
           "adaptive_dense": polar_cache_atten_value_indices_adaptive_k.polar_cache}


def _decode(**kw):
    case = dict(kind="decode", cls="topk", graph=False, offload=False, layers=2, batch=1, kv_heads=8, q_heads=32,
                context_lo=32768, context_hi=32768, sink=4, local=64, interval=128, topk=2048, threshold=2000,
                max_new=4096)
    case.update(kw)
    return case


def _prefill(**kw):
    case = dict(kind="prefill", cls="topk", offload=True, layers=1, batch=1, kv_heads=8, q_heads=32, context_lo=8192,
                context_hi=8192, sink=4, local=64, interval=128, topk=2048, threshold=2000, max_new=512)
    case.update(kw)
    return case


def listed():
    return [
        # a chat turn on a short prompt: below the threshold every row is attended; nothing but launches and host time
        _decode(name="decode_short_prompt", layers=4, context_lo=701, context_hi=701, threshold=4096, topk=100,
                interval=512, max_new=512),
        # the cache class with the defaults of its constructor (top-100, update buffer 512, rows in host memory),
        # called layer by layer from a model runtime; an odd prompt length
        _decode(name="decode_defaults_10k", offload=True, layers=4, context_lo=10007, context_hi=10007, topk=100,
                interval=512, max_new=2048),
        # the 128K-context configuration: rows in pinned host memory, top-2048, replayed as a graph
        _decode(name="decode_128k_host", graph=True, offload=True, layers=2, context_lo=131072, context_hi=131072),
        # the same with the rows in HBM
        _decode(name="decode_128k_hbm", graph=True, layers=4, context_lo=131072, context_hi=131072),
        # the million-token configuration on one GPU, one layer of it
        _decode(name="decode_1m_hbm", graph=True, layers=1, context_lo=1048576, context_hi=1048576),
        # the batched configuration: sequences of different lengths
        _decode(name="decode_varlen_b16", graph=True, layers=2, batch=16, context_lo=16384, context_hi=32768),
        # the same with the adaptive budget of 1024 - 4096 rows per head, called eagerly
        _decode(name="decode_adaptive_b8", cls="adaptive", layers=2, batch=8, context_lo=16384, context_hi=32768),
        # one rank's share of a 64 / 8-head model over 8 GPUs: one KV head with eight query heads, batch 8
        _decode(name="decode_tp_share_b8", graph=True, layers=4, batch=8, kv_heads=1, q_heads=8, context_lo=65536,
                context_hi=65536),
        # a batch of two short prompts of different lengths, rows to host memory
        _prefill(name="prefill_3k_b2", layers=2, batch=2, context_lo=2477, context_hi=3001),
        # a long prompt, rows kept in HBM
        _prefill(name="prefill_128k", offload=False, context_lo=131072, context_hi=131072),
        # the single-layer operator configuration: 32768 keys, 4096 candidates, top-256, plane-major tensors
        dict(name="ops_32k", kind="ops", key_major=False, batch=1, kv_heads=8, q_heads=32, keys=32768, candidates=4096,
             topk=256),
        # the dense part of a decode token, 32 / 8 heads, hidden 4096, feed-forward 12288
        dict(name="dense_4096", kind="dense", layers=2, hidden=4096, q_heads=32, kv_heads=8, ffn=12288),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "decode", "short", "prefill", "prefill", "ops", "dense"])
    kv_heads, group = rng.choice([1, 2, 4, 8]), rng.choice([1, 2, 4, 4, 5, 8])
    shape = dict(kv_heads=kv_heads, q_heads=kv_heads * group)
    if kind == "short":
        n = _log_int(rng, 200, 3500)
        return _decode(offload=rng.random() < 0.5, layers=rng.choice([1, 2, 4]), batch=rng.choice([1, 1, 2, 4]),
                       context_lo=n, context_hi=n, threshold=4096, topk=_log_int(rng, 64, 1024),
                       interval=rng.choice([128, 256, 512]), max_new=512, **shape)
    if kind == "decode":
        graph, cls = rng.random() < 0.5, rng.choice(["topk", "topk", "topk", "adaptive", "adaptive_dense"])
        offload = rng.random() < 0.25
        layers, batch = rng.choice([1, 2, 4]), rng.choice([1, 1, 2, 3, 8, 16])
        budget = (1 << 20 if offload else 1 << 22) // (kv_heads * layers * batch)   # keys per sample and head
        hi = _log_int(rng, 4097, max(4200, min(1 << 20, budget)))
        lo = hi if batch == 1 else max(4097, int(hi * rng.uniform(0.5, 1.0)))
        # contexts lie above the full-attention threshold, which grows with the top-k
        topk = min(_log_int(rng, 64, 2048), (lo - 512) // 2)
        return _decode(cls=cls, graph=graph, offload=offload, layers=layers, batch=batch, context_lo=lo, context_hi=hi,
                       local=rng.choice([16, 64, 256]), interval=rng.choice([64, 128, 256, 512]), topk=topk,
                       max_new=2048, **shape)
    if kind == "prefill":
        cls, offload = rng.choice(["topk", "topk", "adaptive"]), rng.random() < 0.5
        batch = rng.choice([1, 1, 2, 4])
        hi = _log_int(rng, 1000, (1 << 18 if offload else 1 << 20) // (kv_heads * batch))
        lo = hi if batch == 1 else max(700, int(hi * rng.uniform(0.6, 1.0)))
        return _prefill(cls=cls, offload=offload, batch=batch, context_lo=lo, context_hi=hi, **shape)
    if kind == "ops":
        keys = _log_int(rng, 2000, 131072)
        cand = max(64, int(keys * rng.uniform(0.05, 0.3)))
        return dict(kind="ops", key_major=rng.random() < 0.5, batch=rng.choice([1, 1, 2, 4]), keys=keys, candidates=cand,
                    topk=max(16, int(cand * rng.uniform(0.05, 0.5))), **shape)
    hidden = 128 * rng.randint(8, 40)
    heads = max(1, hidden // 128 // (kv_heads * group))
    return dict(kind="dense", layers=2, hidden=hidden, q_heads=kv_heads * group * heads, kv_heads=kv_heads * heads,
                ffn=8 * rng.randint(hidden // 4, 3 * hidden // 8))


# ---------------------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------------------
def _lengths(case):
    """Prompt length of every sample: evenly spread from context_lo to context_hi, the longest last."""
    b, lo, hi = case["batch"], case["context_lo"], case["context_hi"]
    return [hi if b == 1 else lo + (hi - lo) * i // (b - 1) for i in range(b)]


def _rows(g, *shape):
    """K rows with the distribution of cached keys: normal, a few channels eight times larger, log-normal norms."""
    k = torch.randn(*shape, 128, generator=g, device=DEV)
    k[..., list(OUTLIERS)] *= 8.0
    return (k * torch.exp(0.5 * torch.randn(*shape, 1, generator=g, device=DEV))).to(torch.bfloat16)


def _queries(g, keys, G):
    """Queries [.., H * G, 128] that point in part at the given keys [.., H, 128], with the norm of RMS-normed rows."""
    k = keys.float()
    q = (0.3 * k / k.norm(dim=-1, keepdim=True)).unsqueeze(-2).expand(*k.shape[:-1], G, 128)
    q = q + torch.randn(q.shape, generator=g, device=DEV) / math.sqrt(128.0)
    q = q / q.norm(dim=-1, keepdim=True) * math.sqrt(128.0)
    return q.reshape(*k.shape[:-2], k.shape[-2] * G, 128).to(torch.bfloat16)


def _cache(case):
    """The cache object, its samples padded on the left to the longest prompt."""
    lengths = _lengths(case)
    longest, extra = max(lengths), {}
    if case["cls"] == "adaptive":
        extra = dict(adaptive_topk_min_k=1024, adaptive_topk_max_k=4096)
    return CLASSES[case["cls"]](
        valid_start=[longest - n for n in lengths], layer_num=case["layers"], batch_size=case["batch"],
        max_length=longest + case["max_new"], num_key_value_heads=case["kv_heads"], num_heads=case["q_heads"],
        head_dim=128, dtype=torch.bfloat16, layer_mapping={str(i): DEV for i in range(case["layers"])},
        max_new_length=case["max_new"], sink_size=case["sink"], local_size=case["local"], final_topk=case["topk"],
        dynamic_update_interval=case["interval"], full_attention_threshold=case["threshold"],
        enable_offload=case["offload"], **extra)


def _fill(state):
    """The prompt of every sample into the cache."""
    for l, (k, v) in enumerate(state["prompt"]):
        state["cache"].prefill_update_kv_cache(None, k, v, l, 0)
        state["cache"].sync(l, 0)
    state["produced"] = 0


def _prompt(case, g):
    shape = (case["batch"], max(_lengths(case)), case["kv_heads"])
    return [(_rows(g, *shape), torch.randn(*shape, 128, generator=g, device=DEV, dtype=torch.bfloat16))
            for _ in range(case["layers"])]


def _decode_step(state, row):
    """One token through the cache of every layer; row(pool) picks this step's rows out of a pool."""
    cache, outs = state["cache"], []
    for l in range(cache.layer_num):
        cache.decode_update_kv_cache(row(state["k"][l]), row(state["v"][l]), l)
        outs.append(cache.compute(row(state["q"][l]), l))
        outs.append(cache.last_topk_indices)
        outs.append(cache.unified_keys_gpu[l])
        outs.append(cache.unified_values_gpu[l])
    return outs


def _prepare_decode(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    cache, lengths = _cache(case), _lengths(case)
    state = dict(case=case, cache=cache, prompt=_prompt(case, g), q=[], k=[], v=[], graph=None)
    _fill(state)
    H, G = case["kv_heads"], case["q_heads"] // case["kv_heads"]
    for l in range(case["layers"]):
        state["k"].append(_rows(g, POOL, case["batch"], 1, H))
        state["v"].append(torch.randn(POOL, case["batch"], 1, H, 128, generator=g, device=DEV, dtype=torch.bfloat16))
        at = torch.randint(max(lengths) - min(lengths), max(lengths), (POOL,), generator=g, device=DEV)
        picked = state["prompt"][l][0][:, at].transpose(0, 1).unsqueeze(2)       # [POOL, batch, 1, H, 128]
        state["q"].append(_queries(g, picked, G).contiguous())
    if case["graph"]:
        # one graph for the whole generation: every position lives in device words, the step counter too
        step = state["step"] = torch.zeros(1, dtype=torch.int64, device=DEV)   # the graph reads it: kept with it
        cache.queries_precede_append = True
        kept, side, graph = cache.host_state(), torch.cuda.Stream(), torch.cuda.CUDAGraph()
        side.wait_stream(torch.cuda.current_stream())
        _lib.set_pdl(True)
        try:
            with torch.cuda.stream(side):
                graph.capture_begin()
                state["out"] = _decode_step(state, lambda pool: pool.index_select(0, step)[0])
                step.add_(1).remainder_(POOL)
                graph.capture_end()
        finally:
            _lib.set_pdl(False)
        torch.cuda.current_stream().wait_stream(side)
        cache.set_host_state(kept)
        state["graph"] = graph
    return state


def _run_decode(state):
    cache = state["cache"]
    if state["produced"] == state["case"]["max_new"]:   # the generation is over: the next request, same prompt
        _fill(state)
    state["produced"] += 1
    if state["graph"] is not None:
        state["graph"].replay()
        cache.note_replayed_step()
        return state["out"]
    t = state["produced"] % POOL
    return _decode_step(state, lambda pool: pool[t])


def _prepare_prefill(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return dict(case=case, cache=_cache(case), prompt=_prompt(case, g))


def _run_prefill(state):
    _fill(state)
    cache, outs = state["cache"], []
    n = max(max(z) for z in cache.zone_len)
    for l in range(cache.layer_num):
        if cache.enable_offload:
            k, v = cache.unified_keys_cpu[l], cache.unified_values_cpu[l]
        else:
            k, v = cache._store_k[l], cache._store_v[l]
        outs += [cache.codebook_gpu[l][..., :n], cache.key_block_weight_gpu[l][..., :n],
                 cache.key_4bit_packed_gpu[l][..., :n, :], cache.cluster_key_counts_gpu[l], k[:, :, :n], v[:, :, :n],
                 cache.unified_keys_gpu[l], cache.unified_values_gpu[l]]
        if state["case"]["cls"] != "topk":
            outs.append(cache.value_norm_gpu[l][..., :n])
    return outs


def _prepare_ops(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    b, H, N = case["batch"], case["kv_heads"], case["keys"]
    signs = torch.randint(0, 2, (128,), generator=g, device=DEV).to(torch.bfloat16) * 2 - 1
    keys = _rows(g, b, H, N)
    counts = torch.zeros(b, H, 16, 256, dtype=torch.int32, device=DEV)
    codes, weight, packed = ops.encode_keys(keys, signs, cluster_counts=counts)
    if not case["key_major"]:      # the plane-major tensors of the reference's own operators
        codes, weight, packed = codes.contiguous(), weight.contiguous(), packed.contiguous()
    at = torch.randint(0, N, (1,), generator=g, device=DEV)
    q = _queries(g, keys[:, :, at].transpose(1, 2), case["q_heads"] // H).contiguous()
    centers = torch.tensor([0.0420, 0.1266, 0.2130, 0.3025, 0.3973, 0.5001, 0.6169, 0.7633], dtype=torch.bfloat16,
                           device=DEV)
    host_k = torch.empty(b, H, N, 128, dtype=torch.bfloat16, pin_memory=True)
    host_v = torch.empty(b, H, N, 128, dtype=torch.bfloat16, pin_memory=True)
    host_k.copy_(keys)
    host_v.copy_(torch.randn(b, H, N, 128, generator=g, device=DEV, dtype=torch.bfloat16))
    rows_k = torch.zeros(b, H, case["topk"], 128, dtype=torch.bfloat16, device=DEV)
    return dict(case=case, q=q, signs=signs, centers=centers, codes=codes, weight=weight, packed=packed, counts=counts,
                host_k=host_k, host_v=host_v, rows_k=rows_k, rows_v=torch.zeros_like(rows_k),
                tiers=[math.ceil(N * 0.2 * r) for r in TIER_RATIOS])


def _run_ops(s):
    case = s["case"]
    q_blocks, q_norm = ops.query_prep(s["q"], case["kv_heads"], s["signs"])
    order = ops.rank_clusters(q_blocks)
    cnt = update_cache_cnt_cuda_interface(order, s["counts"], s["codes"], s["tiers"])
    cand = bucket_topk(cnt, case["candidates"])
    scores, _ = partial_rerank_cuda(cand, s["packed"], s["weight"], q_blocks, q_norm, s["centers"], 16, 8)
    final = ops.final_topk(scores.float(), cand, case["topk"])
    h2d_gather_kv(s["host_k"], s["host_v"], final, s["rows_k"], s["rows_v"])
    return [q_blocks, q_norm, order, cnt, cand, scores, final, s["rows_k"], s["rows_v"]]


def _prepare_dense(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    hid, ffn, q, kv = case["hidden"], case["ffn"], case["q_heads"], case["kv_heads"]

    def w(*shape, std=0.02):
        return (torch.randn(*shape, generator=g, device=DEV) * std).to(torch.bfloat16)

    layers = [dict(qkv=w((q + 2 * kv) * 128, hid), o=w(hid, q * 128), gate_up=w(2 * ffn, hid), down=w(hid, ffn),
                   norm1=1 + w(hid), norm2=1 + w(hid), head_norm=1 + w(q + kv, 128)) for _ in range(case["layers"])]
    ang = torch.rand(1, 64, generator=g, device=DEV) * 6.28
    cos, sin = torch.cos(ang), torch.sin(ang)
    return dict(case=case, layers=layers, x=w(1, hid, std=1.0), attn=[w(1, q * 128, std=1.0) for _ in layers],
                cos=torch.cat([cos, cos], -1).to(torch.bfloat16), sin=torch.cat([-sin, sin], -1).to(torch.bfloat16))


def _run_dense(s):
    h, outs = s["x"], []
    for w, attn in zip(s["layers"], s["attn"]):
        h, x = ops.add_rmsnorm(h, None, w["norm1"])
        qkv = ops.gemv(w["qkv"], x)
        outs += [qkv, ops.qk_norm_rope(qkv, w["head_norm"], s["cos"], s["sin"])]
        h, x = ops.add_rmsnorm(ops.gemv(w["o"], attn), h, w["norm2"])
        h, _ = ops.add_rmsnorm(ops.gemv(w["down"], ops.gemv(w["gate_up"], x, gated=True)), h, w["norm1"])
        outs += [h, x]
    return outs


def prepare(case, seed):
    return {"decode": _prepare_decode, "prefill": _prepare_prefill, "ops": _prepare_ops,
            "dense": _prepare_dense}[case["kind"]](case, seed)


def run(state):
    return {"decode": _run_decode, "prefill": _run_prefill, "ops": _run_ops,
            "dense": _run_dense}[state["case"]["kind"]](state)


# ---------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "dense":
        hid, ffn, q, kv = case["hidden"], case["ffn"], case["q_heads"], case["kv_heads"]
        params = hid * (q + 2 * kv) * 128 + hid * q * 128 + 3 * hid * ffn
        return {"bytes": 2.0 * params * case["layers"], "flops": 2.0 * params * case["layers"]}
    H, G = case["kv_heads"], case["q_heads"] // case["kv_heads"]
    if kind == "ops":   # codes, counts out, candidate records and scores, rows over the host link and into HBM
        N, C, K = case["keys"], case["candidates"], case["topk"]
        n = 16 * N + 4 * N + (96 + 8 + 2) * C + 8 * K + 2 * 512 * K + 3 * 16 * 256 * 4
        return {"bytes": float(n * H * case["batch"]), "flops": float((16 * N + 288 * C) * H * case["batch"])}
    steady = case["sink"] + case["local"]
    if kind == "prefill":   # K and V rows read, rows and the 112-byte record of a key written
        tokens = sum(_lengths(case)) * H * case["layers"]
        return {"bytes": float(tokens * (512 + 512 + 112 + (4 if case["cls"] != "topk" else 0))),
                "flops": float(tokens * 128 * 12)}
    total_b = total_f = 0.0
    window = steady + case["interval"] // 2
    ratio = ((5000, 0.5), (10000, 0.25), (30000, 0.2), (1 << 40, 0.1 if case["cls"] == "topk" else 0.05))
    for n in _lengths(case):
        zone = n - steady
        if n < max(case["threshold"], steady + 2 * case["topk"]):     # every row is attended
            b, f = 512 * n, 4 * 128 * G * n
        else:
            cand = math.ceil(zone * next(r for bound, r in ratio if zone < bound))
            most = {"topk": case["topk"], "adaptive": 4096, "adaptive_dense": 2048}[case["cls"]]
            rows = min(most, cand) + window
            b = 16 * zone + 96 * cand + 16 * 256 * 4 + 512 * rows + (4 * cand if case["cls"] != "topk" else 0)
            f = 16 * zone + 288 * cand + 4 * 128 * G * rows
        total_b += H * (b + 512 * (G + 1))
        total_f += H * f
    return {"bytes": total_b * case["layers"], "flops": total_f * case["layers"]}


def tolerance(case):
    """bf16 results; indices, codes and counts are whole numbers and the same (ties go to the lowest index).  The
    adaptive selection orders benefits that a differently rounded window logit can move past each other."""
    if case["kind"] == "prefill":   # codes, copies, bf16 weights; value norms are 32-bit sums
        return {"rel": 1e-5}
    if case["kind"] == "decode" and case["cls"] != "topk":
        return {"rel": 1e-2, "differ": 0.005}
    return {"rel": 1e-2}
