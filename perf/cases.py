"""What the speed of this package is judged by: the calls its users make, over the range of sizes they make them at.

Three kinds of program use the package, and every case is one call of one of them on one attention layer:

* a program with its own tensors calls ``hip_attention_12`` (dense keys in prefill, a page pool in decode);
* an inference server calls ``forward_paged_hip`` with its token-granular pools, its per-layer configuration (rotary
  embedding inside the kernels) and, in decode, ``HiPMetadataCachePool`` around the call;
* a very long sequence is decoded in sequence shards with ``hip_attention_12_sequence_sharded``.

Inputs are drawn on the GPU: q, k, v ~ N(0, 1), every hundredth key token four times as long (the heavy hitters that the
estimator looks for), q carrying the softmax scale where the caller applies it.  Where keys arrive already rotated the
rotation is left out: rotating independent normal vectors gives independent normal vectors again.
"""
import math

import torch

from hip_attention_b200 import HiPAttentionArgs, ScanStage, hip_attention_12
from hip_attention_b200.serving import HiPAttentionConfig, HiPMetadataCachePool, forward_paged_hip
from hip_attention_b200.sharded import hip_attention_12_sequence_sharded

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}

# chunk sizes, tokens kept after each stage, query stride per stage, sink, window, query block
PLANS = {
    "long": dict(chunks=(256, 32, 8), keep=(32768, 8192, 2048), strides=(4, 4, 1), sink=256, window=1024, bq=64),
    "gqa": dict(chunks=(256, 32, 8), keep=(65536, 16384, 4096), strides=(4, 4, 1), sink=256, window=2048, bq=128),
    "short": dict(chunks=(32, 8), keep=(1024, 512), strides=(4, 1), sink=64, window=256, bq=64),
}
SERVER_LAYERS = {"dense": 0, "sparse": 5}    # layer ids of the default configuration's two kinds of layer


def listed():
    return [
        # The smallest call: one chat, a few thousand tokens, the mask of an earlier step.  Made once per layer and token.
        dict(name="decode_cached_one", kind="decode", B=1, T=6007, page=16, H=32, HKV=8, D=128, dtype="bf16", plan="long", ragged=False, cached=True),
        # Batched decode at full context as the benchmark has it: the steps between two mask refreshes ...
        dict(name="decode_cached_128k", kind="decode", B=32, T=131072, page=64, H=32, HKV=8, D=128, dtype="bf16", plan="long", ragged=False, cached=True),
        # ... and the refresh itself.
        dict(name="decode_refresh_128k", kind="decode", B=32, T=131072, page=64, H=32, HKV=8, D=128, dtype="bf16", plan="long", ragged=False, cached=False),
        # A server's decode step: a ragged batch, metadata pool around the call, mask estimated from scratch.
        dict(name="server_decode_fresh", kind="server_decode", B=12, ctx=40961, max_ctx=131072, H=32, HKV=8, D=128, dtype="bf16", layer="sparse", fp8=False, stages=0),
        # The commonest of a server's refreshes: restart at the last stage; here on an fp8 cache, in a dense layer.
        dict(name="server_decode_restart_fp8", kind="server_decode", B=5, ctx=21013, max_ctx=65536, H=32, HKV=8, D=128, dtype="bf16", layer="dense", fp8=True, stages=2),
        # One sequence of a million tokens in eight shards, mask estimated anew.
        dict(name="decode_sharded_1m", kind="sharded", B=1, T=1048576, shards=8, page=64, H=32, HKV=8, D=128, dtype="bf16", plan="long", cached=False),
        # A server's prefill chunk deep in a long prompt.
        dict(name="server_prefill_chunk", kind="server_prefill", B=1, chunk=8192, ctx=90112, max_ctx=131072, H=32, HKV=8, D=128, dtype="bf16", layer="sparse", fp8=False),
        # Two short prompts from their first token, in a dense layer (rotation to moving positions), fp8 cache.
        dict(name="server_prefill_first_fp8", kind="server_prefill", B=2, chunk=3001, ctx=3001, max_ctx=32768, H=32, HKV=8, D=128, dtype="fp16", layer="dense", fp8=True),
        # A small fp32 layer (the configuration that also runs on a CPU).
        dict(name="prefill_4k_fp32", kind="prefill", B=1, TQ=4096, T=4096, H=8, HKV=2, D=64, dtype="fp32", plan="short", stats=True),
        # Ragged sizes, small heads, default options.
        dict(name="prefill_odd_fp16", kind="prefill", B=2, TQ=2999, T=20011, H=16, HKV=4, D=64, dtype="fp16", plan="long", stats=True),
        # The benchmark's prefill: the last 32768 queries of a 131072-token prompt.
        dict(name="prefill_128k", kind="prefill", B=1, TQ=32768, T=131072, H=32, HKV=8, D=128, dtype="bf16", plan="long", stats=False),
        # A whole 131072-token prompt of a wide layer at once: the largest call.
        dict(name="prefill_gqa_whole", kind="prefill", B=1, TQ=131072, T=131072, H=64, HKV=8, D=128, dtype="bf16", plan="gqa", stats=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "server_decode", "server_decode", "server_prefill", "server_prefill", "prefill", "prefill", "prefill", "sharded"])
    if kind == "decode":
        T = _log_int(rng, 4096, 131072)
        H, HKV = rng.choice([(32, 8), (32, 8), (64, 8), (16, 4)])
        return dict(kind=kind, B=_log_int(rng, 1, 32), T=T, page=rng.choice([1, 16, 64]), H=H, HKV=HKV, D=128,
                    dtype=rng.choice(["bf16", "bf16", "fp16"]), plan="long", ragged=rng.random() < 0.5, cached=rng.random() < 0.5)
    if kind == "server_decode":
        max_ctx = rng.choice([65536, 131072])
        return dict(kind=kind, B=_log_int(rng, 1, 32), ctx=_log_int(rng, 2048, max_ctx - 1), max_ctx=max_ctx, H=32, HKV=8, D=128,
                    dtype=rng.choice(["bf16", "fp16"]), layer=rng.choice(["dense", "sparse", "sparse"]), fp8=rng.random() < 0.35,
                    stages=rng.choice([0, 1, 2, 3]))
    if kind == "server_prefill":
        chunk = _log_int(rng, 100, 8192)
        max_ctx = rng.choice([32768, 131072])
        ctx = chunk if rng.random() < 0.3 else _log_int(rng, max(chunk, 2048), max_ctx)
        return dict(kind=kind, B=rng.choice([1, 1, 2, 4]), chunk=chunk, ctx=ctx, max_ctx=max_ctx, H=32, HKV=8, D=128,
                    dtype=rng.choice(["bf16", "bf16", "fp16"]), layer=rng.choice(["dense", "sparse", "sparse"]), fp8=rng.random() < 0.35)
    if kind == "prefill":
        dtype = rng.choice(["bf16", "bf16", "fp16", "fp32"])
        if dtype == "fp32":
            TQ = _log_int(rng, 65, 4096)
            return dict(kind=kind, B=1, TQ=TQ, T=_log_int(rng, max(TQ, 1024), 8192), H=8, HKV=2, D=64, dtype=dtype, plan="short", stats=rng.random() < 0.5)
        plan = rng.choice(["long", "long", "gqa"])
        H, HKV, D = (64, 8, 128) if plan == "gqa" else rng.choice([(32, 8, 128), (32, 8, 128), (16, 4, 64), (16, 16, 128)])
        TQ = _log_int(rng, 65, 32768)
        return dict(kind=kind, B=rng.choice([1, 1, 2]), TQ=TQ, T=_log_int(rng, max(TQ, 4096), 131072), H=H, HKV=HKV, D=D, dtype=dtype, plan=plan,
                    stats=rng.random() < 0.5)
    shards = rng.choice([4, 8])
    return dict(kind=kind, B=1, T=shards * 64 * _log_int(rng, 512, 2048), shards=shards, page=64, H=32, HKV=8, D=128, dtype=rng.choice(["bf16", "fp16"]),
                plan="long", cached=rng.random() < 0.5)


# ---------------------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------------------
def _normal(g, shape, dtype):
    return torch.randn(shape, generator=g, device="cuda", dtype=dtype)


def _keys(g, tokens, HKV, D, dtype):
    k = _normal(g, (tokens, HKV, D), dtype)
    heavy = torch.randint(0, tokens, (max(1, tokens // 100),), generator=g, device="cuda").unique()
    k[heavy] = k[heavy] * 4
    return k


def _args(case, **kw):
    p = PLANS[case["plan"]]
    stages = [ScanStage(stage_block_size_q=p["bq"], stage_block_stride_q=s, stage_chunk_size=c, stage_k=k, stage_stride=1)
              for s, c, k in zip(p["strides"], p["chunks"], (None,) + p["keep"][:-1])]
    return HiPAttentionArgs(sink_token_size=p["sink"], sliding_window_size=p["window"], second_stage_k=p["keep"][-1], stages=stages,
                            block_sparse_block_size_q=p["bq"], **kw)


def _lengths(g, B, T, ragged):
    """Live tokens per sequence: all T, or spread over the upper half of it."""
    lens = torch.full((B,), T, dtype=torch.int32, device="cuda")
    if ragged:
        lens[1:] = torch.randint((T + 1) // 2, T + 1, (B - 1,), generator=g, device="cuda", dtype=torch.int32)
    return lens


def _server_config():
    return HiPAttentionConfig()      # the defaults: 256 / 32 / 8 chunks, rotary embedding inside the kernels


def _rope_tables(rows, D):
    inv = 1.0 / (5e5 ** (torch.arange(0, D, 2, device="cuda", dtype=torch.float64) / D))
    ang = torch.arange(rows, device="cuda", dtype=torch.float64)[:, None] * inv
    ang = torch.cat([ang, ang], -1)
    return ang.cos().float(), ang.sin().float()


def prepare(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    H, HKV, D, dt, kind = case["H"], case["HKV"], case["D"], DTYPES[case["dtype"]], case["kind"]
    s = {"kind": kind}
    if kind == "prefill":
        B, TQ, T = case["B"], case["TQ"], case["T"]
        s["k"] = _keys(g, B * T, HKV, D, dt).view(B, T, HKV, D)
        s["v"] = _normal(g, (B, T, HKV, D), dt)
        s["q"] = _normal(g, (B, TQ, H, D), dt).mul_(D ** -0.5)
        s["args"] = _args(case, require_cache_statistics=case["stats"])
    elif kind == "decode":
        B, T, P = case["B"], case["T"], case["page"]
        per_seq = -(-T // P)
        n_pages = B * per_seq + 17
        lens = _lengths(g, B, T, case["ragged"])
        table = torch.randperm(n_pages, generator=g, device="cuda")[:B * per_seq].view(B, per_seq).to(torch.int32)
        s["q"] = _normal(g, (B, 1, H, D), dt).mul_(D ** -0.5)
        s["args"] = _args(case, require_cache_statistics=False, k_cache=_keys(g, n_pages * P, HKV, D, dt).view(n_pages, P, HKV, D),
                          v_cache=_normal(g, (n_pages, P, HKV, D), dt), block_table=table, cache_seq_lens=lens,
                          position_ids=(lens.long() - 1).view(B, 1), extend_context_length=T)
        # between refreshes the mask of an earlier query is in hand
        s["cached"] = hip_attention_12(_normal(g, (B, 1, H, D), dt).mul_(D ** -0.5), None, None, s["args"])[1] if case["cached"] else None
    elif kind == "sharded":
        T, P, S = case["T"], case["page"], case["shards"]
        L = T // S
        n_pages = T // P + 17
        kc, vc = _keys(g, n_pages * P, HKV, D, dt).view(n_pages, P, HKV, D), _normal(g, (n_pages, P, HKV, D), dt)
        table = torch.randperm(n_pages, generator=g, device="cuda")[:T // P].view(1, T // P).to(torch.int32)
        s["shards"] = [(kc, vc, table[:, j * (L // P):(j + 1) * (L // P)].contiguous(), torch.full((1,), L, dtype=torch.int32, device="cuda"))
                       for j in range(S)]
        s["q"] = _normal(g, (1, 1, H, D), dt).mul_(D ** -0.5)
        s["args"] = _args(case, require_cache_statistics=False)
        s["how"] = dict(n_shards=S, shard_len=L, per_shard_k=512)
        s["cached"] = None
        if case["cached"]:
            s["cached"] = hip_attention_12_sequence_sharded(_normal(g, (1, 1, H, D), dt).mul_(D ** -0.5), s["shards"], s["args"], **s["how"])[1]
    else:       # an inference server: token-granular pools shared by the requests, tables as wide as the model's context
        B, ctx, max_ctx = case["B"], case["ctx"], case["max_ctx"]
        n_tok = case["chunk"] if kind == "server_prefill" else 1
        lens = _lengths(g, B, ctx, True) if kind == "server_decode" else torch.full((B,), ctx, dtype=torch.int32, device="cuda")
        total = B * ctx + 31
        kc, vc = _keys(g, total, HKV, D, dt), _normal(g, (total, HKV, D), dt)
        if case["fp8"]:
            kc, vc = kc.to(torch.float8_e5m2), vc.to(torch.float8_e5m2)
        slots = torch.randperm(total, generator=g, device="cuda")[:B * ctx].view(B, ctx).to(torch.int32)
        req_to_tokens = torch.zeros((B + 3, max_ctx), dtype=torch.int32, device="cuda")
        rows = torch.randperm(B + 3, generator=g, device="cuda")[:B]
        req_to_tokens[rows, :ctx] = slots
        positions = (lens.long()[:, None] - n_tok + torch.arange(n_tok, device="cuda")).reshape(-1)
        cos, sin = _rope_tables(max_ctx, D)
        config = _server_config()
        s["layer"] = SERVER_LAYERS[case["layer"]]
        s["call"] = dict(sm_scale=D ** -0.5, batch_size=B, k_cache=kc, v_cache=vc, offload_cache=None, positions=positions, seq_lens=lens,
                         req_to_tokens=req_to_tokens, req_pool_indices=rows, rope_cos=cos, rope_sin=sin, layer_id=s["layer"], logit_cap=0.0,
                         orig_context_len=max_ctx, max_context_len=max_ctx, is_prefill=kind == "server_prefill", hip_config=config,
                         is_decode=kind == "server_decode")
        s["q"] = _normal(g, (B * n_tok, H, D), dt)
        if kind == "server_decode":
            # stages: 0 = estimate from scratch, 1 / 2 = restart at that stage, 3 = the whole mask is reused
            s["B"], s["stages"] = B, case["stages"]
            s["pool"] = HiPMetadataCachePool(total, H, 6, max_ctx, "cuda", config)
            first = _normal(g, (B, H, D), dt)
            s["pool"].set_hip_metadata_cache(s["layer"], B, B, forward_paged_hip(first, cached_metadata=None, **s["call"])[1])
    return s


# ---------------------------------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------------------------------
def _results(context, md):
    out = {"context": context, "indices": md.indices, "ks": md.ks, "ks_count": md.ks_count, "ks_start_end": md.ks_start_end}
    for i, c in enumerate(md.stage_caches or []):
        out["stage%d" % i] = (c.indices_left, c.indices_right, c.out_scores)
    for name in ("mask_cache_statistics", "sa_cache_statistics"):
        st = getattr(md, name)
        if st is not None:
            out[name] = (st.access_counter, st.cache_miss_counter)
    return out


def run(state):
    kind = state["kind"]
    if kind == "prefill":
        return _results(*hip_attention_12(state["q"], state["k"], state["v"], state["args"]))
    if kind == "decode":
        return _results(*hip_attention_12(state["q"], None, None, state["args"], state["cached"]))
    if kind == "sharded":
        out, mds = hip_attention_12_sequence_sharded(state["q"], state["shards"], state["args"], cached=state["cached"], **state["how"])
        return {"context": out, "masks": [(m.indices, m.ks) for m in mds]}
    if kind == "server_prefill":
        return _results(*forward_paged_hip(state["q"], **state["call"]))
    B, layer, pool = state["B"], state["layer"], state["pool"]
    cached = pool.get_hip_metadata_cache(layer, B, B, state["stages"])
    context, md = forward_paged_hip(state["q"], cached_metadata=cached, **state["call"])
    pool.set_hip_metadata_cache(layer, B, B, md)
    out = _results(context, md)
    out["pool"] = {name: buf.buffer for name, buf in pool.cache[layer].items()}
    return out


# ---------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------------------------------
def _scan(chunks, keep, strides, bq, sink, window, T, n_q, last, start, HKV, G, D, eb):
    """Bytes of key rows and operations of the scan stages of one sequence whose ``n_q`` queries end at position ``last``:
    the rows of a chunk that the halving search can reach (all of it, or two per round and head, whichever is fewer), and
    every head's dot products with them.  Prefill reads each key once."""
    flops = rows = 0.0
    n0 = max(0, -(-(T - sink - window) // chunks[0]))
    for d in range(-(-n_q // bq)):
        horizon = last - n_q + 1 + d * bq - max(0, window - chunks[0])
        act = min(n0, max(0, (horizon - sink) // chunks[0] + 1)) if horizon >= sink else 0
        n = n0
        for i, c in enumerate(chunks):
            per_head = max(2, 2 * (int(math.log2(c)) + 1) - 3)
            pooled = max(1, min(bq, n_q - d * bq) // strides[i]) if n_q > 1 else 1
            if i >= start:
                flops += act * per_head * HKV * G * pooled * 2.0 * D
                rows += act * min(c, per_head * G) * HKV
            if i + 1 < len(chunks):
                k = min(keep[i] // c, n)
                act, n = min(act, k) * (c // chunks[i + 1]), k * (c // chunks[i + 1])
    if n_q > 1:
        rows = min(rows, float(last + 1) * HKV)
    return rows * D * eb, flops


def work(case):
    H, HKV, D, kind = case["H"], case["HKV"], case["D"], case["kind"]
    G, B = H // HKV, case["B"]
    eb = 4 if case["dtype"] == "fp32" else 2
    kv_eb = 1 if case.get("fp8") else eb
    p = dict(PLANS[case.get("plan", "long")])
    start, repeat = 0, 1
    if kind == "prefill":
        T, n_q, last = case["T"], case["TQ"], case["T"] - 1
    elif kind == "decode":
        T, n_q, last = case["T"], 1, case["T"] * (0.75 if case["ragged"] and B > 1 else 1.0) - 1
        start = len(p["chunks"]) if case["cached"] else 0
    elif kind == "sharded":
        T, n_q, last = case["T"] // case["shards"], 1, case["T"] // case["shards"] - 1
        start, repeat = (len(p["chunks"]) if case["cached"] else 0), case["shards"]
        p["keep"] = p["keep"][:-1] + (512,)
        p["sink"] = p["window"] = 0
    else:
        T, n_q, last = case["max_ctx"], case.get("chunk", 1), case["ctx"] - 1
        if kind == "server_decode":
            last, start = case["ctx"] * (0.75 if B > 1 else 1.0) - 1, case["stages"]
        if case["layer"] == "dense":
            p["keep"] = p["keep"][:-1] + (4096,)
    sb, sf = _scan(p["chunks"], p["keep"], p["strides"], p["bq"], p["sink"], p["window"], T, n_q, int(last), start, HKV, G, D, kv_eb)
    most = p["keep"][-1] + p["sink"] + p["window"]
    lo = int(last) - n_q + 1
    # a query at position x attends min(x + 1, most) keys
    ramp = max(0, min(most, int(last) + 1) - lo)
    attended = ramp * (lo + 1 + min(most, int(last) + 1)) / 2.0 + (n_q - ramp) * most if ramp else n_q * float(most)
    af = 4.0 * D * H * attended
    if n_q == 1:
        ab, sb = 2.0 * attended * HKV * D * kv_eb, sb
    else:
        ab, sb = 2.0 * (last + 1) * HKV * D * kv_eb, 0.0      # keys and values of the prompt, once
    qo = 2.0 * n_q * H * D * eb
    mask = H * -(-n_q // p["bq"]) * (p["keep"][-1] // p["chunks"][-1]) * 8.0
    return {"bytes": B * (repeat * (sb + ab + mask) + qo), "flops": B * repeat * (sf + af)}


def tolerance(case):
    # the mask is whole numbers and stays the same; the context is rounded to the element type after a softmax whose
    # weights are rounded to it too
    return {"rel": {"fp32": 1e-5, "fp16": 2e-3, "bf16": 1e-2}[case["dtype"]]}
