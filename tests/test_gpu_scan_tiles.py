"""Prefill scans that score whole tiles of keys: masks, later stages' lists and access counters equal the strict kernel's, where every
bound is settled at once and where strict scores are needed."""
import re

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def tiles(monkeypatch, request):
    """The whole-tile kernels wherever they can be had: the calls here are smaller than what they are chosen for."""
    if "by_rule" not in request.keywords:
        monkeypatch.setenv("HIPATTN_SCAN_KERNEL", "tiles")


SHAPES = {
    "heads4": dict(T=9001, TQ=2300),                                                   # 4 heads x 64 rows: a full accumulator
    "heads4_d64": dict(T=6007, TQ=1517, D=64, dtype="fp16"),
    "heads8_rows16": dict(T=5003, TQ=2100, H=8, HKV=1, strides=[4, 4, 4]),             # half of an accumulator
    "heads8_rows128": dict(T=9001, TQ=2200, H=16, bq=128),                             # two passes, two CTAs a unit
    "heads20": dict(T=5003, TQ=1030, H=20, HKV=1),                                     # a CTA with part of its heads
    "heads3": dict(T=5003, TQ=1030, H=6),
    "heads2_rows128": dict(T=7001, TQ=2200, H=4, bq=128, B=2),
    "heads2": dict(T=3000, TQ=3000, H=4, sw=256, sink=0),
    "heads1": dict(T=4500, TQ=4500, H=2, sw=256, sink=0, keep=[8192, 1024, 512]),
    "chunks512": dict(T=9001, TQ=2300, chunks=[512, 32, 8], keep=[8192, 1024, 512]),   # two tiles of keys a chunk
    "odd_sink": dict(T=5003, TQ=1410, sink=101),                                       # narrowed bounds per head
    "short_window": dict(T=4099, TQ=1100, sink=64, sw=128),                            # chunks that end beyond the keys
    "few_kept": dict(T=2049, TQ=2049, keep=[1536, 512, 256], sw=512, sink=0),
}


def problem(shape, keys, rope):
    import bench
    from cases import rope_tables
    w = dict(bench.WORKLOADS["prefill_128k"], H=8, HKV=2, keep=[4096, 1024, 512])
    w.update(shape if isinstance(shape, dict) else SHAPES[shape])
    q, k, v = bench.make_qkv(w, "cuda")
    g = torch.Generator(device="cuda").manual_seed(5)
    if keys == "close":      # neighbours that are equal or one unit in the last place apart
        n = w["T"] // 2
        k[:, 1:2 * n:2] = k[:, 0:2 * n:2]
        k.view(torch.int16)[:, 1::4, :, 3] ^= 1
    elif keys == "not_finite":
        q[:, :, 0] = 0
        for value in (float("inf"), float("-inf"), float("nan")):
            k[:, torch.randint(0, w["T"], (w["T"] // 100,), generator=g, device="cuda"), :, 5] = value
        t = torch.randint(0, w["T"], (w["T"] // 50,), generator=g, device="cuda")
        k[:, t] = torch.where(k[:, t] > 0, 5e4, -5e4).to(k.dtype)
    kw = {}
    if rope:
        cos, sin = rope_tables(w["T"] + 8, w["D"], w["theta"])
        kw = dict(using_extend=True, need_apply_rope=True, rope_cos=torch.from_numpy(cos).cuda(), rope_sin=torch.from_numpy(sin).cuda(),
                  scan_extend_backend=rope)
    args = bench.make_args(w, **kw)
    args.require_cache_statistics = True
    return (q, k, v), args


def launches(call):
    """Names of the scan kernels that a call launches, in order."""
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        call()
        torch.cuda.synchronize()
    names = [re.search(r"scan_(\w+)_kernel", e.name) for e in prof.events()]
    return [n.group(1) for n in names if n and n.group(1) != "prepare_keys"]


def expected(args, H, HKV):
    """What this file's calls launch: whole tiles in the second and third stage as far as their shapes allow it."""
    G, rows = H // HKV, [s.stage_block_size_q // s.stage_block_stride_q for s in args.stages]
    if args.using_extend:
        return ["stage_tcgen05"] * 3
    return ["stage_tcgen05", "key_tiles" if rows[1] == 16 and G in (1, 2, 4, 8, 16) else "stage_tcgen05",
            "query_tiles" if G >= 2 and G * rows[2] >= 128 else "stage_tcgen05"]


@pytest.mark.parametrize("rope", [None, "relative"])
@pytest.mark.parametrize("keys", ["random", "close", "not_finite"])
@pytest.mark.parametrize("shape", list(SHAPES))
def test_masks_equal_strict(shape, keys, rope, monkeypatch):
    from hip_attention_b200 import hip_attention_impl
    qkv, args = problem(shape, keys, rope)
    md = {}
    for mode in ("auto", "strict"):
        monkeypatch.setenv("HIPATTN_SCAN_MODE", mode)
        if mode == "auto" and keys == "random":
            assert launches(lambda: hip_attention_impl(*qkv, args)) == expected(args, qkv[0].shape[2], qkv[1].shape[2])
        md[mode] = hip_attention_impl(*qkv, args)[1]
    a, b = md["auto"], md["strict"]
    for i, (x, y) in enumerate(zip(a.stage_caches[1:], b.stage_caches[1:])):
        assert torch.equal(x.indices_left, y.indices_left) and torch.equal(x.indices_right, y.indices_right), f"stage {i + 1}"
    assert torch.equal(a.indices, b.indices) and torch.equal(a.ks, b.ks)
    assert torch.equal(a.mask_cache_statistics.access_counter, b.mask_cache_statistics.access_counter)


@pytest.mark.parametrize("keys", ["random", "close", "not_finite"])
@pytest.mark.parametrize("shape", ["heads4", "heads4_d64", "heads8_rows16", "heads8_rows128", "heads20", "heads3", "heads1", "odd_sink", "short_window",
                                   "chunks512"])
def test_bounds_and_scores_per_head_equal_strict(shape, keys, monkeypatch):
    """Check mode scores every key by both definitions, in both kernels: none may be taken for certain that is not, and the error
    radius is twice what is needed or more."""
    from hip_attention_b200 import hip_attention_impl
    qkv, args = problem(shape, keys, None)
    got = {}
    stats = torch.zeros(4, dtype=torch.int64, device="cuda")
    for mode in ("auto", "strict", "check"):
        monkeypatch.setenv("HIPATTN_SCAN_MODE", mode)
        dbg = {"scan_stats": stats} if mode == "check" else {}
        names = launches(lambda: hip_attention_impl(*qkv, args, debug=dbg))
        assert mode == "strict" or names == expected(args, qkv[0].shape[2], qkv[1].shape[2])
        got[mode] = dbg["stages"]
    for mode in ("auto", "check"):
        for i, (a, b) in enumerate(zip(got[mode], got["strict"])):
            for key in ("left", "right", "score", "score_max"):
                assert torch.equal(a[key], b[key]), f"{mode} stage {i} {key}"
    keys_seen, uncertain, wrong, ratio = stats.tolist()
    assert 0 < uncertain < keys_seen and wrong == 0, "a score taken without the strict definition is wrong"
    if keys == "random":
        assert torch.tensor([ratio & 0xffffffff], dtype=torch.int64).to(torch.int32).view(torch.float32).item() < 0.5


@pytest.mark.parametrize("rope", [None, "relative"])
@pytest.mark.parametrize("change", ["longer", "shorter", "moved", "shuffled"])
def test_restart_from_lists_of_a_callers_own(change, rope, monkeypatch):
    """Chunks that are longer than the stage's size, empty, off the grid, in no order: each restarted stage as in strict mode."""
    from hip_attention_b200 import HiPAttentionOutputMetadata, hip_attention_impl
    from hip_attention_b200.metadata import HiPAttentionStageInputCache
    qkv, args = problem("heads4", "random", rope)
    md = hip_attention_impl(*qkv, args)[1]
    caches = list(md.stage_caches)
    for stage in (1, 2):
        c = caches[stage]
        l, r = c.indices_left.clone(), c.indices_right.clone()
        if change == "longer":
            r[..., ::3] += 13
        elif change == "shorter":
            r[..., ::2] = torch.maximum(l[..., ::2], r[..., ::2] - 5)
            r[..., ::7] = l[..., ::7]
        elif change == "moved":
            l, r = (l + 3).clamp(max=8990), (r + 3).clamp(max=8999)
        else:
            p = torch.randperm(l.shape[-1], device="cuda")
            l, r = l[..., p], r[..., p]
        got = {}
        for mode in ("auto", "strict"):
            monkeypatch.setenv("HIPATTN_SCAN_MODE", mode)
            # (a call completes the list of stage inputs that it is given)
            part = HiPAttentionOutputMetadata(None, None, None, None, None, None, caches[:stage] + [HiPAttentionStageInputCache(l, r, c.out_scores)])
            got[mode] = hip_attention_impl(*qkv, args, cached_metadata=part)[1]
        a, b = got["auto"], got["strict"]
        assert torch.equal(a.indices, b.indices) and torch.equal(a.ks, b.ks), f"stage {stage}"
        assert torch.equal(a.mask_cache_statistics.access_counter, b.mask_cache_statistics.access_counter), f"stage {stage}"


@pytest.mark.parametrize("form", ["dense", "dense_d64", "paged", "q_by_heads", "positions_falling", "heads16", "heads16_paged"])
def test_sequences_of_their_own(form, monkeypatch):
    """Two sequences whose queries end at different tokens, nothing but NaN behind the last chunk that they reach: whole tiles, rounds
    and the strict kernel give the same lists, masks and counters, through a page table too."""
    import bench
    from hip_attention_b200 import hip_attention_impl, read_status
    B, T, TQ, live, page = 2, 8200, 3200, 7003, 16
    w = dict(bench.WORKLOADS["prefill_128k"], B=B, TQ=TQ, T=T, H=8, HKV=2, keep=[4096, 1024, 512], sink=64, sw=320)
    if form.startswith("heads16"):
        w["H"] = 32
    if form == "dense_d64":
        w.update(D=64, dtype="fp16")
    q, k, v = bench.make_qkv(w, "cuda")
    k[:, live + 512:], v[:, live + 512:] = float("nan"), float("nan")
    pos = (torch.arange(TQ) + torch.tensor([[live - TQ], [live - 1300 - TQ]])).cuda()
    if form == "positions_falling":
        pos = pos.flip(1)
    if form == "q_by_heads":
        q = q.permute(0, 2, 1, 3).contiguous().permute(0, 2, 1, 3)
    args = bench.make_args(w, position_ids=pos)
    args.require_cache_statistics = True
    if form.endswith("paged"):
        g = torch.Generator(device="cuda").manual_seed(9)
        n = -(-T // page)
        table = torch.randperm(B * n + 3, generator=g, device="cuda")[:B * n].view(B, n).to(torch.int32)
        pools = []
        for x in (k, v):
            x = torch.nn.functional.pad(x, (0, 0, 0, 0, 0, n * page - T)).view(B * n, page, w["HKV"], -1)
            pool = torch.full((B * n + 3, *x.shape[1:]), float("nan"), dtype=x.dtype, device="cuda")
            pool[table.view(-1).long()] = x
            pools.append(pool)
        args.k_cache, args.v_cache = pools
        args.block_table, args.cache_seq_lens, args.extend_context_length = table, torch.full((B,), T, dtype=torch.int32, device="cuda"), T
        args.update_flags()
        k = v = None
    md = {}
    for name in ("tiles", "rounds", "strict"):
        monkeypatch.setenv("HIPATTN_SCAN_MODE", "strict" if name == "strict" else "auto")
        monkeypatch.setenv("HIPATTN_SCAN_KERNEL", name)
        read_status("cuda")
        names = launches(lambda: md.update({name: hip_attention_impl(q, k, v, args)[1]}))
        assert read_status("cuda") == 0
        assert name == "strict" or names == (["stage_tcgen05", "key_tiles", "query_tiles"] if name == "tiles" else ["stage_tcgen05"] * 3)
    for name in ("tiles", "rounds"):
        a, b = md[name], md["strict"]
        for i, (x, y) in enumerate(zip(a.stage_caches[1:], b.stage_caches[1:])):
            assert torch.equal(x.indices_left, y.indices_left), f"{name} stage {i + 1}"
        assert torch.equal(a.indices, b.indices) and torch.equal(a.ks, b.ks), name
        assert torch.equal(a.mask_cache_statistics.access_counter, b.mask_cache_statistics.access_counter), name
    assert int(md["tiles"].mask_cache_statistics.access_counter.sum()) > 0


def test_waits_that_run_out_are_reported_and_leave_nothing(monkeypatch):
    """Every wait of both kernels that is not over at once counts as one that ran out: the call ends, says so, and the next one, which
    needs all of the tensor memory, is right."""
    from hip_attention_b200 import _lib, hip_attention_impl, read_status
    qkv, args = problem("heads4", "random", None)
    read_status("cuda")
    want = hip_attention_impl(*qkv, args)[1]
    assert read_status("cuda") == 0
    for _ in range(3):
        monkeypatch.setenv("HIPATTN_SCAN_WAIT", "none")
        hip_attention_impl(*qkv, args)
        torch.cuda.synchronize()
        assert read_status("cuda") & _lib.STATUS_TIMEOUT
        monkeypatch.delenv("HIPATTN_SCAN_WAIT")
        md = hip_attention_impl(*qkv, args)[1]
        assert read_status("cuda") == 0
        assert torch.equal(md.indices, want.indices) and torch.equal(md.ks, want.ks)


@pytest.mark.parametrize("shape", [dict(T=33001, TQ=33001, H=64, HKV=8), dict(T=9001, TQ=9001, H=64, HKV=8, B=5)], ids=["blocks", "sequences"])
def test_key_tiles_in_several_launches(shape, monkeypatch):
    """More query blocks, or sequences, than one launch has scratch for (258 KB a block here, 128 MB in all: 516 blocks of one sequence,
    141 of five)."""
    from hip_attention_b200 import hip_attention_impl
    qkv, args = problem(shape, "random", None)
    md = {}
    for mode in ("auto", "strict"):
        monkeypatch.setenv("HIPATTN_SCAN_MODE", mode)
        if mode == "auto":
            assert launches(lambda: hip_attention_impl(*qkv, args)).count("key_tiles") == 2
        md[mode] = hip_attention_impl(*qkv, args)[1]
    a, b = md["auto"], md["strict"]
    assert torch.equal(a.stage_caches[2].indices_left, b.stage_caches[2].indices_left)
    assert torch.equal(a.indices, b.indices) and torch.equal(a.ks, b.ks)
    assert torch.equal(a.mask_cache_statistics.access_counter, b.mask_cache_statistics.access_counter)


def test_without_memory_for_the_scratch():
    """The rounds need none: a call that finds no room for the key tiles' scratch (68 MB here) goes by them."""
    from hip_attention_b200 import hip_attention_impl
    qkv, args = problem(dict(T=16500, TQ=16500, H=64, HKV=8), "random", None)
    want = hip_attention_impl(*qkv, args)[1]
    total = torch.cuda.mem_get_info()[1]
    calls, held = [], []

    def after_stage(score):    # (called after each scan stage; the second one asks for scratch)
        calls.append(1)
        if len(calls) == 1:
            torch.cuda.empty_cache()
            torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (16 << 20)) / total)
            with pytest.raises(torch.OutOfMemoryError):
                while True:
                    held.append(torch.empty(32 << 20, dtype=torch.uint8, device="cuda"))
        else:
            held.clear()
            torch.cuda.set_per_process_memory_fraction(1.0)

    try:
        md = hip_attention_impl(*qkv, args, score_reduce=after_stage)[1]
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert len(calls) == 3
    assert torch.equal(md.indices, want.indices) and torch.equal(md.ks, want.ks)


def test_under_capture():
    """Lists, pooled queries and scratch are made anew at every replay."""
    from hip_attention_b200 import hip_attention_impl, read_status
    (q, k, v), args = problem("heads4", "random", None)
    args.position_ids = (torch.arange(q.shape[1], device="cuda") + k.shape[1] - q.shape[1])[None]
    other = torch.randn_like(q) * 128 ** -0.5
    want = hip_attention_impl(other, k, v, args)
    assert not torch.equal(want[1].indices, hip_attention_impl(q, k, v, args)[1].indices)
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        out, md = hip_attention_impl(q, k, v, args)
    q.copy_(other)
    for _ in range(2):
        out.zero_(), md.indices.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want[0]) and torch.equal(md.indices, want[1].indices) and torch.equal(md.ks, want[1].ks)
        assert torch.equal(md.mask_cache_statistics.access_counter, want[1].mask_cache_statistics.access_counter)
    assert read_status("cuda") == 0


# heads, KV heads, query rows of a block, pooling strides, queries, tokens, kept -> kernels of the second and third stage
RULE = [
    # (few CTAs, one with a list of all blocks: 2.4 to 2.5 times the rounds' time by key tiles)
    (32, 2, 64, (4, 4, 1), 3000, 3000, (32768, 8192, 2048), ("stage_tcgen05", "query_tiles")),
    (16, 1, 64, (4, 4, 1), 4202, 7692, (32768, 8192, 2048), ("stage_tcgen05", "query_tiles")),
    # (blocks listed, but few active)
    (32, 8, 64, (4, 4, 1), 2500, 2500, (32768, 8192, 2048), ("stage_tcgen05", "query_tiles")),
    (64, 8, 64, (4, 4, 1), 2048, 2048, (32768, 8192, 2048), ("stage_tcgen05", "query_tiles")),
    (32, 8, 64, (4, 4, 1), 4096, 4096, (32768, 8192, 2048), ("key_tiles", "query_tiles")),
    (16, 4, 64, (4, 4, 1), 2999, 20011, (32768, 8192, 2048), ("key_tiles", "query_tiles")),
    (64, 8, 64, (4, 4, 1), 1100, 8192, (32768, 8192, 2048), ("key_tiles", "query_tiles")),
    # (short lists: 2.4, 1.8 and 1.5 times the rounds' time by query tiles)
    (64, 8, 64, (4, 4, 2), 357, 16723, (4096, 512, 256), ("stage_tcgen05", "stage_tcgen05")),
    (8, 1, 64, (4, 4, 1), 2652, 73875, (4096, 512, 256), ("stage_tcgen05", "stage_tcgen05")),
    (32, 8, 64, (4, 4, 2), 16384, 32938, (4096, 512, 256), ("key_tiles", "stage_tcgen05")),
    (64, 8, 128, (4, 4, 1), 2000, 32768, (65536, 16384, 4096), ("stage_tcgen05", "query_tiles")),
]


@pytest.mark.by_rule
@pytest.mark.parametrize("H,HKV,bq,strides,TQ,T,keep,want", RULE)
def test_tiles_where_they_are_faster(H, HKV, bq, strides, TQ, T, keep, want, monkeypatch):
    """Kernels that the rules choose, on calls whose times with either are far apart."""
    from hip_attention_b200 import hip_attention_impl
    import bench
    g = torch.Generator(device="cuda").manual_seed(1)
    q = torch.randn((1, TQ, H, 128), generator=g, device="cuda", dtype=torch.bfloat16) * 128 ** -0.5
    k = torch.randn((1, T, HKV, 128), generator=g, device="cuda", dtype=torch.bfloat16)
    args = bench.make_args(dict(chunks=(256, 32, 8), bq=bq, strides=strides, keep=keep, sink=256, sw=1024))
    assert tuple(launches(lambda: hip_attention_impl(q, k, k, args))[1:]) == want
    monkeypatch.setenv("HIPATTN_SCAN_KERNEL", "rounds")
    assert launches(lambda: hip_attention_impl(q, k, k, args)) == ["stage_tcgen05"] * 3
