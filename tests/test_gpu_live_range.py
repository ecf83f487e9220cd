"""Key buffers and rope tables longer than the sequence: only what a call can reach is prepared.  The rest is poisoned here, and
masks and outputs equal the strict scan's on the live part; fp32 tables give what tables converted beforehand give."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("backend", [None, "relative", "streaming"])
@pytest.mark.parametrize("tq", [1, 70, 300])
@pytest.mark.parametrize("live", [701, 3000])
def test_only_the_live_range_matters(live, tq, backend, monkeypatch):
    import bench
    from cases import rope_tables
    from hip_attention_b200 import hip_attention_impl, read_status
    w = dict(bench.WORKLOADS["prefill_128k"], B=2, TQ=tq, T=6000, H=8, HKV=2, keep=[2048, 1024, 512], sink=64, sw=320)
    q, k, v = bench.make_qkv(w, "cuda")
    # batch element 1 is 130 tokens shorter
    pos = torch.stack([torch.arange(tq) + live - tq, torch.arange(tq) + live - 130 - tq]).cuda()
    # beyond the last query block's rows and its chunk nothing may be read
    k[:, live + 512:], v[:, live + 512:] = float("nan"), float("nan")
    outs = {}
    for name, mode, dtype in (("auto", "auto", torch.float32), ("strict", "strict", torch.float32), ("converted", "auto", torch.bfloat16)):
        kw = {}
        if backend:
            cos, sin = (torch.from_numpy(t).cuda().to(dtype) for t in rope_tables(9000, 128, w["theta"]))
            if dtype == torch.float32:   # rows that no call here reaches
                cos[live + 300:], sin[live + 300:] = float("nan"), float("nan")
            kw = dict(using_extend=True, need_apply_rope=True, rope_cos=cos, rope_sin=sin, scan_extend_backend=backend)
        monkeypatch.setenv("HIPATTN_SCAN_MODE", mode)
        read_status("cuda")
        outs[name] = hip_attention_impl(q, k, v, bench.make_args(w, position_ids=pos, **kw))
        assert read_status("cuda") == 0
    for name in ("strict", "converted"):
        assert torch.equal(outs["auto"][1].indices, outs[name][1].indices) and torch.equal(outs["auto"][1].ks, outs[name][1].ks)
        assert torch.equal(outs["auto"][0], outs[name][0])
    assert torch.isfinite(outs["auto"][0].float()).all()


def test_split_prefill_equals_two_calls():
    """A server's prefill chunk (parts share prepared keys and one output) against two operator calls of its own."""
    from cases import rope_tables
    from hip_attention_b200 import HiPAttentionConfig, forward_paged_hip, hip_attention_12
    import hip_attention_b200.serving as S
    g = torch.Generator(device="cuda").manual_seed(3)
    B, n, ctx, H, HKV, D, width = 2, 200, 3001, 8, 2, 128, 8192
    kc, vc = (torch.randn((B * ctx + 5, HKV, D), generator=g, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    q = torch.randn((B * n, H, D), generator=g, device="cuda", dtype=torch.bfloat16)
    req = torch.zeros((4, width), dtype=torch.int32, device="cuda")
    rows = torch.tensor([2, 0], device="cuda")
    req[rows, :ctx] = torch.randperm(B * ctx, generator=g, device="cuda").view(B, ctx).to(torch.int32)
    lens = torch.tensor([ctx, ctx - 7], dtype=torch.int32, device="cuda")
    pos = (lens.long()[:, None] - n + torch.arange(n, device="cuda")).reshape(-1)
    cos, sin = (torch.from_numpy(t).cuda() for t in rope_tables(width, D, 5e5))
    calls = []

    def record(q_, k_, v_, args, cached=None, **kw):
        calls.append((q_, args, kw))
        return S_impl(q_, k_, v_, args, cached, **kw)
    S_impl, S.hip_attention_impl = S.hip_attention_impl, record
    try:
        for layer in (0, 5):
            calls.clear()
            out, md = forward_paged_hip(q, D ** -0.5, B, kc, vc, None, pos, lens, req, rows, cos, sin, layer, 0.0, width, width, True, HiPAttentionConfig())
            assert len(calls) == 2 and calls[0][2]["shared"] is calls[1][2]["shared"]
            ref = [hip_attention_12(q_, None, None, a) for q_, a, _ in calls]
            assert torch.equal(out, torch.cat([r[0] for r in ref], 1))
            assert torch.equal(md.indices, ref[1][1].indices) and torch.equal(md.ks, ref[1][1].ks)
    finally:
        S.hip_attention_impl = S_impl


@pytest.mark.parametrize("backend", ["relative", "streaming"])
def test_both_windows_of_a_split_chunk_reach_converted_table_rows(backend):
    """A layer window below the 777 of the last queries, sink 0 and a short prompt: the last queries' scan rotates to rows that
    the first part does not reach.  Memory the tables are made in is poisoned; masks and the keys the scans load equal those of
    two calls of their own."""
    from cases import rope_tables
    from hip_attention_b200 import HiPAttentionConfig, forward_paged_hip, hip_attention_12
    from hip_attention_b200.serving import HiPAttentionPerLayerConfig
    import hip_attention_b200.serving as S
    g = torch.Generator(device="cuda").manual_seed(4)
    n, H, HKV, D, width = 200, 8, 2, 128, 2048
    kc, vc = (torch.randn((n + 5, HKV, D), generator=g, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    q = torch.randn((n, H, D), generator=g, device="cuda", dtype=torch.bfloat16)
    req = torch.zeros((2, width), dtype=torch.int32, device="cuda")
    req[1, :n] = torch.randperm(n, generator=g, device="cuda").to(torch.int32)
    cos, sin = (torch.from_numpy(t).cuda() for t in rope_tables(16384, D, 5e5))
    layer = HiPAttentionPerLayerConfig(second_stage_k=64, sliding_window_size=512, sink_token_size=0, scan_extend_backend=backend)
    cfg = HiPAttentionConfig(layers=[layer, layer], prefill_layers=[layer, layer])
    calls = []

    def record(q_, k_, v_, args, cached=None, **kw):
        calls.append((q_, args))
        return impl(q_, k_, v_, args, cached, **kw)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    poison = torch.full((64 << 20,), 0x7fc07fc0, dtype=torch.int32, device="cuda")   # NaN in either 16-bit type
    del poison
    impl, S.hip_attention_impl = S.hip_attention_impl, record
    try:
        out, md = forward_paged_hip(q, D ** -0.5, 1, kc, vc, None, torch.arange(n, device="cuda"), torch.tensor([n], dtype=torch.int32, device="cuda"),
                                    req, torch.tensor([1], device="cuda"), cos, sin, 5, 0.0, width, width, True, cfg)
    finally:
        S.hip_attention_impl = impl
    ref = [hip_attention_12(q_, None, None, a) for q_, a in calls]
    assert torch.equal(out, torch.cat([r[0] for r in ref], 1))
    assert torch.equal(md.indices, ref[1][1].indices) and torch.equal(md.ks, ref[1][1].ks)
    assert torch.equal(md.mask_cache_statistics.access_counter, ref[1][1].mask_cache_statistics.access_counter)


def test_split_prefill_takes_a_query_of_any_strides():
    """Queries stored head-major, or as columns of a fused projection, against a contiguous copy."""
    from hip_attention_b200 import HiPAttentionConfig, forward_paged_hip
    g = torch.Generator(device="cuda").manual_seed(6)
    n, ctx, H, HKV, D, width = 150, 2000, 8, 2, 128, 4096
    kc, vc = (torch.randn((ctx, HKV, D), generator=g, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    req = torch.randperm(ctx, generator=g, device="cuda").to(torch.int32).view(1, ctx)
    req = torch.nn.functional.pad(req, (0, width - ctx))
    cfg = HiPAttentionConfig(json_or_path='{"using_extend": false}')
    head_major = torch.randn((H, n, D), generator=g, device="cuda", dtype=torch.bfloat16).permute(1, 0, 2)
    fused = torch.randn((n, H + 2 * HKV, D), generator=g, device="cuda", dtype=torch.bfloat16)[:, :H]

    def call(q):
        return forward_paged_hip(q, D ** -0.5, 1, kc, vc, None, torch.arange(ctx - n, ctx, device="cuda"), torch.tensor([ctx], dtype=torch.int32, device="cuda"),
                                 req, torch.tensor([0], device="cuda"), None, None, 5, 0.0, width, width, True, cfg)
    for q in (head_major, fused):
        assert not q.is_contiguous()
        out, md = call(q)
        ref, ref_md = call(q.contiguous())
        assert out.is_contiguous() and torch.equal(out, ref) and torch.equal(md.indices, ref_md.indices)
