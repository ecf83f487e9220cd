"""Decode scan of small chunks on the tensor cores: per-head bounds and scores of every stage equal the strict kernels', and
in check mode no score taken without the strict definition is wrong."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [
    dict(B=2, H=8, HKV=1, D=128, T=8192),                                  # eight heads per pass
    dict(B=1, H=12, HKV=1, D=128, T=4999, keep=[4096, 1024, 512]),         # two passes, the second part-filled; ragged last chunk
    dict(B=3, H=6, HKV=2, D=64, T=3001, keep=[2048, 1024, 512]),           # three heads per KV head
    dict(B=2, H=2, HKV=2, D=128, T=2600, chunks=[64, 4], keep=[1024, 512], strides=[4, 1]),   # chunk 4, one head
]


@pytest.mark.parametrize("rope", [None, "relative", "streaming"])
@pytest.mark.parametrize("kv", ["bf16", "fp16", "fp8"])
@pytest.mark.parametrize("shape", SHAPES)
def test_decode_chunk_scan_is_exact(shape, kv, rope, monkeypatch):
    import bench
    from cases import rope_tables
    from hip_attention_b200 import hip_attention_impl, read_status
    w = dict(bench.WORKLOADS["decode_128k"], kind="prefill", keep=[4096, 2048, 1024], dtype="fp16" if kv == "fp16" else "bf16")
    w.update(shape)
    q, k, v = bench.make_qkv(w, "cuda")
    if kv == "fp8":
        k, v = k.to(torch.float8_e5m2), v.to(torch.float8_e5m2)
    kw = {}
    if rope:
        cos, sin = rope_tables(w["T"] + 8, w["D"], w["theta"])
        kw = dict(using_extend=True, need_apply_rope=True, rope_cos=torch.from_numpy(cos).cuda(), rope_sin=torch.from_numpy(sin).cuda(),
                  scan_extend_backend=rope)
    read_status("cuda")
    got, mds = {}, {}
    stats = torch.zeros(4, dtype=torch.int64, device="cuda")
    for mode in ("auto", "strict", "check"):
        monkeypatch.setenv("HIPATTN_SCAN_MODE", mode)
        dbg = {"scan_stats": stats} if mode == "check" else {}
        _, mds[mode] = hip_attention_impl(q, k, v, bench.make_args(w, **kw), debug=dbg)
        got[mode] = dbg["stages"]
    assert read_status("cuda") == 0
    for mode in ("auto", "check"):
        for i, (a, b) in enumerate(zip(got[mode], got["strict"])):
            for key in ("left", "right", "score", "score_max"):
                assert torch.equal(a[key], b[key]), f"{mode} stage {i} {key}"
        assert torch.equal(mds[mode].indices, mds["strict"].indices) and torch.equal(mds[mode].ks, mds["strict"].ks)
    keys, fallbacks, wrong, ratio = stats.cpu().tolist()
    ratio = torch.tensor([ratio & 0xffffffff], dtype=torch.int64).to(torch.int32).view(torch.float32).item()
    assert keys > 0 and wrong == 0 and fallbacks < 0.25 * keys
    assert ratio < 0.5, f"deviation reached {ratio:.3f} of the assumed radius"
    print(f"{shape} {kv} {rope}: keys {keys} fallbacks {fallbacks} ratio {ratio:.3f}")


@pytest.mark.parametrize("keys", ["close", "not_finite"])
@pytest.mark.parametrize("rope", [None, "relative", "streaming"])
@pytest.mark.parametrize("kv", ["bf16", "fp16", "fp8"])
@pytest.mark.parametrize("shape", SHAPES + [dict(B=2, H=8, HKV=2, D=128, T=3333, keep=[2048, 1024, 512])])
def test_search_on_bounds_equals_strict_scores(shape, kv, rope, keys, monkeypatch):
    """The call as users make it, without per-head outputs, which would have every score computed strictly before the search:
    neighbouring keys that are equal or one unit in the last place apart leave the bounds open; infinities, NaN, keys whose
    magnitudes overflow 16 bits and a query head of zeros give bounds that are not numbers."""
    import bench
    from cases import rope_tables
    from hip_attention_b200 import hip_attention_impl, read_status
    w = dict(bench.WORKLOADS["decode_128k"], kind="prefill", keep=[4096, 2048, 1024], dtype="fp16" if kv == "fp16" else "bf16")
    w.update(shape)
    q, k, v = bench.make_qkv(w, "cuda")
    g = torch.Generator(device="cuda").manual_seed(5)
    if keys == "close":
        n = w["T"] // 2
        k[:, 1:2 * n:2] = k[:, 0:2 * n:2]
        bits = k.view(torch.int16)
        bits[:, 1::4, :, 3] ^= 1
    else:
        q[:, :, 0] = 0
        for value in (float("inf"), float("-inf"), float("nan")):
            t = torch.randint(0, w["T"], (w["T"] // 100,), generator=g, device="cuda")
            k[:, t, :, 5] = value
        t = torch.randint(0, w["T"], (w["T"] // 50,), generator=g, device="cuda")
        k[:, t] = torch.where(k[:, t] > 0, 5e4, -5e4).to(k.dtype)
    if kv == "fp8":
        k, v = k.to(torch.float8_e5m2), v.to(torch.float8_e5m2)
    kw = {}
    if rope:
        cos, sin = rope_tables(w["T"] + 8, w["D"], w["theta"])
        kw = dict(using_extend=True, need_apply_rope=True, rope_cos=torch.from_numpy(cos).cuda(), rope_sin=torch.from_numpy(sin).cuda(),
                  scan_extend_backend=rope)
    read_status("cuda")
    md = {}
    for mode in ("auto", "strict"):
        monkeypatch.setenv("HIPATTN_SCAN_MODE", mode)
        args = bench.make_args(w, **kw)
        args.require_cache_statistics = True
        md[mode] = hip_attention_impl(q, k, v, args)[1]
    assert read_status("cuda") == 0
    a, b = md["auto"], md["strict"]
    for i, (x, y) in enumerate(zip(a.stage_caches[1:], b.stage_caches[1:])):
        assert torch.equal(x.indices_left, y.indices_left) and torch.equal(x.indices_right, y.indices_right), f"stage {i + 1}"
    assert torch.equal(a.indices, b.indices) and torch.equal(a.ks, b.ks)
    assert torch.equal(a.mask_cache_statistics.access_counter, b.mask_cache_statistics.access_counter)
