"""Prefill attention cut into key ranges, on 16-bit and fp8 caches: every kernel, head dims 64 and 128, ragged blocks, ranges
of a single tile and ranges that stay empty, against the fp64 recompute on the oracle's mask."""
import pytest
import torch

from oracle import hip_oracle as O
from util import output_tolerance

pytestmark = pytest.mark.gpu

SHAPES = {
    "d128": dict(D=128, H=8, HKV=2, bq=64, dtype="bf16"),
    "d128_wide_block": dict(D=128, H=8, HKV=1, bq=128, dtype="fp16"),
    "d64": dict(D=64, H=4, HKV=2, bq=64, dtype="fp16"),
    "mha": dict(D=128, H=2, HKV=2, bq=64, dtype="bf16"),
    "fp32": dict(D=64, H=4, HKV=2, bq=64, dtype="fp32"),
    "fp32_d128": dict(D=128, H=4, HKV=1, bq=128, dtype="fp32"),
    "fp8_bf16": dict(D=128, H=8, HKV=2, bq=64, dtype="bf16", fp8=True),
    "fp8_fp16_d64": dict(D=64, H=4, HKV=2, bq=64, dtype="fp16", fp8=True),
}


@pytest.mark.parametrize("ranges", [1, 3, 64])
@pytest.mark.parametrize("tq", [64, 201])
@pytest.mark.parametrize("shape", list(SHAPES))
def test_key_ranges_match_oracle(shape, tq, ranges, monkeypatch):
    import bench
    from hip_attention_b200 import hip_attention_impl, read_status
    monkeypatch.setenv("HIPATTN_PREFILL_SPLITS", str(ranges))
    w = dict(bench.WORKLOADS["prefill_128k"], TQ=tq, T=3001, keep=[2048, 1024, 512], sink=64, sw=256, **SHAPES[shape])
    fp8 = w.pop("fp8", False)
    q, k, v = bench.make_qkv(w, "cuda")
    kk, vv = (k.to(torch.float8_e5m2), v.to(torch.float8_e5m2)) if fp8 else (k, v)
    read_status("cuda")
    out, md, lse = hip_attention_impl(q, kk, vv, bench.make_args(w), return_lse=True)
    assert read_status("cuda") == 0
    cfg = bench.oracle_config(w)
    pos = (torch.arange(tq) + w["T"] - tq)[None]
    qc, kc, vc = q.cpu(), kk.to(q.dtype).cpu(), vv.to(q.dtype).cpu()
    m = O.estimate_mask(qc, O.DenseKV(kc), pos, cfg)
    assert torch.equal(md.indices.cpu(), m.indices) and torch.equal(md.ks.cpu(), m.ks)
    ref, lse_ref = O.attention_on_mask(qc, O.DenseKV(kc), O.DenseKV(vc), pos, m, sink=cfg.sink, sw=max(cfg.sw, cfg.stages[0].chunk_size),
                                       return_lse=True)
    mx, mean = output_tolerance(q.dtype)
    err = (out.float().cpu().double() - ref.double()).abs()
    assert err.max().item() <= mx and err.mean().item() <= mean
    assert (lse.cpu().double() - lse_ref).abs().max().item() < 2e-2


@pytest.mark.parametrize("kernel", ["tcgen05", "mma"])
@pytest.mark.parametrize("shape", ["d128", "d64", "d128_wide_block", "fp32", "fp8_bf16"])
def test_cached_mask_in_any_order(shape, kernel, monkeypatch):
    """A caller's mask whose blocks do not ascend attends the same keys: a context of a few windows, where part of the selection
    lies inside the window of some rows only.  The mask as the operator returned it gives the bits of the call that made it."""
    import bench
    from hip_attention_b200 import HiPAttentionOutputMetadata, hip_attention_impl, read_status
    monkeypatch.setenv("HIPATTN_PREFILL_KERNEL", kernel)
    w = dict(bench.WORKLOADS["prefill_128k"], TQ=201, T=1501, keep=[1024, 1024, 1024], sink=64, sw=256, **SHAPES[shape])
    fp8 = w.pop("fp8", False)
    q, k, v = bench.make_qkv(w, "cuda")
    if fp8:
        k, v = k.to(torch.float8_e5m2), v.to(torch.float8_e5m2)
    read_status("cuda")
    out, md = hip_attention_impl(q, k, v, bench.make_args(w))
    again, _ = hip_attention_impl(q, k, v, bench.make_args(w), md)
    assert torch.equal(out, again)
    n = int(md.ks.min())
    assert n > 64 and bool((md.ks == n).all())
    order = torch.randperm(n, generator=torch.Generator().manual_seed(2)).cuda()
    idx = md.indices.clone()
    idx[:, :, :n] = md.indices[:, :, :n][:, :, order]
    mixed, _ = hip_attention_impl(q, k, v, bench.make_args(w), HiPAttentionOutputMetadata(idx, md.ks, md.ks_count, md.ks_start_end, None, None, None))
    assert read_status("cuda") == 0
    mx, mean = output_tolerance(q.dtype)
    err = (mixed.double() - out.double()).abs()
    assert err.max().item() <= mx and err.mean().item() <= mean
