"""Decode attention against the fp64 recompute on the oracle's mask: key lists that leave warps and CTAs of a cluster without
keys, group sizes one to eight, both head dims, 16-bit and fp8 rows, explicit key ranges."""
import pytest
import torch

from oracle import hip_oracle as O
from util import output_tolerance

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ranges", [None, 3])
@pytest.mark.parametrize("kv", ["bf16", "fp16", "fp8"])
@pytest.mark.parametrize("shape", [
    dict(B=1, H=8, HKV=1, D=128, T=1, sw=256),            # a single key
    dict(B=1, H=3, HKV=1, D=128, T=330),                  # nothing selected, window and sink only
    dict(B=2, H=4, HKV=2, D=64, T=2049),
    dict(B=1, H=2, HKV=2, D=128, T=5003),
    dict(B=40, H=32, HKV=8, D=128, T=1500),               # more units than the GPU has room for
    dict(B=5, H=32, HKV=8, D=128, T=5003),                # clusters whose size is no power of two
    dict(B=24, H=16, HKV=4, D=64, T=3001),
    dict(B=3, H=32, HKV=8, D=128, T=5003),
])
def test_decode_attention_matches_oracle(shape, kv, ranges, monkeypatch):
    import bench
    from hip_attention_b200 import hip_attention_impl, read_status
    if ranges:
        monkeypatch.setenv("HIPATTN_DECODE_SPLITS", str(ranges))
    w = dict(bench.WORKLOADS["decode_128k"], kind="prefill", keep=[2048, 1024, 512], sink=64, sw=320, dtype="fp16" if kv == "fp16" else "bf16")
    w.update(shape)
    q, k, v = bench.make_qkv(w, "cuda")
    if kv == "fp8":
        k, v = k.to(torch.float8_e5m2), v.to(torch.float8_e5m2)
    read_status("cuda")
    out, md, lse = hip_attention_impl(q, k, v, bench.make_args(w), return_lse=True)
    assert read_status("cuda") == 0
    cfg = bench.oracle_config(w)
    n = min(w["B"], 3)
    pos = torch.full((n, 1), w["T"] - 1)
    qc, kf, vf = q[:n].cpu(), k[:n].to(q.dtype).cpu(), v[:n].to(q.dtype).cpu()
    m = O.estimate_mask(qc, O.DenseKV(kf), pos, cfg)
    rows = n * w["H"]
    assert torch.equal(md.indices[:rows].cpu(), m.indices) and torch.equal(md.ks[:rows].cpu(), m.ks)
    ref, lse_ref = O.attention_on_mask(qc, O.DenseKV(kf), O.DenseKV(vf), pos, m, sink=cfg.sink, sw=max(cfg.sw, cfg.stages[0].chunk_size), return_lse=True)
    mx, mean = output_tolerance(q.dtype)
    err = (out[:n].float().cpu().double() - ref.double()).abs()
    assert err.max().item() <= mx and err.mean().item() <= mean
    assert (lse[:n].cpu().double() - lse_ref).abs().max().item() < 2e-2
