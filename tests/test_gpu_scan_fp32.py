"""fp32 prefill scan: rows left out by their distance from the largest approximate score.  Masks equal the oracle's for 32 to
256 pooled rows, head dims 64 to 256, ragged blocks, and for query rows that repeat or differ by one unit in the last place,
where several rows lie within the radius."""
import pytest
import torch

from oracle import hip_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", ["random", "repeated", "close"])
@pytest.mark.parametrize("bq,stride,D", [(64, 2, 64), (64, 1, 128), (128, 1, 256), (256, 1, 64)])
def test_masks_match_oracle(bq, stride, D, rows):
    import bench
    from hip_attention_b200 import hip_attention_impl, read_status
    w = dict(bench.WORKLOADS["prefill_4k_fp32"], TQ=201, T=1501, keep=[512, 256], sink=32, sw=64, H=4, HKV=2, D=D, bq=bq,
             strides=[stride, stride])
    q, k, v = bench.make_qkv(w, "cuda")
    if rows != "random":
        q = q[:, (torch.arange(w["TQ"], device="cuda") // 5) * 5].contiguous()
    if rows == "close":
        q[:, 1::2] = torch.nextafter(q[:, 1::2], torch.full_like(q[:, 1::2], 9.0))
    read_status("cuda")
    _, md = hip_attention_impl(q, k, v, bench.make_args(w))
    assert read_status("cuda") == 0
    pos = (torch.arange(w["TQ"]) + w["T"] - w["TQ"])[None]
    m = O.estimate_mask(q.cpu(), O.DenseKV(k.cpu()), pos, bench.oracle_config(w))
    assert torch.equal(md.indices.cpu(), m.indices) and torch.equal(md.ks.cpu(), m.ks)
