"""The metadata pool on the GPU (all copies of a step in one launch) against the same pool on the CPU (one tensor operation
each): expanded, strided and narrowed values, INT64_MAX padding, rows beyond the batch left alone."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [1, 3, 32])
@pytest.mark.parametrize("layer", [0, 5])
def test_pool_on_gpu_equals_pool_on_cpu(batch, layer):
    from hip_attention_b200 import (HiPAttentionConfig, HiPAttentionOutputMetadata, HiPAttentionStageInputCache, HiPMetadataCachePool)
    cfg, H = HiPAttentionConfig(), 8
    pools = {d: HiPMetadataCachePool(4096, H, 6, 65536, d, cfg) for d in ("cpu", "cuda")}
    g = torch.Generator().manual_seed(batch * 10 + layer)
    n_idx = pools["cpu"].cache[layer]["indices"].buffer.shape[-1]
    idx = torch.randint(0, 2 ** 31 - 1, (batch * H, 1, n_idx), generator=g)
    idx[:, :, -5:] = torch.iinfo(torch.int64).max
    ks = torch.randint(0, n_idx, (batch * H, 1), generator=g)
    caches = [HiPAttentionStageInputCache(None, None, None)]
    for i in (1, 2):
        n = pools["cpu"].cache[layer][f"stage_{i}_indices_left"].buffer.shape[-1]
        lr = [torch.randint(0, 65536, (batch, 1, 1, n), generator=g).expand(batch, 1, H, n) for _ in range(2)]
        caches.append(HiPAttentionStageInputCache(lr[0], lr[1], torch.randn((batch, 1, n, H), generator=g).transpose(2, 3)))

    def on(dev, c):
        return HiPAttentionStageInputCache(*[None if t is None else t.to(dev) for t in (c.indices_left, c.indices_right, c.out_scores)])
    got = {}
    for dev, pool in pools.items():
        for b in pool.cache[layer].values():
            b.buffer.fill_(7)
        md = HiPAttentionOutputMetadata(idx.to(dev), ks.to(dev), ks.unsqueeze(-1).to(dev),
                                        torch.stack([torch.zeros_like(ks), ks], -1).to(torch.int32).to(dev), None, None, [on(dev, c) for c in caches])
        pool.set_hip_metadata_cache(layer, batch, batch, md)
        whole, part = pool.get_hip_metadata_cache(layer, batch, batch, None), pool.get_hip_metadata_cache(layer, batch, batch, 2)
        got[dev] = [b.buffer for b in pool.cache[layer].values()] + [whole.indices, whole.ks, whole.ks_count, whole.ks_start_end]
        got[dev] += [t for c in part.stage_caches[1:] for t in (c.indices_left, c.indices_right, c.out_scores)]
    for a, b in zip(got["cpu"], got["cuda"]):
        assert a.dtype == b.dtype and a.shape == b.shape and torch.equal(a.to(torch.float64), b.cpu().to(torch.float64))


@pytest.mark.parametrize("order", [(3, 2, 1, 0), (0, 3, 2, 1), (2, 0, 3, 1)])
def test_values_of_any_stride_in_one_launch(order):
    """Several values whose dimensions do not merge: each arrives in its own buffer, the rows behind it untouched."""
    from hip_attention_b200.operator import host
    g = torch.Generator(device="cuda").manual_seed(sum(i * x for i, x in enumerate(order)))
    shape = (3, 4, 5, 6)
    back = [order.index(i) for i in range(4)]
    vals = [torch.randint(0, 1000, [shape[i] for i in order], generator=g, device="cuda").permute(back) for _ in range(9)]
    bufs = [torch.full((5, 4, 5, 6), -1, dtype=torch.int32, device="cuda") for _ in vals]
    assert vals[0].shape == shape and host().pool_write([(b, v, 5) for b, v in zip(bufs, vals)]) == []
    for b, v in zip(bufs, vals):
        assert torch.equal(b[:3].long(), v) and bool((b[3:] == -1).all())
