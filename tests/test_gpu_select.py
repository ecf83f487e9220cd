"""Selection between stages and final conversion against torch sorts: row lengths around the kernels' limits, rows full of equal
scores, everything kept, lists out of order, duplicates."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rows(n, rows, kind, seed):
    g = torch.Generator().manual_seed(seed)
    score = torch.randn((rows, n), generator=g)
    if kind == "ties":
        score = torch.randint(-3, 3, (rows, n), generator=g).float()
    elif kind == "half_init":
        score[:, n // 2:] = -32000.0
    left = (torch.arange(n) * 32 + 64)[None].repeat(rows, 1)
    if kind == "unordered":
        left = torch.stack([left[0, torch.randperm(n, generator=g)] for _ in range(rows)])
        left[:, ::7] = left[:, :1].clone()          # duplicates
    return score, left


def _codes(score):
    bits = score.view(torch.int32)
    return torch.where(bits < 0, bits ^ 0x7fffffff, bits).to(torch.int32)


@pytest.mark.parametrize("kind", ["random", "ties", "half_init", "unordered"])
@pytest.mark.parametrize("n,keep", [(1, 1), (31, 7), (33, 33), (1000, 999), (1024, 256), (1025, 512), (4096, 2048), (4097, 1), (16384, 2048)])
def test_selection_equals_sorting(n, keep, kind):
    from hip_attention_b200 import _lib as L
    lib, rows, sink, H = L.load(), 3, 64, 2
    score, left = _rows(n, rows, kind, n + keep)
    order = torch.sort(score, dim=1, descending=True, stable=True).indices[:, :keep]
    la = torch.gather(left, 1, order).sort(1).values          # already on the grid of 32
    ref_l = (la[:, :, None] + torch.arange(4) * 8).flatten(1)
    code, l32 = _codes(score).cuda(), left.to(torch.int32).cuda()
    out = [torch.empty((rows, keep * 4), dtype=torch.int32, device="cuda") for _ in range(3)]
    st = torch.cuda.current_stream().cuda_stream
    L.check(lib.hipattn_select_stage(code.data_ptr(), l32.data_ptr(), rows, n, keep, sink, 32, 8, *[o.data_ptr() for o in out], st), "select_stage")
    assert torch.equal(out[0].cpu().long(), ref_l) and torch.equal(out[1].cpu().long(), ref_l + 8)
    assert bool((out[2].cpu() == lib.hipattn_encode_score(-32000.0)).all())
    # final conversion: ascending, duplicates (wrapping around) to padding behind the rest
    pad = torch.iinfo(torch.int64).max
    ref = la // 8 * 8
    own = ref != torch.roll(ref, 1, 1)
    ref_i = torch.where(own, ref, torch.full_like(ref, pad)).sort(1).values
    pos = torch.tensor([[n * 16 + 3]] * rows, device="cuda")
    idx = torch.empty((rows * H, 1, keep), dtype=torch.int64, device="cuda")
    ks = torch.empty((rows * H, 1), dtype=torch.int64, device="cuda")
    kse = torch.empty((rows * H, 1, 2), dtype=torch.int32, device="cuda")
    L.check(lib.hipattn_finalize_indices(code.data_ptr(), l32.data_ptr(), n, 0, pos.data_ptr(), 1, 1, rows, 1, H, n, keep, 8, 64,
                                         idx.data_ptr(), ks.data_ptr(), kse.data_ptr(), st), "finalize_indices")
    ref_k = (ref_i < n * 16 + 3 + 64).sum(1)
    assert torch.equal(idx.cpu()[:, 0], ref_i.repeat_interleave(H, 0))
    assert torch.equal(ks.cpu()[:, 0], ref_k.repeat_interleave(H)) and torch.equal(kse.cpu()[:, 0, 1].long(), ref_k.repeat_interleave(H))
