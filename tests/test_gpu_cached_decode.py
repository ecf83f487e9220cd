"""Cached decode calls, whose attention reads the mask it is given and runs beside the copies of it that the call returns."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def call(B, dtype, T=6007):
    from hip_attention_b200 import HiPAttentionArgs, ScanStage, hip_attention_12
    g = torch.Generator(device="cuda").manual_seed(B)
    H, HKV, D, P = 16, 4, 128, 16
    pages = B * -(-T // P)
    kc, vc = (torch.randn((pages, P, HKV, D), generator=g, device="cuda", dtype=dtype) for _ in range(2))
    table = torch.randperm(pages, generator=g, device="cuda").view(B, -1).to(torch.int32)
    lens = torch.full((B,), T, dtype=torch.int32, device="cuda")
    stages = [ScanStage(64, 4, c, k, 1) for c, k in ((256, None), (32, 2048), (8, 1024))]
    args = HiPAttentionArgs(sink_token_size=64, sliding_window_size=512, second_stage_k=512, stages=stages, block_sparse_block_size_q=64, k_cache=kc,
                            v_cache=vc, block_table=table, cache_seq_lens=lens, position_ids=(lens.long() - 1).view(B, 1), extend_context_length=T,
                            require_cache_statistics=False)
    q = torch.randn((B, 1, H, D), generator=g, device="cuda", dtype=dtype) * D ** -0.5
    return hip_attention_12, q, args


def fields(md):
    return md.indices, md.ks, md.ks_count, md.ks_start_end


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("B", [1, 3, 32])
def test_cached_call_equals_fresh_call(B, dtype):
    run, q, args = call(B, dtype)
    context, md = run(q, None, None, args)
    narrow = type(md)(md.indices.clamp(max=2 ** 31 - 1).to(torch.int32), *fields(md)[1:], None, None, None)   # read from the copies
    chain = md
    for step in range(20):    # each call's mask is the copy that the call before returned
        out, chain = run(q, None, None, args, chain)
        assert torch.equal(out, context), step
        assert all(torch.equal(a, b) for a, b in zip(fields(chain), fields(md))), step
        assert chain.indices.data_ptr() != md.indices.data_ptr()
    out, m = run(q, None, None, args, narrow)
    assert torch.equal(out, context) and torch.equal(m.ks, md.ks)


def test_cached_call_under_capture_and_on_another_stream():
    run, q, args = call(2, torch.bfloat16)
    context, md = run(q, None, None, args)
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        out, m = run(q, None, None, args, md)
        out2, m2 = run(q, None, None, args, m)
    for _ in range(3):
        out.zero_(), out2.zero_(), m.indices.zero_(), m2.indices.zero_()
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, context) and torch.equal(out2, context)
    assert torch.equal(m.indices, md.indices) and torch.equal(m2.indices, md.indices)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        out, m = run(q, None, None, args, md)
        total = m.indices.sum() + m.ks.sum()    # ordinary work behind the call finds the copies complete
    torch.cuda.current_stream().wait_stream(side)
    assert torch.equal(out, context) and int(total) == int(md.indices.sum() + md.ks.sum())
