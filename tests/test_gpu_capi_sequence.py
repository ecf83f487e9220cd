"""The sequence of C calls a host in another language issues, function by function, against the operator: key copies, chunk
list, scans, selections, final conversion, attention; then the small helpers."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _scales(D, dtype):
    root = np.sqrt(np.float32(D)).astype(np.float32)
    ss = np.sqrt(root).astype(np.float32)
    return [torch.tensor(float(x)).to(dtype).item() for x in (root / ss, np.float32(1.0) / ss)]


@pytest.mark.parametrize("rope", [None, "relative", "streaming"])
@pytest.mark.parametrize("shape", [
    dict(TQ=201, T=3001, H=8, HKV=2, D=128),
    dict(TQ=130, T=2500, H=4, HKV=4, D=64, dtype="fp16"),
    dict(TQ=1, T=5003, H=8, HKV=2, D=128, B=3),
])
def test_calls_of_the_c_interface_equal_the_operator(shape, rope):
    import bench
    from cases import rope_tables
    from hip_attention_b200 import _lib as L, hip_attention_impl, read_status
    from hip_attention_b200.operator import _DT, _tokens, status_word
    lib = L.load()
    w = dict(bench.WORKLOADS["prefill_128k"], keep=[2048, 1024, 512], sink=64, sw=320)
    w.update(shape)
    B, TQ, T, H, HKV, D, bq, sink, sw = (w[n] for n in ("B", "TQ", "T", "H", "HKV", "D", "bq", "sink", "sw"))
    q, k, v = bench.make_qkv(w, "cuda")
    dt, rows, BDST = q.dtype, B * -(-TQ // bq), -(-TQ // bq)
    pos = (torch.arange(TQ, device="cuda") + T - TQ)[None].expand(B, TQ).contiguous()
    tables, kw = None, {}
    if rope:
        tables = [torch.from_numpy(t).cuda().to(dt) for t in rope_tables(T + 8, D, w["theta"])]
        kw = dict(using_extend=True, need_apply_rope=True, rope_cos=tables[0], rope_sin=tables[1], scan_extend_backend=rope)
    read_status("cuda")
    out, md, lse = hip_attention_impl(q, k, v, bench.make_args(w, position_ids=pos, **kw), return_lse=True)

    st, status = torch.cuda.current_stream().cuda_stream, status_word("cuda").data_ptr()
    q_scale, k_scale = _scales(D, dt)
    ktok, vtok = _tokens(k, None, None, None, "k"), _tokens(v, None, None, None, "v")

    def i32(*size):
        return torch.empty(size, dtype=torch.int32, device="cuda")
    key_abs = copy = None
    sides = 0
    if TQ > 1:
        if rope == "relative":
            sides = 2
            key_abs, copy = torch.empty((2, B, HKV, T), device="cuda"), torch.empty((2, B, HKV, T, D), dtype=dt, device="cuda")
            for side in range(2):
                L.check(lib.hipattn_scan_prepare_keys_rope(C.byref(ktok), _DT[dt], D, B, T, HKV, k_scale, tables[0].data_ptr(), tables[1].data_ptr(),
                                                           tables[0].stride(0), tables[0].shape[0], side, key_abs[side].data_ptr(), copy[side].data_ptr(),
                                                           status, st), "scan_prepare_keys_rope")
        elif rope is None or D == 128:
            sides = 1
            key_abs, copy = torch.empty((B, HKV, T), device="cuda"), torch.empty((B, HKV, T, D), dtype=dt, device="cuda")
            scale = 1.0 if rope else k_scale
            L.check(lib.hipattn_scan_prepare_keys(C.byref(ktok), _DT[dt], D, B, T, HKV, scale, key_abs.data_ptr(), copy.data_ptr(), status, st), "prepare")
            ref = (k * torch.tensor(scale, dtype=dt, device="cuda")).permute(0, 2, 1, 3)
            assert torch.equal(copy, ref)
            assert torch.allclose(key_abs, ref.float().abs().sum(-1), rtol=1e-5)
            alone = torch.empty_like(key_abs)
            L.check(lib.hipattn_key_abs_sum(C.byref(ktok), _DT[dt], D, B, T, HKV, scale, alone.data_ptr(), status, st), "key_abs_sum")
            assert torch.allclose(alone, key_abs, rtol=1e-5)
    c0, window = w["chunks"][0], max(0, sw - w["chunks"][0])
    n = -(-max(0, T - sink - sw) // c0)
    left, right, score = i32(rows, n), i32(rows, n), i32(rows, n)
    L.check(lib.hipattn_init_chunks(left.data_ptr(), right.data_ptr(), score.data_ptr(), rows, n, sink, c0, T, window, st), "init_chunks")
    assert torch.equal(left[0].cpu(), sink + torch.arange(n, dtype=torch.int32) * c0)
    assert torch.equal(right, (left + c0).clamp(max=T - window)) and bool((score == lib.hipattn_encode_score(-32000.0)).all())
    group = 64
    for i, c in enumerate(w["chunks"]):
        group = max(16, 1 << (min(n, group) - 1).bit_length())
        sp = L.ScanParams()
        sp.q, sp.q_stride_b, sp.q_stride_t, sp.q_stride_h = q.data_ptr(), q.stride(0), q.stride(1), q.stride(2)
        sp.pos, sp.pos_stride_b, sp.pos_stride_t, sp.k = pos.data_ptr(), pos.stride(0), pos.stride(1), ktok
        sp.left, sp.right, sp.score_max, sp.status = left.data_ptr(), right.data_ptr(), score.data_ptr(), status
        if sides:
            sp.key_abs, sp.k_scaled, sp.k_scaled_sides = key_abs.data_ptr(), copy.data_ptr(), sides
        sp.dtype, sp.D, sp.B, sp.TQ, sp.H, sp.HKV, sp.T = _DT[dt], D, B, TQ, H, HKV, T
        sp.block_size_q, sp.stride_q, sp.n_chunks, sp.block_chunk = bq, w["strides"][i], n, group
        sp.scan_window, sp.q_scale, sp.k_scale, sp.mode, sp.chunk_size = window, q_scale, k_scale, L.SCAN_AUTO, c
        if rope:
            sp.rope_cos, sp.rope_sin, sp.rope_stride, sp.rope_rows = tables[0].data_ptr(), tables[1].data_ptr(), tables[0].stride(0), tables[0].shape[0]
            sp.rope_mode = L.ROPE_RELATIVE if rope == "relative" else L.ROPE_STREAMING
        L.check(lib.hipattn_scan_stage(C.byref(sp), st), "scan_stage")
        if i + 1 < len(w["chunks"]):
            nxt = w["chunks"][i + 1]
            keep = min(w["keep"][i] // c, n)
            n2 = keep * (c // nxt)
            nl, nr, ns = i32(rows, n2), i32(rows, n2), i32(rows, n2)
            L.check(lib.hipattn_select_stage(score.data_ptr(), left.data_ptr(), rows, n, keep, sink, c, nxt, nl.data_ptr(), nr.data_ptr(), ns.data_ptr(), st),
                    "select_stage")
            left, right, score, n = nl, nr, ns, n2
    K = min(w["keep"][-1] // w["chunks"][-1], n)
    idx, ks = (torch.empty(s, dtype=torch.int64, device="cuda") for s in ((B * H, BDST, K), (B * H, BDST)))
    kse = i32(B * H, BDST, 2)
    L.check(lib.hipattn_finalize_indices(score.data_ptr(), left.data_ptr(), n, 0, pos.data_ptr(), pos.stride(0), pos.stride(1), B, BDST, H, n, K,
                                         w["chunks"][-1], bq, idx.data_ptr(), ks.data_ptr(), kse.data_ptr(), st), "finalize_indices")
    assert torch.equal(idx, md.indices) and torch.equal(ks, md.ks) and torch.equal(kse, md.ks_start_end)

    bp = L.BsaParams()
    got, got_lse = torch.empty_like(out), torch.empty_like(lse)
    bp.q, bp.q_stride_b, bp.q_stride_t, bp.q_stride_h = q.data_ptr(), q.stride(0), q.stride(1), q.stride(2)
    bp.out, bp.o_stride_b, bp.o_stride_t, bp.o_stride_h = got.data_ptr(), got.stride(0), got.stride(1), got.stride(2)
    bp.pos, bp.pos_stride_b, bp.pos_stride_t, bp.k, bp.v = pos.data_ptr(), pos.stride(0), pos.stride(1), ktok, vtok
    bp.indices, bp.idx_stride_n, bp.idx_stride_d = idx.data_ptr(), idx.stride(0), idx.stride(1)
    bp.ks, bp.ks_stride_n, bp.ks_stride_d, bp.status = ks.data_ptr(), ks.stride(0), ks.stride(1), status
    bp.dtype, bp.D, bp.B, bp.TQ, bp.H, bp.HKV, bp.T = _DT[dt], D, B, TQ, H, HKV, T
    bp.block_size_q, bp.index_block_q, bp.block_size_k, bp.K = min(bq, 1 << (TQ - 1).bit_length()), bq, w["chunks"][-1], K
    bp.sink, bp.window, bp.heads_share_mask, bp.indices_ascending = sink, max(sw, c0), 1, 1
    if rope:
        bp.rope_cos, bp.rope_sin, bp.rope_stride, bp.rope_rows = tables[0].data_ptr(), tables[1].data_ptr(), tables[0].stride(0), tables[0].shape[0]
    bp.n_splits = lib.hipattn_attention_splits(C.byref(bp))
    if bp.n_splits > 1:
        part_o, part_lse = (torch.empty((B, TQ, H, bp.n_splits) + x, device="cuda") for x in ((D,), ()))
        bp.part_o, bp.part_lse = part_o.data_ptr(), part_lse.data_ptr()
        L.check(lib.hipattn_bsa_attention(C.byref(bp), st), "bsa_attention")
        L.check(lib.hipattn_merge_partials(part_o.data_ptr(), part_lse.data_ptr(), B * TQ * H, bp.n_splits, D, _DT[dt], got.data_ptr(), D,
                                           got_lse.data_ptr(), st), "merge_partials")
    else:
        bp.lse_out = got_lse.data_ptr()
        L.check(lib.hipattn_bsa_attention(C.byref(bp), st), "bsa_attention")
    assert read_status("cuda") == 0
    assert torch.equal(got, out) and torch.equal(got_lse, lse)


def test_score_and_bound_helpers():
    from hip_attention_b200 import _lib as L
    lib, st = L.load(), torch.cuda.current_stream().cuda_stream
    x = torch.randn(70001, device="cuda") * 100
    codes = torch.tensor([lib.hipattn_encode_score(v) for v in x[:300].tolist()], dtype=torch.int32, device="cuda")
    back = torch.empty(300, device="cuda")
    L.check(lib.hipattn_decode_scores(codes.data_ptr(), back.data_ptr(), 300, st), "decode_scores")
    assert torch.equal(back, x[:300])
    src = torch.randint(-2 ** 31, 2 ** 31 - 1, (70001,), device="cuda", dtype=torch.int32)
    dst = torch.empty(70001, dtype=torch.int64, device="cuda")
    L.check(lib.hipattn_widen_i32(src.data_ptr(), dst.data_ptr(), src.numel(), st), "widen_i32")
    assert torch.equal(dst, src.long())
