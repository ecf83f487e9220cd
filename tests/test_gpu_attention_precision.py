"""Attention whose softmax weights go through the tensor cores in two 16-bit terms, against 64 bits on the mask it used: what is
left besides the rounding of the output itself is small.

The bound: two terms keep 16 (bf16) or 22 (fp16) significant bits of a weight, 1.5e-5 or 2.4e-7, and a score is a fp32 sum of 64
or 128 products, good to a few 1e-6 after the exponential: the context before it is rounded is within p = 4e-5 (bf16) or 8e-6
(fp16) of the exact one, relative.  The rounding of the output alone is r = 1.6e-3 or 2.0e-4, and the two add in quadrature:
sqrt(1 + (p / r)^2) r < 1.0005 r and 1.001 r.  With single 16-bit weights p is 1e-4 to 9e-4 in bf16 and 1.2e-5 to 1e-4 in fp16, and
the sum 1.0018 r to 1.08 r on all of these shapes but the ones a whole cluster or fp32 weights served."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rotate(x, tables, pos):
    """Rows x [n, heads, D] at table positions pos [n]; products and sum rounded to the element type, as the kernels do."""
    cos, sin = (t.to(x.dtype)[pos][:, None] for t in tables)
    half = x.shape[-1] // 2
    return x * cos + torch.cat([-x[..., half:], x[..., :half]], -1) * sin


def _exact(q, k, v, md, rows, w, tables):
    """[n, H, D] in 64 bits: queries ``rows`` (batch, index, position) of q [B, TQ, H, D] over sink, selected blocks, window."""
    H, G, c, window = w["H"], w["H"] // w["HKV"], w["chunks"][-1], max(w["sw"], w["chunks"][0])
    out = []
    for b, r, p in rows:
        t = torch.arange(w["T"], device=q.device)
        blocks = md.indices[b * H, r // w["bq"], :int(md.ks[b * H, r // w["bq"]])]
        sel = torch.zeros(w["T"] + c, dtype=torch.bool, device=q.device)
        sel[(blocks[:, None] + torch.arange(c, device=q.device)).flatten()] = True
        far = ((t < w["sink"]) | sel[:w["T"]]) & (t <= p - window)
        t = t[far | ((t > p - window) & (t <= p))]
        qr, kk = q[b, r], k[b, t]
        if tables is not None:   # one row per block: a far key goes to its rank in [sink | selected], shifted
            n_far, n_sel = int(far.sum()), blocks.numel() * c
            order = torch.cat([torch.arange(w["sink"], device=q.device), (blocks[:, None] + torch.arange(c, device=q.device)).flatten()])
            rank = torch.zeros(w["T"] + c, dtype=torch.int64, device=q.device)
            rank[order] = torch.arange(order.numel(), device=q.device)
            pos = torch.cat([(rank[t[:n_far]] + p - window - w["sink"] - n_sel + 1).clamp(min=0), t[n_far:]])
            qr, kk = _rotate(qr[None], tables, torch.tensor([p], device=q.device))[0], _rotate(kk, tables, pos)
        kk, vv = kk.double().repeat_interleave(G, 1), v[b, t].double().repeat_interleave(G, 1)
        s = torch.einsum("hd,nhd->hn", qr.double(), kk)
        out.append(torch.einsum("hn,nhd->hd", torch.softmax(s, -1), vv))
    return torch.stack(out)


@pytest.mark.parametrize("dtype", ["bf16", "fp16"])
@pytest.mark.parametrize("shape", [
    dict(TQ=201, T=9001, D=64, bq=64),                       # prefill, two heads per CTA
    dict(TQ=130, T=9001, D=64, bq=128),                      # one head, 128 rows
    dict(TQ=1, T=20011, D=128, bq=64, fp8=True),             # decode, a list shared by a whole cluster
    dict(TQ=1, T=20011, D=64, bq=64, rope=True),
    dict(TQ=1, T=20011, D=128, bq=64, B=12, H=32, HKV=8),    # by two CTAs
    dict(TQ=1, T=20011, D=64, bq=64, B=12, H=32, HKV=8),
    dict(TQ=1, T=5003, D=128, bq=64, B=40, rope=True),       # by one CTA
    dict(TQ=1, T=5003, D=128, bq=64, B=40, H=16, rope=True, fp8=True),   # eight heads per KV head
])
def test_error_is_the_rounding_of_the_output(shape, dtype):
    import bench
    from cases import rope_tables
    from hip_attention_b200 import hip_attention_impl, read_status
    w = dict(bench.WORKLOADS["prefill_128k"], H=8, HKV=2, keep=[4096, 2048, 1024], dtype=dtype)
    w.update(shape)
    g = torch.Generator(device="cuda").manual_seed(9)
    dt = bench._DT[dtype]
    q, k, v = (torch.randn((w["B"], n, h, w["D"]), generator=g, device="cuda", dtype=dt) for n, h in ((w["TQ"], w["H"]), (w["T"], w["HKV"]), (w["T"], w["HKV"])))
    q = q * w["D"] ** -0.5
    k[:, ::100] *= 4
    if w.get("fp8"):
        k, v = k.to(torch.float8_e5m2), v.to(torch.float8_e5m2)
    tables, kw = None, {}
    if w.get("rope"):
        tables = [torch.from_numpy(t).cuda() for t in rope_tables(w["T"] + 8, w["D"], 5e5)]
        kw = dict(using_extend=True, need_apply_rope=True, rope_cos=tables[0], rope_sin=tables[1])
    read_status("cuda")
    out, md = hip_attention_impl(q, k, v, bench.make_args(w, **kw))
    assert read_status("cuda") == 0
    rows = [(b, r, w["T"] - w["TQ"] + r) for b in range(w["B"]) for r in range(0, w["TQ"], max(1, w["TQ"] // 24))]
    ref = _exact(q, k.to(dt), v.to(dt), md, rows, w, tables)
    err = (out[[b for b, _, _ in rows], [r for _, r, _ in rows]].double() - ref).norm().item()
    rounding = (ref.to(dt).double() - ref).norm().item()
    print(f"{shape} {dtype}: error {err / ref.norm().item():.4e}, rounding alone {rounding / ref.norm().item():.4e}, ratio {err / rounding:.4f}")
    assert err <= (1.0005 if dtype == "bf16" else 1.001) * rounding
