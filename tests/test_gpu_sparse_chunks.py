"""Sparse attention where chunks of the selection hold no key: a short sequence, gaps in the middle, no key at all; one and
several blocks a chunk, the merge alone and with the value rows of one to five tokens.  Against the plain f64 result on the same bf16
rows; probabilities are rounded to bf16 and so is the result: 2^-8 of the largest value each."""

import pytest
import torch

pytestmark = pytest.mark.gpu
BF16, F32, F64, I32 = torch.bfloat16, torch.float32, torch.float64, torch.int32


@pytest.fixture(scope="module")
def ops():
    import tilert_b200 as tb
    from tilert_b200.models.deepseek_v3_2 import ops

    tb.load_backend("deepseek_v3_2")
    tb.tilert_init(0)
    yield ops
    assert tb.device_status(0) == 0


def selection(kind, tokens, topk, pos, gen):
    sel = torch.full((tokens, topk), -1, dtype=I32)
    for t in range(tokens):
        n = min(pos + t + 1, topk)
        rows = torch.randperm(pos + t + 1, generator=gen)[:n].sort()[0].to(I32)
        if kind == "front":
            sel[t, :n] = rows
        elif kind == "gap":          # the first chunk and one in the middle are empty
            keep = min(n, 40)
            sel[t, 70: 70 + keep // 2] = rows[: keep // 2]
            sel[t, topk - keep + keep // 2:] = rows[keep // 2: keep]
        elif kind == "late":         # rows past the position do not count
            sel[t, :n] = rows
            sel[t, n:] = pos + tokens + 3
    return sel


@pytest.mark.parametrize("tokens", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("split", [64, 128])
@pytest.mark.parametrize("kind,pos", [("front", 3), ("front", 64), ("gap", 300), ("late", 20), ("none", 5), ("front", 600)])
def test_chunks_without_keys(ops, tokens, split, kind, pos):
    heads, topk, rows, scale = 40, 512, 700, 0.05
    gen = torch.Generator().manual_seed(pos + tokens)
    q, qp, kv, pe = (torch.randn(*s, generator=gen).to(BF16) for s in ((1, tokens, heads, 512), (1, tokens, heads, 64), (1, rows, 512), (1, rows, 64)))
    sel = selection(kind, tokens, topk, pos, gen)
    ns = topk // split
    acc = torch.full((tokens, heads, ns, 512), float("nan"), device="cuda")
    lse_acc, lse = torch.zeros(tokens, heads, ns, device="cuda"), torch.zeros(tokens, heads, device="cuda")
    out = torch.zeros(1, tokens, heads, 512, dtype=BF16, device="cuda")
    cur = torch.tensor([pos], dtype=I32, device="cuda")
    args = (q.cuda(), qp.cuda(), kv.cuda(), pe.cuda(), sel.view(1, tokens, topk).cuda(), cur)
    ops.flash_sparse_mla(*args, out, softmax_scale=scale, split_size=split, out_acc=acc, lse=lse, lse_acc=lse_acc)
    empty = torch.tensor([[not any(0 <= int(i) <= pos + t for i in sel[t, c * split: (c + 1) * split]) for c in range(ns)] for t in range(tokens)])
    for t in range(tokens):
        ok = [int(i) for i in sel[t] if 0 <= int(i) <= pos + t]
        if ok:
            k, p = kv[0, ok].to(F64), pe[0, ok].to(F64)
            z = (q[0, t].to(F64) @ k.T + qp[0, t].to(F64) @ p.T) * scale
            want = torch.softmax(z, -1) @ k
            assert float((lse[t].cpu().to(F64) - torch.logsumexp(z, -1)).abs().max()) < 0.02
        else:
            want = torch.zeros(heads, 512, dtype=F64)
            assert bool((lse[t] == -float("inf")).all())
        assert float((out[0, t].cpu().to(F64) - want).abs().max()) <= 2.0 ** -7 * float(kv.abs().max())
    e = empty[:, None].expand(tokens, heads, ns).cuda()
    assert bool((acc[e] == 0).all()) and bool((lse_acc[e] == -float("inf")).all()) and bool(torch.isfinite(acc).all())
    # the merge with value rows sees the same latent output, whatever tokens share a thread block
    w_v = torch.randint(0, 0x40, (heads, 4, 16448), dtype=torch.uint8, generator=gen)
    w_v[..., 16384:] = torch.full((heads, 4, 16), 0.01).view(torch.uint8)
    w_v, o2, lat = w_v.cuda(), torch.zeros(1, tokens, heads, 128, dtype=BF16, device="cuda"), torch.zeros_like(out)
    ops.flash_sparse_mla(*args, lat, softmax_scale=scale, split_size=split, out_acc=acc, lse_acc=lse_acc, w_v=w_v, o_out=o2)
    assert torch.equal(lat, out)
    for t in range(tokens):
        one, cur1 = torch.zeros(1, 1, heads, 128, dtype=BF16, device="cuda"), torch.tensor([pos + t], dtype=I32, device="cuda")
        a1, l1, lat1 = torch.zeros(1, heads, ns, 512, device="cuda"), torch.zeros(1, heads, ns, device="cuda"), torch.zeros(1, 1, heads, 512, dtype=BF16, device="cuda")
        ops.flash_sparse_mla(args[0][:, t: t + 1].contiguous(), args[1][:, t: t + 1].contiguous(), args[2], args[3], args[4][:, t: t + 1].contiguous(), cur1,
                             lat1, softmax_scale=scale, split_size=split, out_acc=a1, lse_acc=l1, w_v=w_v, o_out=one)
        assert torch.equal(one[0, 0], o2[0, t])


@pytest.mark.parametrize("tokens", [1, 4])
@pytest.mark.parametrize("split", [64, 128])
@pytest.mark.parametrize("kind", ["nan_row", "nan_alone", "nan_query", "inf_alone", "inf_row"])
def test_what_is_no_number_is_not_lost(ops, tokens, split, kind):
    """A cache row or a query with a NaN, or with an infinity that makes scores +inf (the result is no number) or -inf (no weight, but
    its values are infinite), among other keys and alone in its chunk.  NaN where the plain f64 result has it, close elsewhere."""
    heads, topk, rows, pos, scale = 40, 1280, 700, 600, 0.05  # (ten or twenty chunks: the merge's first batch and the next)
    gen = torch.Generator().manual_seed(tokens)
    q, qp, kv, pe = (torch.randn(*s, generator=gen).to(BF16) for s in ((1, tokens, heads, 512), (1, tokens, heads, 64), (1, rows, 512), (1, rows, 64)))
    bad = 3
    if kind == "nan_query":
        q[0, 0, 1, 7] = float("nan")
    elif kind.startswith("nan"):
        kv[0, bad, 9] = float("nan")
    else:
        kv[0, bad, 9] = float("inf")
    sel = torch.full((tokens, topk), -1, dtype=I32)
    sel[:, :200] = torch.arange(10, 210, dtype=I32)
    sel[:, 1279 if kind.endswith("alone") else 70] = bad
    acc = torch.zeros(tokens, heads, topk // split, 512, device="cuda")
    lse_acc, lse = torch.zeros(tokens, heads, topk // split, device="cuda"), torch.zeros(tokens, heads, device="cuda")
    out, lat = (torch.zeros(1, tokens, heads, 512, dtype=BF16, device="cuda") for _ in range(2))
    args = (q.cuda(), qp.cuda(), kv.cuda(), pe.cuda(), sel.view(1, tokens, topk).cuda(), torch.tensor([pos], dtype=I32, device="cuda"))
    ops.flash_sparse_mla(*args, out, softmax_scale=scale, split_size=split, out_acc=acc, lse=lse, lse_acc=lse_acc)
    w_v, o2 = torch.zeros(heads, 4, 16448, dtype=torch.uint8, device="cuda"), torch.zeros(1, tokens, heads, 128, dtype=BF16, device="cuda")
    ops.flash_sparse_mla(*args, lat, softmax_scale=scale, split_size=split, out_acc=acc, lse_acc=lse_acc, w_v=w_v, o_out=o2)
    for t in range(tokens):
        ok = [int(i) for i in sel[t] if i >= 0]
        k, p = kv[0, ok].to(F64), pe[0, ok].to(F64)
        z = (q[0, t].to(F64) @ k.T + qp[0, t].to(F64) @ p.T) * scale
        want, norm = torch.softmax(z, -1) @ k, torch.logsumexp(z, -1)
        for got in (out, lat):
            a = got[0, t].cpu().to(F64)
            assert torch.equal(a.isnan(), want.isnan())
            assert float((a - want).nan_to_num(0.0).abs().max()) <= 2.0 ** -7 * float(kv[kv.isfinite()].abs().max())
        fine = norm.isfinite()
        assert float((lse[t].cpu().to(F64) - norm)[fine].abs().max()) < 0.02 if bool(fine.any()) else True
        assert bool(lse[t].cpu()[~fine].isnan().all()) and bool(want.isnan().any()) == (kind != "nan_query" or t == 0)
