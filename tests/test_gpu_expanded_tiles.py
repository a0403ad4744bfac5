"""Attention over expanded keys and values on 128 x 128 tiles against the plain f64 restatement on the same bf16 operands.

The probabilities and the result are rounded to bf16 (2^-9 of a value each, independent) and the exponentials are good to a
few f32 ulps of an argument: the 2-norm of the error stays below 2^-8 of the result's, and a row's below twice that."""

import types

import pytest
import torch

pytestmark = pytest.mark.gpu

BF16, F32, F64, I32 = torch.bfloat16, torch.float32, torch.float64, torch.int32


@pytest.fixture(scope="module")
def ops():
    import tilert_b200 as tb
    from tilert_b200 import gqa_ops

    tb.load_backend("ralasun")
    tb.tilert_init(0, "ralasun")
    yield gqa_ops
    assert tb.device_status(0, "ralasun") == 0


def rnd(gen, *shape, std=1.0, dtype=BF16):
    return (torch.randn(*shape, generator=gen, device="cuda") * std).to(dtype)


def pad16(n):
    return (n + 15) // 16 * 16


# heads, dim, rot, vdim, rank, rows, position of row 0, window (0: none), sink, gate, size of scores
CASES = [
    (2, 128, 64, 128, 512, 128, 0, 0, False, None, 1.0),          # one tile
    (3, 128, 64, 128, 512, 129, 0, 0, False, "element", 1.0),     # a second tile of one row
    (1, 96, 32, 128, 256, 255, 77, 0, True, "head", 1.0),
    (5, 64, 32, 64, 384, 256, 0, 128, True, "element", 1.0),
    (2, 64, 64, 96, 512, 257, 1000, 129, False, "head", 1.0),
    (160, 64, 32, 64, 256, 384, 5, 0, True, None, 1.0),           # two query tiles per CTA, the last CTA with one
    (80, 128, 64, 128, 512, 300, 700, 200, True, "element", 1.0),
    (150, 96, 64, 96, 384, 130, 4000, 1024, False, "head", 1.0),
    (2, 128, 64, 128, 512, 200, 3333, 30, True, "head", 1.0),     # a window smaller than a tile, a ring wound many times
    (150, 128, 64, 128, 512, 300, 1999, 1, False, None, 1.0),     # every query sees itself alone
    (4, 40, 6, 72, 48, 131, 200, 0, False, "element", 1.0),       # parts of pieces
    (3, 17, 6, 9, 24, 140, 0, 64, True, "element", 1.0),
    (2, 24, 2, 100, 130, 128, 513, 513, False, None, 1.0),
    (150, 128, 64, 128, 512, 512, 100, 0, True, "element", 40.0), # maxima that grow along the keys: sums are rescaled
    (2, 128, 64, 128, 512, 512, 100, 0, False, None, 40.0),
]


@pytest.mark.parametrize("case", CASES)
def test_against_plain_attention(ops, case):
    heads, dim, rot, vdim, rank, rows, pos, window, with_sink, gating, size = case
    gen = torch.Generator(device="cuda").manual_seed(heads * 1000 + rows)
    t = pos + rows
    ring = window - 1 + rows if window else t + 3
    dimp, rotp, vdimp, rankp, row = pad16(dim), pad16(rot), pad16(vdim), pad16(rank), ops.latent_row_len(rank, rot)
    mix = types.SimpleNamespace(heads=heads, dim=dim, rot_dim=rot, vdim=vdim, kv_rank=rank, scale=(dim + rot) ** -0.5)
    q = torch.zeros(rows, heads, dimp + rotp, dtype=BF16, device="cuda")
    q[..., :dim], q[..., dimp: dimp + rot] = rnd(gen, rows, heads, dim), rnd(gen, rows, heads, rot)
    grow = torch.linspace(0, size, t, device="cuda")[:, None, None] if size > 1 else 1.0
    k, v, kr = (rnd(gen, t, heads, dim, dtype=F32) * grow).to(BF16), rnd(gen, t, heads, vdim), rnd(gen, t, rot)
    cached = min(t, ring)
    # rows behind those in use hold no numbers
    kv = torch.full((cached + 128, heads * (dimp + vdimp)), float("nan"), dtype=BF16, device="cuda")
    cache = types.SimpleNamespace(rows=torch.zeros(ring, row, dtype=BF16, device="cuda"), ring=ring, window=window)
    slots = torch.arange(max(0, t - cached), t, device="cuda")
    at = slots % ring
    kvk, kvv = torch.zeros(cached, heads, dimp, dtype=BF16, device="cuda"), torch.zeros(cached, heads, vdimp, dtype=BF16, device="cuda")
    kvk[at, :, :dim], kvv[at, :, :vdim] = k[slots], v[slots]
    kv[:cached] = torch.cat([kvk.flatten(1), kvv.flatten(1)], 1)
    cache.rows[at, rankp: rankp + rot] = kr[slots]
    sink = rnd(gen, heads, dtype=F32) if with_sink else None
    gate = {None: None, "head": rnd(gen, rows, heads, dtype=F32), "element": rnd(gen, rows, heads * vdim, dtype=F32)}[gating]
    out = torch.zeros(rows, ops.pad(heads * vdim), dtype=BF16, device="cuda")
    ops.expanded_attn(q, kv, cache, rows, mix, torch.tensor([pos], dtype=I32, device="cuda"), sink, gate, gating == "head", out)
    got = out[:, : heads * vdim].view(rows, heads, vdim).to(F64)

    i, j = torch.arange(pos, t, device="cuda")[:, None], torch.arange(t, device="cuda")[None]
    hidden = (j > i) | ((i - j >= window) if window else torch.zeros_like(j > i))
    want = torch.empty_like(got)
    for h in range(heads):
        s = (q[:, h, :dim].to(F64) @ k[:, h].to(F64).T + q[:, h, dimp: dimp + rot].to(F64) @ kr.to(F64).T) * mix.scale
        s = s.masked_fill(hidden, float("-inf"))
        if sink is not None:
            s = torch.cat([s, sink[h].to(F64).expand(rows, 1)], 1)
        want[:, h] = torch.softmax(s, -1)[:, :t] @ v[:, h].to(F64)
    if gating == "head":
        want *= torch.sigmoid(gate.to(F64))[..., None]
    elif gating == "element":
        want *= torch.sigmoid(gate.to(F64)).view_as(want)
    off = got - want
    assert float(off.norm()) <= 2.0 ** -8 * float(want.norm())
    assert float((off.norm(dim=-1) - 2.0 ** -7 * want.norm(dim=-1)).max()) <= 1e-6


@pytest.mark.parametrize("rows,pos,window,spread", [(256, 0, 0, 1.0), (256, 0, 0, 4.0), (512, 700, 128, 1.0), (777, 1000, 0, 2.0)])
def test_error_of_the_probabilities(ops, rows, pos, window, spread):
    """Probabilities are rounded relative to the largest score of a row after every 64 keys: the error against f64 is that of a
    restatement which rounds there and nowhere else but in the result.  (References every 128 keys raise it by 0.3 to 0.8 %; the
    exponentials' own errors and another place of the first tile move it by less than 0.1 %.)"""
    heads, dim, rot, vdim, rank, t = 8, 128, 64, 128, 64, pos + rows
    ring, cat = window - 1 + rows if window else t, torch.cat
    gen = torch.Generator(device="cuda").manual_seed(rows)
    mix = types.SimpleNamespace(heads=heads, dim=dim, rot_dim=rot, vdim=vdim, kv_rank=rank, scale=(dim + rot) ** -0.5)
    q, k, v, kr = rnd(gen, rows, heads, dim + rot, std=spread), rnd(gen, t, heads, dim), rnd(gen, t, heads, vdim), rnd(gen, t, rot)
    cache = types.SimpleNamespace(rows=torch.zeros(ring, ops.latent_row_len(rank, rot), dtype=BF16, device="cuda"), ring=ring, window=window)
    kv = torch.zeros(ring, heads * (dim + vdim), dtype=BF16, device="cuda")
    used = torch.arange(max(0, t - ring), t, device="cuda")
    kv[used % ring] = cat([k[used].flatten(1), v[used].flatten(1)], 1)
    cache.rows[used % ring, rank: rank + rot] = kr[used]
    out = torch.zeros(rows, heads * vdim, dtype=BF16, device="cuda")
    ops.expanded_attn(q, kv, cache, rows, mix, torch.tensor([pos], dtype=I32, device="cuda"), None, None, False, out)

    s = torch.einsum("thd,khd->htk", q.to(F64), cat([k, kr[:, None].expand(-1, heads, -1)], -1).to(F64)) * mix.scale
    i, j = torch.arange(pos, t, device="cuda")[:, None], torch.arange(t, device="cuda")[None]
    s = s.masked_fill((j > i) | ((i - j >= window) if window else False), float("-inf"))
    want = torch.einsum("htk,khv->thv", torch.softmax(s, -1), v.to(F64))
    top = torch.full((heads, rows, 1), float("-inf"), dtype=F64, device="cuda")
    den, num = torch.zeros_like(top), torch.zeros(heads, rows, vdim, dtype=F64, device="cuda")
    for a in range(max(0, pos - window + 1) if window else 0, t, 64):
        part = s[..., a: a + 64]
        new = torch.maximum(top, part.amax(-1, keepdim=True))
        ref = new.masked_fill(new == float("-inf"), 0.0)
        p = torch.exp(part - ref)
        den = den * torch.exp(top - ref) + p.sum(-1, keepdim=True)
        num = num * torch.exp(top - ref) + torch.einsum("htk,khv->htv", p.to(BF16).to(F64), v[a: a + 64].to(F64))
        top = new
    rounded = (num / den).to(BF16).to(F64).transpose(0, 1)
    assert float((out.view_as(want).to(F64) - want).norm()) <= 1.001 * float((rounded - want).norm())


@pytest.mark.parametrize("rows,pos,window,ring", [(200, 1189, 30, 600), (129, 700, 1, 300), (300, 2 * 450 - 7, 70, 450), (640, 1000, 129, 801)])
def test_rows_that_no_query_sees(ops, rows, pos, window, ring):
    """Cache rows of positions before the window of the first query change nothing, whatever they hold; tiles that end with the
    ring have keys of other tiles, or such rows, next to them."""
    heads, dim, rot, vdim, rank, t = 3, 64, 32, 64, 64, pos + rows
    gen = torch.Generator(device="cuda").manual_seed(rows)
    mix = types.SimpleNamespace(heads=heads, dim=dim, rot_dim=rot, vdim=vdim, kv_rank=rank, scale=(dim + rot) ** -0.5)
    q, kv = rnd(gen, rows, heads, dim + rot), rnd(gen, ring, heads * (dim + vdim))
    cache = types.SimpleNamespace(rows=rnd(gen, ring, ops.latent_row_len(rank, rot)), ring=ring, window=window)
    unseen = torch.ones(ring, dtype=torch.bool, device="cuda")
    unseen[torch.arange(pos - window + 1, t, device="cuda") % ring] = False
    outs = []
    for other in (0.0, float("nan"), float("inf")):
        kv[unseen], cache.rows[unseen] = other, other
        out = torch.zeros(rows, heads * vdim, dtype=BF16, device="cuda")
        ops.expanded_attn(q, kv, cache, rows, mix, torch.tensor([pos], dtype=I32, device="cuda"), None, None, False, out)
        outs.append(out)
    assert bool(outs[0].isfinite().all()) and torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
