"""The row kernels that work in pieces of eight elements against the same operators an element at a time: one operand
moved off its 16-byte boundary takes the general form.  Both compute in f32 and, but for layer norms, in the same order: equal
bits.  A layer norm's sums over at most 8192 values are taken in another order (relative error below 1e-6 of a statistic): f32
results agree to 4e-6 of their value and of their row's rms, bf16 ones to a unit in the last place more."""

import types

import pytest
import torch

pytestmark = pytest.mark.gpu

BF16, F32, I32, I64 = torch.bfloat16, torch.float32, torch.int32, torch.int64
TYPES = [F32, BF16]


@pytest.fixture(scope="module")
def ops():
    import tilert_b200 as tb
    from tilert_b200 import gqa_ops

    tb.load_backend("ralasun")
    tb.tilert_init(0, "ralasun")
    yield gqa_ops
    assert tb.device_status(0, "ralasun") == 0


def rnd(seed, *shape, std=1.0, mean=0.0, dtype=F32):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * std + mean).to(dtype).cuda()


def moved(t):
    """The same values one element off a 16-byte boundary, with the same strides."""
    buf = torch.zeros(t.numel() + 8, dtype=t.dtype, device=t.device)
    v = buf[1: 1 + t.numel()].view(t.shape)
    v.copy_(t)
    return v


def same(name, a, b):
    lim = 2.0 ** -7 if a.dtype == BF16 else 4e-6
    a, b = a.double(), b.double()
    off = (a - b).abs() - lim * b.abs() - 4e-6 * b.square().mean(-1, keepdim=True).sqrt()
    assert float(off.max()) <= 0, name


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("dim", [8, 256, 2048, 2056, 4096, 4104, 8192])
def test_residual_and_embedding(ops, dtype, dim):
    rows, top = 5, 3
    y, add, x0 = rnd(0, rows, dim, mean=3.0), rnd(1, dim), rnd(2, rows, dim)
    n1, n2 = (ops.Norm(rnd(s, dim), rnd(s + 1, dim), centered=True) for s in (3, 5))
    gain = rnd(7, dim)
    ye, ysh = rnd(8, rows * top, dim, dtype=dtype), rnd(9, rows, dim, dtype=dtype)
    slot = torch.randperm(rows * top, generator=torch.Generator().manual_seed(1)).to(I32).view(rows, top).cuda()
    w = rnd(10, rows, top)
    forms = [dict(norm=n1, y=y, add=add, norm2=n2), dict(norm=n1, y=y), dict(norm=None, add=add, norm2=n2),
             dict(norm=gain, experts=ye, slot_row=slot, slot_w=w, shared=ysh), dict(norm=gain, experts=ye, slot_row=slot, slot_w=w)]
    for i, f in enumerate(forms):
        out = []
        for general in (False, True):
            x, xh = x0.clone(), torch.zeros(rows, dim, dtype=dtype, device="cuda")
            if general:
                x = moved(x)
            ops.residual_norm(x, None if i == 1 and dtype == F32 else xh, eps=1e-5, dim=dim, rows=rows, **f)
            out.append((x.clone(), xh))
        if "norm2" in f or i == 1:  # layer norms
            same(f"x of form {i}", out[0][0], out[1][0])
            same(f"xh of form {i}", out[0][1], out[1][1])
        else:
            assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1]), i
    table, toks = rnd(11, 9, dim, dtype=BF16), torch.tensor([8, 0, 3], device="cuda")
    for g in (gain, None):
        out = []
        for general in (False, True):
            x, xh = torch.zeros(3, dim, device="cuda"), torch.zeros(3, dim, dtype=dtype, device="cuda")
            ops.embed_norm(toks, table, g, 1e-5, dim, moved(x) if general else x, xh)
            out.append(xh)
            if not general:
                assert torch.equal(x.to(dtype), xh)
        assert torch.equal(*out)


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(3, 1, 8, 24), (8, 2, 96, 64), (16, 16, 128, 128), (64, 8, 128, 256)])
def test_queries_keys_values(ops, dtype, heads, kv_heads, dim, vdim):
    rows, ring, pos = 7, 16, 12
    mix = types.SimpleNamespace(heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim)
    qkv, qg, kg = rnd(0, rows, heads * dim + kv_heads * (dim + vdim)), rnd(1, heads * dim), rnd(2, kv_heads * dim)
    lam, first, cur = torch.tensor([0.3], device="cuda"), rnd(3, rows, kv_heads * vdim), torch.tensor([pos], dtype=I32, device="cuda")
    for mode in (ops.VMIX_NONE, ops.VMIX_FIRST, ops.VMIX_BLEND):
        out = []
        for general in (False, True):
            vf = torch.zeros_like(first) if mode == ops.VMIX_FIRST else first
            cache = types.SimpleNamespace(k=torch.zeros(kv_heads, ring, ops.pad(dim, 16), dtype=dtype, device="cuda"),
                                          v=torch.zeros(kv_heads, ring, ops.pad(vdim, 16), dtype=dtype, device="cuda"), ring=ring)
            q = torch.zeros(rows, heads, ops.pad(dim, 16), dtype=dtype, device="cuda")
            ops.qkv_rows(qkv, moved(qg) if general else qg, kg, 1e-5, mode, lam, vf, rows, mix, cache, cur, q)
            out.append((q, cache.k, cache.v, vf.to(dtype)))
        for name, a, b in zip(("q", "k", "v", "first"), *out):
            assert torch.equal(a, b), f"{name}, mode {mode}"


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("dim", [8, 1992, 2048, 2816, 4096, 7168, 8192])
def test_rms_forms_have_the_same_bits(ops, dtype, dim):
    """An expert is chosen behind these norms: the form a row takes may not decide a near tie."""
    rows, top = 19, 6
    gain, gain2, x0, y = rnd(0, dim), rnd(1, dim), rnd(2, rows, dim), rnd(3, rows, dim)
    ye, ysh = rnd(4, rows * top, dim, dtype=dtype), rnd(5, rows, dim, dtype=dtype)
    slot = torch.randperm(rows * top, generator=torch.Generator().manual_seed(1)).to(I32).view(rows, top).cuda()
    w = rnd(6, rows, top).softmax(-1)
    for f in (dict(norm=gain, y=y), dict(norm=gain, y=y, norm2=gain2), dict(norm=gain, experts=ye, slot_row=slot, slot_w=w, shared=ysh)):
        got = []
        for x in (x0.clone(), moved(x0)):
            xh = torch.zeros(rows, dim, dtype=dtype, device="cuda")
            ops.residual_norm(x, xh, eps=1e-6, dim=dim, rows=rows, **f)
            got.append((x, xh))
        assert all(torch.equal(a, b) for a, b in zip(*got)), list(f)
    table, toks = rnd(7, 50, dim, dtype=BF16), torch.arange(rows, device="cuda") * 2
    got = []
    for x in (torch.zeros(rows, dim, device="cuda"), moved(torch.zeros(rows, dim, device="cuda"))):
        ops.embed_norm(toks, table, gain, 1e-6, dim, x)
        got.append(x)
    assert torch.equal(*got)


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("interleaved", [False, True])
@pytest.mark.parametrize("heads,dim,rot,rank,q_rank", [(1, 8, 16, 8, 8), (5, 96, 32, 72, 304), (16, 128, 64, 512, 1536), (3, 40, 128, 1024, 24)])
def test_latents_and_queries(ops, dtype, interleaved, heads, dim, rot, rank, q_rank):
    rows, ring, pos = 6, 9, 40
    mix = types.SimpleNamespace(heads=heads, dim=dim, rot_dim=rot, vdim=64, kv_rank=rank)
    rope = ops.Rotation(ops.rotation_table(1e4, rot, 64, "cuda"), interleaved)
    cur, ldh = torch.tensor([pos], dtype=I32, device="cuda"), dim + rot
    z, qg, cg = rnd(0, rows, q_rank + rank + rot), rnd(1, q_rank), rnd(2, rank)
    q = rnd(3, rows, heads * ldh)
    out = []
    for general in (False, True):
        cache = types.SimpleNamespace(rows=torch.zeros(ring, ops.latent_row_len(rank, rot), dtype=dtype, device="cuda"), ring=ring)
        cq = torch.zeros(rows, q_rank, dtype=dtype, device="cuda")
        ops.latent_tokens(z, q_rank, q_rank + rank, q_rank, moved(qg) if general else qg, cg, 1e-5, rows, mix, rope, cache, cur, cq)
        src = moved(q) if general else q
        wide = torch.zeros(rows, heads, ops.pad(dim, 16) + ops.pad(rot, 16), dtype=dtype, device="cuda")
        ops.latent_queries(src, rows, mix, rope, cur, wide)
        qn, lat = torch.zeros(heads, rows, dim, dtype=dtype, device="cuda"), torch.zeros(heads, rows, ops.latent_row_len(rank, rot), device="cuda")
        ops.latent_queries(src, rows, mix, rope, cur, qn, lat)
        out.append((cache.rows, cq, wide, qn, lat))
    for name, a, b in zip(("cache", "cq", "expanded", "absorbed", "rotated"), *out):
        assert torch.equal(a, b), name
