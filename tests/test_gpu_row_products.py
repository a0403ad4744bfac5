"""Products with bf16 weight rows in the forms that the number of rows chooses: tiles of 64 and of 128 features on single SMs, a
pair of SMs on a tile, groups of equal size; the exact mode's two tile shapes; long weights of the FP8 models' head and input
product, a row or four rows a warp.  References are f64 on the same operands.  f32 sums of up to 18432 products in any order:
relative rms error below 1e-5 (the sums of the exact mode, with f32 inputs, below 2e-6); bf16 results a rounding more, 2^-8."""

import pytest
import torch

pytestmark = pytest.mark.gpu

BF16, F32, F64 = torch.bfloat16, torch.float32, torch.float64
ALPHA = 1.702


@pytest.fixture(scope="module")
def ops():
    import tilert_b200 as tb
    from tilert_b200 import gqa_ops

    tb.load_backend("ralasun")
    tb.tilert_init(0, "ralasun")
    yield gqa_ops
    assert tb.device_status(0, "ralasun") == 0


def rnd(seed, *shape, dtype=F32, std=1.0):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * std).to(dtype).cuda()


def padded(t):
    k = t.shape[-1]
    return torch.nn.functional.pad(t, (0, -k % 8)).contiguous()


def close(name, ref, out, lim):
    err = float((out.to(F64) - ref).norm() / ref.norm())
    assert err < lim, f"{name}: {err:.2e}"


def unit(r, n, limit):
    g, u = r[..., :n].clamp(max=limit), r[..., n:].clamp(-limit, limit)
    return g * torch.sigmoid(ALPHA * g) * (u + 1)


@pytest.mark.parametrize("out", [F32, BF16])
@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("rows,n,k", [(1, 1, 256), (2, 3, 257), (37, 130, 1000), (64, 256, 2048), (65, 129, 640), (100, 31, 5632), (128, 2048, 1024),
                                      (129, 70, 4096), (173, 3072, 2048), (37, 5632, 512), (300, 900, 700)])
def test_few_rows(ops, rows, n, k, gated, out):
    x, w = rnd(0, rows, k, dtype=BF16), rnd(1, n * (1 + gated), k, dtype=BF16, std=k ** -0.5)
    o = torch.full((rows + 1, n + 5), 7.0, dtype=out, device="cuda")
    ops.gemm(padded(x), padded(w), o, rows, n, k, gated=(1.5, ALPHA) if gated else None)
    r = x.to(F64) @ w.to(F64).T
    close("product", unit(r, n, 1.5) if gated else r, o[:rows, :n], 1e-5 if out == F32 else 2.0 ** -8)
    assert bool((o[rows] == 7.0).all()) and bool((o[:, n:] == 7.0).all()), "wrote outside its rows"
    if not gated:
        b = rnd(2, n)
        o8 = torch.zeros(rows, n + -n % 4, dtype=out, device="cuda")
        ops.gemm(padded(x), padded(w), o8, rows, n, k, bias=b)
        close("bias", r + b.to(F64), o8[:, :n], 1e-5 if out == F32 else 2.0 ** -8)


@pytest.mark.parametrize("groups,rows,n,k", [(3, 5, 40, 300), (16, 37, 128, 512), (7, 65, 100, 1024), (2, 200, 256, 640)])
def test_few_rows_in_groups_of_equal_size(ops, groups, rows, n, k):
    x, w = rnd(0, groups, rows, k, dtype=BF16), rnd(1, groups, n, k, dtype=BF16, std=k ** -0.5)
    o = torch.zeros(groups * rows, n, device="cuda")
    ops.gemm(padded(x).flatten(0, 1), padded(w), o, rows, n, k, n_groups=groups)
    close("groups", torch.einsum("grk,gnk->grn", x.to(F64), w.to(F64)).flatten(0, 1), o, 1e-5)


@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("rows,n,k", [(1, 1, 1), (5, 33, 130), (31, 32, 128), (33, 65, 1027), (47, 8000, 96), (64, 700, 64), (200, 2048, 300), (1000, 1500, 72)])
def test_exact_mode(ops, rows, n, k, gated):
    x, w = rnd(0, rows, k), rnd(1, n * (1 + gated), k, dtype=BF16, std=k ** -0.5)
    # what lies between k and the end of a row is no operand
    xp = torch.full((rows, k + -k % 8), float("nan"), device="cuda")
    wp = torch.full((w.shape[0], k + -k % 8), float("nan"), dtype=BF16, device="cuda")
    xp[:, :k], wp[:, :k] = x, w
    o = torch.full((rows + 1, n + 3), 7.0, device="cuda")
    ops.gemm(xp, wp, o, rows, n, k, gated=(1.5, ALPHA) if gated else None)
    r = x.to(F64) @ w.to(F64).T
    close("product", unit(r, n, 1.5) if gated else r, o[:rows, :n], 2e-6)
    assert bool((o[rows] == 7.0).all()) and bool((o[:, n:] == 7.0).all()), "wrote outside its rows"


@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("counts", [[3, 0, 5, 1], [70, 64, 0, 130, 33], [1] * 40])
def test_exact_mode_in_groups(ops, counts, gated):
    n, k, total = 90, 200, sum(counts)
    x, w = rnd(0, total, k), rnd(1, len(counts), n * (1 + gated), k, dtype=BF16, std=k ** -0.5)
    o = torch.zeros(total, n, device="cuda")
    ops.gemm(x, w, o, total, n, k, gated=(1.5, ALPHA) if gated else None, n_groups=len(counts), counts=torch.tensor(counts, dtype=torch.int32, device="cuda"))
    r = torch.cat([p.to(F64) @ w[g].to(F64).T for g, p in enumerate(x.split(counts))])
    close("groups", unit(r, n, 1.5) if gated else r, o, 2e-6)


@pytest.mark.parametrize("tokens", [1, 2, 3, 4])
@pytest.mark.parametrize("n,k", [(2049, 256), (4099, 1280), (16160, 7168)])
def test_long_head(ops, tokens, n, k):
    """RMS norm and vocabulary head of the FP8 models: f32 activations."""
    from tilert_b200.models.deepseek_v3_2 import ops as dsa

    x, g, w = rnd(0, 1, tokens, k, dtype=BF16), rnd(1, k), rnd(2, n, k, dtype=BF16, std=k ** -0.5)
    o = torch.zeros(1, tokens, n, device="cuda")
    dsa.rmsnorm_head_proj(x, g, w, None, o, eps=1e-6)
    xd = x.to(F64)
    ref = xd / torch.sqrt((xd * xd).mean(-1, keepdim=True) + 1e-6) * g.to(F64) @ w.to(F64).T
    close("head", ref, o, 1e-5)


@pytest.mark.parametrize("tokens", [1, 2, 3, 4])
@pytest.mark.parametrize("dim", [128, 1024, 7168])
def test_two_segments(ops, tokens, dim):
    """Both halves of the input normalised on their own and rounded to bf16, bf16 result."""
    from tilert_b200.models.deepseek_v3_2 import ops as dsa

    e, h, ge, gh = rnd(0, 1, tokens, dim, dtype=BF16), rnd(1, 1, tokens, dim, dtype=BF16, std=3.0), rnd(2, dim), rnd(3, dim)
    w, o = rnd(4, dim, 2 * dim, dtype=BF16, std=(2 * dim) ** -0.5), torch.zeros(1, tokens, dim, dtype=BF16, device="cuda")
    dsa.mtp_preprocess(e, h, ge, gh, w, o, eps=1e-6)

    def norm(x, g):
        x = x.to(F64)
        return x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-6) * g.to(F64)

    # (the two normalised vectors are bf16 values: 2^-9 each, as the result)
    close("eh_proj", torch.cat([norm(e, ge), norm(h, gh)], -1) @ w.to(F64).T, o, 2.0 ** -8)


def in_order(x, w, piece):
    """The sums of a long product as the kernel takes them, in f32: a lane's pieces of `piece` elements a warp's width apart, each
    summed on its own and added to the lane's sum, then halves of the warp."""
    x, w = x.to(F64), w.to(F64)
    z = lambda v: v.reshape(*v.shape[:-1], -1, 32, piece)
    x, w = z(x)[:, None], z(w)[None]
    acc = torch.zeros(x.shape[0], w.shape[1], 32, device="cuda")
    for s in range(w.shape[2]):
        part = (x[:, :, s, :, 1] * w[:, :, s, :, 1]).to(F32)
        for j in (0, *range(2, piece)):
            part = (x[:, :, s, :, j] * w[:, :, s, :, j] + part.to(F64)).to(F32)  # an fma: the product is exact in f64
        acc += part
    while acc.shape[-1] > 1:
        acc = acc[..., : acc.shape[-1] // 2] + acc[..., acc.shape[-1] // 2:]
    return acc[..., 0]


@pytest.mark.parametrize("tokens", [1, 2, 3, 4])
@pytest.mark.parametrize("n,k,dtype", [(2050, 256, BF16), (2053, 1280, BF16), (2368, 1280, F32), (33, 8448, F32), (2369, 768, F32), (4099, 256, BF16)])
def test_order_of_long_sums(tokens, n, k, dtype):
    """However many rows a warp works on, a sum has the bits of a row at a time: a choice between near ties may hang on them."""
    from tilert_b200.models.deepseek_v3_2 import ops as dsa

    x, w = rnd(0, 1, tokens, k, dtype=BF16), rnd(1, n, k, dtype=dtype, std=k ** -0.5)
    o = torch.zeros(1, tokens, n, device="cuda")
    dsa.rmsnorm_expert_proj(x, None, w, o, None, eps=1e-6)
    assert torch.equal(o[0], in_order(x[0], w, 8 if dtype == BF16 else 4))


@pytest.mark.parametrize("dim,rows", [(128, 128), (1024, 5), (4096, 2400)])
def test_gains_off_their_boundary(dim, rows):
    """Gains at any address: the general form of the loads gives the same bits."""
    from tilert_b200.models.deepseek_v3_2 import ops as dsa

    e, h, w = rnd(0, 1, 3, dim, dtype=BF16), rnd(1, 1, 3, dim, dtype=BF16), rnd(2, dim, 2 * dim, dtype=BF16)
    g, outs = (rnd(3, dim + 4), rnd(4, dim + 4)), []
    for at_e, at_h in ((0, 0), (1, 0), (0, 3), (2, 1)):
        ge, gh = (torch.empty(dim + 4, device="cuda")[at: at + dim].copy_(v[:dim]) for v, at in zip(g, (at_e, at_h)))
        o = torch.zeros(1, 3, dim, dtype=BF16, device="cuda")
        dsa.mtp_preprocess_rows(e, h, ge, gh, w, o, 0, rows)
        outs.append(o)
    assert all(torch.equal(outs[0], o) for o in outs[1:]) and bool(outs[0].any())


@pytest.mark.parametrize("tokens", [1, 4])
def test_few_long_rows(tokens):
    """A rank's row share of an input product, fewer rows than the GPU has warps: no walk of a warp over four rows, which takes as
    long as four times the SMs' warps in rows do.  (Measured: two thirds of the whole product's time, was nine tenths.)"""
    from tilert_b200.models.deepseek_v3_2 import ops as dsa

    dim = 7168
    e, h, ge, gh = rnd(0, 1, tokens, dim, dtype=BF16), rnd(1, 1, tokens, dim, dtype=BF16), rnd(2, dim), rnd(3, dim)
    w, o = torch.zeros(dim, 2 * dim, dtype=BF16, device="cuda"), torch.zeros(1, tokens, dim, dtype=BF16, device="cuda")

    def us(rows):
        def call():
            dsa.mtp_preprocess_rows(e, h, ge, gh, w, o, 0, rows)

        call()
        torch.cuda.synchronize()
        graph, (begin, end) = torch.cuda.CUDAGraph(), (torch.cuda.Event(enable_timing=True) for _ in range(2))
        with torch.cuda.graph(graph):  # (launched one by one they may wait for the host)
            for _ in range(40):
                call()
        graph.replay()
        begin.record()
        graph.replay()
        end.record()
        torch.cuda.synchronize()
        return begin.elapsed_time(end)

    assert min(us(512) for _ in range(3)) < 0.8 * min(us(dim) for _ in range(3))
