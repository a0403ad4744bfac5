"""Products of many rows on pairs of SMs, and of few rows on single ones, against f64 on the same bf16 operands, at the edges of their tiles.

The tensor cores add sixteen products at a time to an f32 sum and may cut off what does not fit: up to 2^-23 of the sum (of
size 8 at most here) in each of k / 16 steps, and a few more such roundings in the bias or the gated unit.  A bf16 result adds
2^-9 of its value."""

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


def padded(ops, gen, rows, k, std):
    t = torch.zeros(rows, ops.pad(k), dtype=BF16, device="cuda")
    t[:, :k] = torch.randn(rows, k, generator=gen, device="cuda") * std
    return t


def check(ops, n, k, gated, out_type, counts, rows=None):
    gen = torch.Generator(device="cuda").manual_seed(n * 31 + k)
    total = rows or sum(counts)
    groups = 0 if counts is None else len(counts)
    x = padded(ops, gen, total, k, 1.0)
    w = padded(ops, gen, max(groups, 1) * (2 if gated else 1) * n, k, 1.5 * k ** -0.5)
    bias = None if groups or gated else torch.randn(n, generator=gen, device="cuda")
    out = torch.full((total + 3, ops.pad(n)), 77.0, dtype=out_type, device="cuda")
    ops.gemm(x, w, out, total, n, k, gated=(1.5, 1.702) if gated else None, n_groups=groups,
             counts=None if counts is None else torch.tensor(counts, dtype=I32, device="cuda"), bias=bias)
    bound = (k / 16 + 8) * 2.0 ** -23 * 8
    ws = w.to(F64).view(max(groups, 1), 2 if gated else 1, n, -1)
    lo = 0
    for g, c in enumerate(counts or [total]):
        z = torch.einsum("tk,hnk->htn", x[lo: lo + c].to(F64), ws[g])
        if gated:
            a, u = z[0].clamp(max=1.5), z[1].clamp(-1.5, 1.5)
            want = a * torch.sigmoid(1.702 * a) * (u + 1)
        else:
            want = z[0] + (0 if bias is None else bias.to(F64))
        off = (out[lo: lo + c, :n].to(F64) - want).abs()
        assert float((off - (2.0 ** -8 * want.abs() if out_type == BF16 else 0)).max() if c else 0) <= bound, (g, c)
        lo += c
    assert bool((out[total:] == 77).all()) and bool((out[:, n:] == 77).all())  # nothing beyond the rows and features


@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("out_type", [BF16, F32])
@pytest.mark.parametrize("n,k", [(7, 8), (129, 72), (136, 64), (258, 200), (512, 136)])
@pytest.mark.parametrize("counts", [[0, 1, 300], [64, 64, 65, 63], [257, 512, 0, 255, 1]])
def test_groups(ops, gated, out_type, n, k, counts):
    check(ops, n, k, gated, out_type, counts)


@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("n,k", [(7, 8), (65, 72), (136, 200), (20000, 64)])
@pytest.mark.parametrize("counts", [[1, 0, 2, 0], [63, 64, 0, 65, 1], [40] * 7])
def test_few_rows_a_group(ops, gated, n, k, counts):
    check(ops, n, k, gated, BF16, counts)


@pytest.mark.parametrize("rows,n,k,gated,out_type", [
    (1, 64, 200, False, F32), (37, 2048, 1032, False, F32), (64, 65, 64, False, BF16), (65, 12000, 136, False, BF16), (173, 129, 72, True, BF16),
    (2048, 700, 2000, False, F32), (2047, 1288, 1000, True, BF16), (1357, 4104, 520, False, BF16), (1025, 2049, 1032, True, BF16),
    (700, 3000, 2000, False, F32), (37, 5632, 1024, True, BF16), (257, 20001, 72, False, F32)])
def test_one_weight(ops, rows, n, k, gated, out_type):
    check(ops, n, k, gated, out_type, None, rows)


@pytest.mark.parametrize("out_type", [BF16, F32])
@pytest.mark.parametrize("rows,n,k", [  # tiles of 64 features: 32 rows (the last two: 64), stages of four blocks of K, the last one short
    (1, 7, 8), (31, 65, 64), (32, 64, 256), (33, 200, 264), (97, 130, 448), (37, 2048, 1032), (300, 64, 3000), (150, 2048, 200), (173, 3000, 330)])
def test_small_tiles(ops, rows, n, k, out_type):
    check(ops, n, k, False, out_type, None, rows)


@pytest.mark.parametrize("out_type", [BF16, F32])
@pytest.mark.parametrize("gated", [False, True])
def test_forms_have_the_same_bits(ops, gated, out_type):
    """A row's result does not depend on the tile it is in (64 or 128 features on one SM, 256 on a pair with 64 to 256 rows, one or
    two blocks of K a stage): a choice of experts behind a product may hang on a last bit.  The sizes make the rule choose each on
    148 SMs; without groups gated products are always a pair's."""
    n, k = (1500, 520) if gated else (2048, 1032)
    sizes = [1, 400, 600, 800, 1000, 1200, 1400, 1440] if gated else [1, 37, 300, 600, 900, 1200, 1500, 1800, 2048]
    gen = torch.Generator(device="cuda").manual_seed(n)
    x, w = padded(ops, gen, sizes[-1], k, 1.0), padded(ops, gen, (1 + gated) * n, k, 1.5 * k ** -0.5)

    def product(rows, groups=0, counts=None):
        out = torch.zeros(rows, ops.pad(n), dtype=out_type, device="cuda")
        ops.gemm(x, w if not groups else w.repeat(groups, 1), out, rows, n, k, gated=(1.5, 1.702) if gated else None, n_groups=groups,
                 counts=None if counts is None else torch.tensor(counts, dtype=I32, device="cuda"))
        return out

    whole = product(sizes[-1])
    for rows in sizes[:-1]:
        assert torch.equal(product(rows), whole[:rows]), rows
    for counts in ([37, 0, 60], [40] * 13, [64] * 4, [100, 200, 130], [300, 256, 1]):  # 64 features, 128, pairs of 96, 192, 224 rows
        assert torch.equal(product(sum(counts), len(counts), counts), whole[: sum(counts)]), counts


@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("counts", [[260, 0, 513, 33, 256, 100], [80, 70, 129, 64, 200, 5], [288, 287, 289, 1]])
@pytest.mark.parametrize("n,k", [(300, 200), (640, 72)])
def test_short_last_tiles_of_groups(ops, n, k, counts, gated):
    check(ops, n, k, gated, BF16, counts)


@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("n,k", [(7, 8), (130, 264)])
@pytest.mark.parametrize("counts", [[0] * 20 + [33] + [0] * 19, [1, 0, 1] * 7, [0, 64] + [0] * 70])
def test_fewer_rows_than_groups(ops, n, k, counts, gated):
    """Tiles of 32 rows, of which a group may need two."""
    rows = sum(counts)
    assert ops.gemm_tile(rows, n, k, gated=gated, n_groups=len(counts), counted=True)[1:] == (64, 32)
    check(ops, n, k, gated, BF16, counts)
