"""Products of the exact mode at the edges of their tiles and steps: a last step of K of one to 127 elements that ends inside a piece of
16 bytes, rows and features around 32 and 64, groups of no row, one, 31 to 33 and 70 rows.  What lies beyond K in the operands' padding
is no number here and must not be read as one.  f64 on the same operands; k f32 products in any order: relative rms error below 2e-6."""

import pytest
import torch

pytestmark = pytest.mark.gpu
F32, F64, BF16 = torch.float32, torch.float64, torch.bfloat16


@pytest.fixture(scope="module")
def ops():
    import tilert_b200 as tb
    from tilert_b200 import gqa_ops

    tb.load_backend("ralasun")
    tb.tilert_init(0, "ralasun")
    yield gqa_ops
    assert tb.device_status(0, "ralasun") == 0


@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("k", [1, 7, 64, 129, 255, 259, 1000])
@pytest.mark.parametrize("rows,n,counts", [(1, 1, None), (31, 33, None), (33, 65, None), (200, 1300, None), (137, 70, [0, 1, 31, 33, 32, 70 - 30]),
                                           (640, 700, [70, 0, 300, 270])])
def test_edges(ops, rows, n, counts, k, gated):
    gen = torch.Generator(device="cuda").manual_seed(rows * 7 + k)
    groups, kp = 0 if counts is None else len(counts), ops.pad(k)
    assert counts is None or sum(counts) == rows
    x = torch.full((rows, kp), float("nan"), device="cuda")
    x[:, :k] = torch.randn(rows, k, generator=gen, device="cuda")
    w = torch.full((max(groups, 1), 2 if gated else 1, n, kp), float("nan"), dtype=BF16, device="cuda")
    w[..., :k] = torch.randn(*w.shape[:3], k, generator=gen, device="cuda") * k ** -0.5
    out = torch.full((rows + 1, n + 3), 7.0, device="cuda")
    bias = torch.randn(n, generator=gen, device="cuda") if counts is None and not gated else None
    ops.gemm(x, w, out, rows, n, k, gated=(1.5, 1.702) if gated else None, n_groups=groups, bias=bias,
             counts=None if counts is None else torch.tensor(counts, dtype=torch.int32, device="cuda"))
    want, lo = [], 0
    for g, c in enumerate(counts or [rows]):
        z = torch.einsum("tk,hnk->htn", x[lo: lo + c, :k].to(F64), w[g, ..., :k].to(F64))
        if gated:
            a, u = z[0].clamp(max=1.5), z[1].clamp(-1.5, 1.5)
            want.append(a * torch.sigmoid(1.702 * a) * (u + 1))
        else:
            want.append(z[0] + (0 if bias is None else bias.to(F64)))
        lo += c
    want = torch.cat(want)
    assert float((out[:rows, :n].to(F64) - want).norm() / want.norm()) < 2e-6
    assert bool((out[rows] == 7).all()) and bool((out[:, n:] == 7).all())
