"""Attention of a portion on mma.sync tiles where its copies and addresses can go wrong: sizes with constant addresses (128 / 128,
64 / 64) and without, rows of pieces that are no power of two, tiles that cross the ring's end or the last key, windows that
begin inside a tile.  Against the plain 64-bit result; the bound is that of test_gpu_ralasun_ops.py for bf16."""

import pytest
import torch

from test_gpu_ralasun_ops import Attn, close, mix_of, ops  # noqa: F401  (ops: the fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(8, 2, 128, 128, None), (8, 2, 128, 128, 97), (16, 1, 128, 128, 64), (6, 6, 64, 64, 70), (4, 1, 64, 64, None),
                                   (9, 3, 80, 72, 61), (3, 1, 264, 120, 50), (5, 1, 128, 64, 33)])
def test_tiles_against_the_plain_result(ops, shape):  # noqa: F811
    mix, t = mix_of(*shape), 330
    a = Attn(ops, mix, torch.bfloat16, t, portion=129)
    lo = 0
    for n in (129, 1, 64, 63, 65, 8):
        out, _ = a.rows(lo, lo + n)
        close(f"portion at {lo}", a.ref[lo: lo + n], out, torch.bfloat16, exact=3e-6, half=1e-2)
        lo += n
