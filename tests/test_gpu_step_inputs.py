"""What a pass begins with, exact: embedding rows and rotary rows gathered; negative tokens from the end; what lies outside of a table is
refused with status 4 and nothing stored."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [7168, 4104, 250, 7])
@pytest.mark.parametrize("n,pos", [(1, 0), (4, 13), (4, 96)])
def test_gathered_rows(dim, n, pos):
    import tilert_b200 as tb
    from tilert_b200.models.deepseek_v3_2 import ops

    tb.load_backend("deepseek_v3_2")
    tb.tilert_init(0)
    gen = torch.Generator().manual_seed(dim + pos)
    table, freqs = torch.randn(50, dim, generator=gen).to(torch.bfloat16).cuda(), torch.randn(100, 32, 2, generator=gen).cuda()
    toks = torch.randint(-50, 50, (n,), generator=gen).cuda()
    x, fr = torch.zeros(1, n, dim, dtype=torch.bfloat16, device="cuda"), torch.zeros(n, 32, 2, device="cuda")
    cur = torch.tensor([pos], dtype=torch.int32, device="cuda")
    ops.step_inputs(toks, table, cur, freqs, x, fr)
    assert torch.equal(x[0], table[toks]) and torch.equal(fr, freqs[pos: pos + n]) and tb.device_status(0) == 0
    for bad, at in ((50, pos), (-51, pos), (0, 100), (0, -1)):
        x.fill_(7), fr.fill_(7), cur.fill_(at)
        ops.step_inputs(torch.tensor([bad], device="cuda"), table, cur, freqs, x[:, :1].contiguous(), fr[:1].contiguous())
        assert tb.device_status(0) == 4 and bool((x == 7).all()) and bool((fr == 7).all())
