"""The 256 largest of a row that the sampler exports: rows on and off 16-byte boundaries, ties, infinities, fewer eligible
values than are asked for.  Exact: equal values in the order of their indices."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    import tilert_b200 as tb
    from tilert_b200 import gqa_ops

    tb.load_backend("ralasun")
    tb.tilert_init(0, "ralasun")
    yield gqa_ops
    assert tb.device_status(0, "ralasun") == 0


@pytest.mark.parametrize("kind", ["plain", "ties", "few", "equal"])
@pytest.mark.parametrize("vocab", [5, 1023, 1024, 1025, 4099, 16160, 33333])
def test_largest_values_in_order(ops, vocab, kind):
    gen = torch.Generator().manual_seed(vocab)
    logits = torch.randn(3, vocab, generator=gen) * 3  # rows 1 and 2 off the boundary unless vocab is a multiple of four
    if kind == "ties":
        logits = logits.round()
    elif kind == "few":
        logits[torch.rand(3, vocab, generator=gen) < 0.97] = float("-inf")
        logits[:, 0] = 0.0
    elif kind == "equal":
        logits = torch.zeros(3, vocab)
    tok, lp = torch.zeros(3, dtype=torch.int32, device="cuda"), torch.zeros(3, device="cuda")
    top, ids = torch.zeros(3, 256, device="cuda"), torch.zeros(3, 256, dtype=torch.int32, device="cuda")
    ops.sample(logits.cuda(), torch.tensor([0.0, 1.0, 0.0, 0.0], device="cuda"), tok, token_logprob=lp, topn_logprobs=top, topn_indices=ids)
    for r in range(3):
        order = torch.sort(logits[r], descending=True, stable=True)[1]
        order = order[torch.isfinite(logits[r][order])][:256]
        want = torch.full((256,), -1)
        want[: order.numel()] = order
        assert ids[r].cpu().tolist() == want.tolist() and int(tok[r]) == int(order[0])
