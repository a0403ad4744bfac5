"""The launch that ends a step: arg-max and sampled token as a 64-bit number, the position moved on.  Exact: the largest value's
index, the lowest of equal ones; a value that is no number before all others (as torch has it)."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=["deepseek_v3_2", "ralasun"])
def ops(request):
    import tilert_b200 as tb

    tb.load_backend(request.param)
    tb.tilert_init(0, request.param)
    if request.param == "ralasun":
        from tilert_b200 import gqa_ops as ops
    else:
        from tilert_b200.models.deepseek_v3_2 import ops
    yield ops
    assert tb.device_status(0, request.param) == 0


@pytest.mark.parametrize("kind", ["plain", "ties", "equal", "nan", "low"])
@pytest.mark.parametrize("vocab", [1, 5, 31, 4095, 4096, 16160, 33333, 129280])
def test_arg_max(ops, vocab, kind):
    gen = torch.Generator().manual_seed(vocab)
    logits = torch.randn(3, vocab, generator=gen)
    if kind == "ties":
        logits = logits.round()
    elif kind == "equal":
        logits = torch.zeros(3, vocab) * torch.tensor([1.0, -1.0, 1.0])[:, None]  # a zero of either sign
    elif kind == "nan":
        logits[:, vocab // 2:] = float("nan")
        logits[:, 0] = float("inf")
    elif kind == "low":
        logits = torch.full((3, vocab), float("-inf"))
        logits[1, -1] = torch.finfo(torch.float32).min
    tok, pos = torch.full((3,), -7, device="cuda"), torch.tensor([11], dtype=torch.int32, device="cuda")
    ops.next_token(logits.cuda(), tok, pos=pos, advance=5)
    assert tok.cpu().tolist() == [int(torch.argmax(row)) for row in logits] and int(pos) == 16


@pytest.mark.parametrize("vocab", [3, 1025, 33333, 300000])
def test_sampled_token_as_the_sampler_draws_it(ops, vocab):
    gen = torch.Generator().manual_seed(vocab)
    logits = torch.randn(2, vocab, generator=gen).cuda()
    config = torch.tensor([0.8, 0.9, 0.0, 1.0], device="cuda")
    tok, one = torch.zeros(2, dtype=torch.int64, device="cuda"), torch.zeros(2, dtype=torch.int32, device="cuda")
    step, pos, seen = torch.zeros(2, dtype=torch.int64, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda"), []
    for i in range(6):
        ops.next_token(logits, tok, pos=pos, advance=1, config=config, seed=5, step=step, sampled=one)
        assert tok.tolist() == one.tolist()
        again = torch.zeros_like(one)
        ops.sample(logits, config, again, seed=5, step_value=i)
        assert again.tolist() == one.tolist()
        seen.append(one.tolist())
    assert int(pos) == 6 and step.tolist() == [6, 0] and (vocab == 3 or len({tuple(s) for s in seen}) > 1)


@pytest.mark.parametrize("fill", [0.0, float("nan")])
def test_rows_of_one_value(ops, fill):
    """More equal values than candidates: the lowest indices; of values that are no number no more either."""
    logits = torch.full((1, 40000), fill, device="cuda")
    tok = torch.zeros(1, dtype=torch.int32, device="cuda")
    top, ids = torch.zeros(1, 256, device="cuda"), torch.zeros(1, 256, dtype=torch.int32, device="cuda")
    ops.sample(logits, torch.tensor([0.0, 1.0, 0.0, 0.0], device="cuda"), tok, topn_logprobs=top, topn_indices=ids)
    assert ids[0].tolist() == list(range(256)) and int(tok) == 0
