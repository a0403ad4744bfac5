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


@pytest.mark.parametrize("vocab", [3, 1025, 33333, 262144, 262177, 300000])
def test_sampled_token_by_the_restated_rule(ops, vocab):
    """Rows kept in shared memory (up to 262144 values) and read again from memory (beyond) against the f64 restatement: the token that
    the same uniform number falls to, the 256 largest, their log-probabilities.  The sums have f32 exponentials of differences up to
    20 (an error of 2^-20 each, relative) in eight parts: bounds of 1e-4 and 2e-4, as for one part in test_gpu_ops.py."""
    from oracle import ops as oo

    gen = torch.Generator().manual_seed(vocab)
    logits = torch.randn(2, vocab, generator=gen) * 2.5
    logits[1, vocab // 2:] = logits[1, vocab // 2:].round()  # ties, across the CTAs' parts
    tok, lp = torch.zeros(2, dtype=torch.int64, device="cuda"), torch.zeros(2, device="cuda")
    one, top, ids = torch.zeros(2, dtype=torch.int32, device="cuda"), torch.zeros(2, 256, device="cuda"), torch.zeros(2, 256, dtype=torch.int32, device="cuda")
    for cfg, seed in (((0.0, 1.0, 0.0, 0.0), 1), ((1.0, 1.0, 50.0, 0.0), 2), ((0.7, 0.9, 0.0, 1.0), 3), ((1.3, 0.5, 40.0, 1.0), 4), ((1.0, 1.0, 0.0, 0.0), 5)):
        step = torch.tensor([11, 0], device="cuda")
        ops.next_token(logits.cuda(), tok, config=torch.tensor(cfg, device="cuda"), seed=seed, step=step, sampled=one, token_logprob=lp, topn_logprobs=top,
                       topn_indices=ids)
        assert step.tolist() == [12, 0] and one.tolist() == tok.tolist()
        for t in range(2):
            order, bounds, logp = oo.sample_intervals(logits[t], cfg[0], cfg[1], int(cfg[2]), cfg[3] != 0)
            all_ids = torch.argsort(-logits[t].double(), stable=True)[:1024]
            got, u, n = int(tok[t]), oo.sample_uniform(seed, 11, t), min(256, vocab)
            j = int((order == got).nonzero()[0])
            assert j == 0 if cfg[0] == 0.0 else (float(bounds[j - 1]) if j else 0.0) - 1e-4 <= u < float(bounds[j]) + 1e-4
            assert ids[t, :n].tolist() == all_ids[:n].tolist() and bool((ids[t, n:] == -1).all())
            assert float((top[t, :n].cpu().double() - logp[:n]).abs().max()) < 2e-4 and abs(float(lp[t]) - float(logp[(all_ids == got).nonzero()[0]])) < 2e-4
