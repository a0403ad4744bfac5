"""What a pass begins with, exact: embedding rows and rotary rows gathered; negative tokens from the end; what lies outside of a table is
refused with status 4 and gives rows that are no number, so that a model's logits say so; the drivers refuse what the host knows."""

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
        ops.step_inputs(torch.tensor([bad], device="cuda"), table, cur, freqs, x[:, :1], fr[:1])
        assert tb.device_status(0) == 4 and bool(x[0, 0].isnan().all()) and bool(fr[0].isnan().all())
        assert bool((x[0, 1:] == 7).all()) and bool((fr[1:] == 7).all())


def toy(kind, **kw):
    from oracle import model as om
    from tilert_b200.models.deepseek_v3_2.model import DsaModel
    from tilert_b200.models.deepseek_v3_2.model_args import toy_model_args
    from tilert_b200.models.deepseek_v3_2.mtp import MtpDsaModel

    a = om.toy_args()
    sd = om.random_state_dict(a, seed=0, with_mtp=kind == "mtp")
    return a.vocab_size, (MtpDsaModel if kind == "mtp" else DsaModel)(toy_model_args(), sd, "cuda", cache_len=256, **kw)


@pytest.mark.parametrize("use_graph", [False, True])
def test_a_model_does_not_run_on_a_token_that_is_none(use_graph):
    import tilert_b200 as tb

    vocab, model = toy("plain", use_graph=use_graph)
    for bad in (vocab, -vocab - 1, torch.tensor([vocab]), 1 << 40):
        with pytest.raises(ValueError):
            model.forward(bad, 0)
    with pytest.raises(ValueError):
        model.generate([1, 2, vocab], 1)
    model.reset_sequence()
    model.forward(-1, 0)
    assert bool(model.logits.isfinite().all()) and tb.device_status(0) == 0
    model.forward(torch.tensor([vocab], device="cuda"), 1)
    assert bool(model.logits.isnan().all()) and tb.device_status(0) == 4
    model.reset_sequence()
    model.forward(vocab - 1, 0)  # the sequence after it is not touched
    assert bool(model.logits.isfinite().all()) and tb.device_status(0) == 0


def test_speculative_steps_do_not_run_on_a_token_that_is_none():
    import tilert_b200 as tb

    vocab, model = toy("mtp", use_graph=False)
    for bad in ([1, 2, 3, vocab], torch.tensor([-vocab - 1, 2, 3, 4])):
        with pytest.raises(ValueError):
            model.forward(bad)
    model.set_prefill_mtp_extra_token(vocab)
    model.set_prefill_valid_tokens(4)
    with pytest.raises(ValueError):
        model.forward([1, 2, 3, 4])
    model.set_prefill_valid_tokens(0)
    model.forward([1, 2, 3, -1])  # (the token behind a chunk is read by chunks alone)
    assert bool(model.logits.isfinite().all()) and tb.device_status(0) == 0
    model.reset_sequence()
    model.forward(torch.tensor([1, 2, vocab, 3], device="cuda"))
    assert bool(model.logits[0, 2].isnan().all()) and bool(model.logits[0, :2].isfinite().all()) and tb.device_status(0) == 4
    model.reset_sequence()
    model.forward([1, 2, 3, 4])
    assert bool(model.logits.isfinite().all()) and tb.device_status(0) == 0
    model.set_cur_pos(model.freqs.shape[0] - 3)  # the caches may be longer than the rotary table
    model.cache_len = model.freqs.shape[0] + 100
    with pytest.raises(ValueError):
        model.forward([1, 2, 3, 4])
