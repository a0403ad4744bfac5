"""Routing where scores are no numbers or minus infinity: the ids address weights, so they are top_k distinct experts always, in the
order of a stable descending sort (what is no number first, of equal ones the lowest).  Exact; through the gate/up operator on weights of
zero, with the routing inside the product (one token) and in a launch of its own."""

import pytest
import torch

from oracle import ops as oo

pytestmark = pytest.mark.gpu
BF16, F32, I32 = torch.bfloat16, torch.float32, torch.int32
NAN, INF = float("nan"), float("inf")


@pytest.mark.parametrize("kind", ["nan_some", "nan_all", "nan_bias", "low_bias", "low_all"])
@pytest.mark.parametrize("tokens", [1, 3])
@pytest.mark.parametrize("experts,top,groups,limited", [(256, 8, 8, 4), (256, 8, 1, 1), (64, 8, 1, 1), (37, 31, 1, 1), (5, 5, 1, 1)])
def test_ids_are_experts(experts, top, groups, limited, tokens, kind):
    import tilert_b200 as tb
    from tilert_b200.models.deepseek_v3_2 import ops

    tb.load_backend("deepseek_v3_2")
    tb.tilert_init(0)
    gen = torch.Generator().manual_seed(experts + tokens)
    scores, bias, dim, inter = torch.randn(1, tokens, experts, generator=gen), torch.randn(experts, generator=gen) * 0.1, 256, 64
    if kind == "nan_some":
        scores[:, -1, 1::3] = NAN
    elif kind == "nan_all":
        scores[:] = NAN
    elif kind == "nan_bias":
        bias[experts // 2] = NAN
    elif kind == "low_bias":
        bias[3:] = -INF
    else:
        bias[:] = -INF
    w = torch.zeros(experts + 1, 1, dim // 128, 16448, dtype=torch.uint8, device="cuda")
    x, hid = torch.zeros(1, tokens, dim, dtype=BF16, device="cuda"), torch.zeros(1, tokens, top + 1, inter, dtype=BF16, device="cuda")
    probs, ids = torch.zeros(1, tokens, top, device="cuda"), torch.full((1, tokens, top), -7, dtype=I32, device="cuda")
    ops.expert_select_up_gate_silu(x, scores.cuda(), bias.cuda(), w, hid, probs, ids, dim=dim, n_groups=groups, n_limited_groups=limited, route_scale=2.5)
    rp, ri = oo.expert_select_ds(scores, bias, groups, limited, top, 2.5)
    assert torch.equal(ids.cpu(), ri.to(I32)) and tb.device_status(0) == 0
    assert torch.equal(probs.cpu().isnan(), rp.isnan()) and torch.allclose(probs.cpu(), rp, rtol=1e-5, atol=0, equal_nan=True)
    if experts == 5:  # more than there are: refused on the host
        with pytest.raises(tb.TilertError):
            ops.expert_select_up_gate_silu(x, scores.cuda(), bias.cuda(), w, torch.zeros(1, tokens, 7, inter, dtype=BF16, device="cuda"),
                                           torch.zeros(1, tokens, 6, device="cuda"), torch.zeros(1, tokens, 6, dtype=I32, device="cuda"), dim=dim, n_groups=1,
                                           n_limited_groups=1, route_scale=2.5)
