"""The small router's ranking against the chunked kernel's."""

import pytest
import torch

from uma_qmoe_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("experts,top_k", [(64, 8), (60, 4), (9, 8), (33, 1)])
def test_small_router_ranks_as_the_chunked_one(experts, top_k):
    """Ties (equal rows of the router matrix) go to the lower expert and the weights have the same bits, one to nine tokens;
    a NaN logit leaves its token without an expert and the others as they are."""
    gen = torch.Generator(device=DEV).manual_seed(experts)
    x = torch.randn(2500, 2048, device=DEV, generator=gen).to(torch.bfloat16)
    weight = (torch.randn(experts, 2048, device=DEV, generator=gen) * 0.05).to(torch.bfloat16)
    weight[experts // 2] = weight[1]
    weight[experts - 1] = weight[0]
    for renormalize in (False, True):
        w, idx, logits = ops.route_topk(x, weight, top_k, renormalize, return_logits=True)
        for tokens in (1, 2, 5, 9, 150):
            got = ops.route_topk(x[:tokens], weight, top_k, renormalize, return_logits=True)
            same = (got[2] == logits[:tokens]).all(dim=1)              # sums of other runs: a BF16 ulp in 10^4 logits
            assert same.float().mean() > 0.9 if tokens > 100 else same.any() or tokens < 5
            assert torch.equal(got[1][same], idx[:tokens][same]) and torch.equal(got[0][same], w[:tokens][same])
    dirty = x[:6].clone()
    dirty[4, 7] = float("nan")
    clean, (w, idx) = ops.route_topk(x[:6], weight, top_k, False), ops.route_topk(dirty, weight, top_k, False)
    keep = torch.tensor([0, 1, 2, 3, 5], device=DEV)
    assert torch.equal(idx[keep], clean[1][keep]) and torch.equal(w[keep], clean[0][keep])
    assert (idx[4] == 0x7fffffff).all() and (w[4] == -1).all()
