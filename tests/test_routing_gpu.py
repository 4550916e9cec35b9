"""The small router's ranking against the chunked kernel's, and the sort around its change-overs."""

import pytest
import torch

from uma_qmoe_b200 import _native, ops

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


@pytest.mark.parametrize("tokens,top_k,experts", [(1, 1, 1), (128, 8, 64), (1025, 1, 60), (512, 8, 64),
                                                  (2048, 8, 64), (2049, 8, 7), (5000, 4, 128)])
def test_sort_in_one_launch_and_in_two(tokens, top_k, experts):
    """Around a CTA's 1024 routes, at the change-over to two launches, and beyond it without scratch (one launch then)."""
    gen = torch.Generator(device=DEV).manual_seed(tokens)
    idx = torch.randint(-1, experts, (tokens, top_k), device=DEV, generator=gen)
    w = torch.rand(tokens, top_k, device=DEV, generator=gen)
    many = ops.route_sort(idx, w, experts)
    flat = idx.reshape(-1)
    order = torch.where(flat < 0, experts, flat).sort(stable=True).indices[:int((flat >= 0).sum())]
    n = len(order)
    assert torch.equal(many.sorted_route[:n].long(), order) and torch.equal(many.sorted_weight[:n], w.reshape(-1)[order])
    one = ops.SortedRoutes(*(torch.zeros_like(t) if torch.is_tensor(t) else t for t in vars(many).values()))
    code = _native.lib().umaq_route_sort(
        idx.data_ptr(), 1, w.data_ptr(), tokens, top_k, experts, one.counts.data_ptr(), one.offsets.data_ptr(),
        one.sorted_route.data_ptr(), one.route_pos.data_ptr(), one.sorted_weight.data_ptr(), one.num_tiles.data_ptr(),
        one.tile_table.data_ptr(), one.max_tiles, one.status.data_ptr(), None, 0, torch.cuda.current_stream().cuda_stream)
    assert code == 0
    tiles = int(one.num_tiles)
    assert torch.equal(one.counts, many.counts) and torch.equal(one.offsets, many.offsets) and tiles == int(many.num_tiles)
    assert torch.equal(one.sorted_route[:n], many.sorted_route[:n]) and torch.equal(one.route_pos, many.route_pos)
    assert torch.equal(one.tile_table.view(3, -1)[:, :tiles], many.tile_table.view(3, -1)[:, :tiles])
    assert int(one.status) == 0 and int(many.status) == 0


@pytest.mark.parametrize("hidden", [4096, 5632, 5888, 6144, 8192])
@pytest.mark.parametrize("tokens", [1, 7, 192, 193])
def test_router_takes_hidden_sizes_around_48_kb_of_rows(hidden, tokens):
    """Four rows and the ranks beside them pass what an ordinary launch may use.  Weights against float64: a logit of 64 terms of size
    one is rounded to BF16 (2^-9 of at most 4 here), which a softmax passes on as a relative error of 2^-7."""
    gen = torch.Generator(device=DEV).manual_seed(hidden)
    x = torch.randn(tokens, hidden, device=DEV, generator=gen).to(torch.bfloat16)
    weight = torch.zeros(64, hidden, device=DEV)
    weight[:, torch.randperm(hidden, device=DEV, generator=gen)[:64]] = torch.randn(64, 64, device=DEV, generator=gen) / 8
    weight = weight.to(torch.bfloat16)
    w, idx = ops.route_topk(x, weight, 8, False)
    exact = (x.double() @ weight.double().T).softmax(1).gather(1, idx)
    assert ((w.double() - exact).abs() <= 2.0 ** -6 * exact).all()


@pytest.mark.parametrize("tokens,top_k,experts", [(303104, 1, 64), (303105, 1, 64), (50003, 7, 60), (700001, 1, 128), (40000, 8, 1)])
def test_sort_without_scratch_of_more_routes_than_run_at_once(tokens, top_k, experts):
    """A CTA then places several batches of 1024 routes; some of the last one's may be empty."""
    gen = torch.Generator(device=DEV).manual_seed(tokens)
    idx = torch.randint(-1, experts, (tokens, top_k), device=DEV, generator=gen)
    w = torch.rand(tokens, top_k, device=DEV, generator=gen)
    r = ops.route_sort(idx, w, experts)
    for t in (r.counts, r.offsets, r.sorted_route, r.route_pos, r.sorted_weight, r.num_tiles, r.tile_table):
        t.zero_()
    code = _native.lib().umaq_route_sort(
        idx.data_ptr(), 1, w.data_ptr(), tokens, top_k, experts, r.counts.data_ptr(), r.offsets.data_ptr(), r.sorted_route.data_ptr(),
        r.route_pos.data_ptr(), r.sorted_weight.data_ptr(), r.num_tiles.data_ptr(), r.tile_table.data_ptr(), r.max_tiles,
        r.status.data_ptr(), None, 0, torch.cuda.current_stream().cuda_stream)
    flat = idx.reshape(-1)
    order = torch.where(flat < 0, experts, flat).sort(stable=True).indices[:int((flat >= 0).sum())]
    n = len(order)
    pos = torch.full_like(flat, -1)
    pos[order] = torch.arange(n, device=DEV)
    assert code == 0 and int(r.status) == 0
    assert torch.equal(r.counts.long(), torch.bincount(flat[flat >= 0], minlength=experts))
    assert torch.equal(r.sorted_route[:n].long(), order) and torch.equal(r.route_pos.long(), pos)
    assert torch.equal(r.sorted_weight[:n], w.reshape(-1)[order])


@pytest.mark.parametrize("experts,top_k", [(64, 8), (60, 4), (9, 8), (33, 1)])
@pytest.mark.parametrize("tokens", [1, 2, 3, 5, 9, 150, 192, 193])
def test_every_row_is_ranked_by_its_own_logits(experts, top_k, tokens):
    """Whatever run of sums the logits come from: the softmax of the logits that the same call returns, ties to the lower expert.
    A logit is the BF16 rounding of a sum that is off by 2^-20 of its terms' sizes at most, so it lies between the roundings of the ends.
    Weights: float32 exponentials, a sum of 64 and a quotient, 2^-20 together."""
    gen = torch.Generator(device=DEV).manual_seed(100 * experts + tokens)
    x = torch.randn(tokens, 2048, device=DEV, generator=gen).to(torch.bfloat16)
    weight = (torch.randn(experts, 2048, device=DEV, generator=gen) * 0.05).to(torch.bfloat16)
    weight[experts // 2] = weight[1]
    weight[experts - 1] = weight[0]
    exact = x.double() @ weight.double().T
    off = 2.0 ** -20 * (x.double().abs() @ weight.double().abs().T)
    for renormalize in (False, True):
        w, idx, logits = ops.route_topk(x, weight, top_k, renormalize, return_logits=True)
        assert ((logits >= (exact - off).to(torch.bfloat16)) & (logits <= (exact + off).to(torch.bfloat16))).all()
        order = logits.float().sort(dim=1, descending=True, stable=True).indices[:, :top_k]
        assert torch.equal(idx, order)
        p = logits.double().softmax(1).gather(1, order)
        if renormalize:
            p = p / p.sum(1, keepdim=True)
        assert ((w.double() - p).abs() <= 2.0 ** -20 * p).all()
