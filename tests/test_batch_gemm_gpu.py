"""Grouped GEMMs between few routes and full 256-row tiles: wide transposed tiles (grouped_wide.cu), bit for bit against the
one-CTA kernel, and batches of Q8 layers: small values beside large ones, and the same bits in a batch of any size."""

import pytest
import torch

from tests.test_prefill_gpu import DEV, _reference_layer, _stagewise
from uma_qmoe_b200 import synthetic as syn

pytestmark = pytest.mark.gpu


def _layer(model, encoding, seed):
    from uma_qmoe_b200.stack import random_layer
    shape = syn.OLMOE if model == "olmoe" else syn.QWEN
    return shape, random_layer(shape, encoding, seed, torch.device(DEV))


def _prefill(layer, x, idx, w):
    from uma_qmoe_b200 import ops
    ws = ops.prefill_workspace(layer, x.shape[0], idx.shape[1], None, torch.device(DEV))
    y = ops.moe_prefill(layer, x, idx, w, ws)
    assert ops.prefill_status(ws) == 0
    return y


def _launched(call, tmp_path):
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        call()
        graph = torch.cuda.CUDAGraph(keep_graph=True)
        graph.enable_debug_mode()
        with torch.cuda.graph(graph, stream=stream):
            call()
    graph.debug_dump(str(tmp_path / "graph.dot"))
    text = (tmp_path / "graph.dot").read_text()
    return {n for n in ("grouped_gemm_kernel", "grouped_ts_kernel", "grouped_wide_kernel") if n in text}


@pytest.mark.parametrize("model", ["olmoe", "qwen"])
@pytest.mark.parametrize("encoding", ["q4_group128", "q8_group128"])
@pytest.mark.parametrize("counts", [[192, 193, 16, 0, 385, 47, 191, 1], [2100, 0, 1, 15, 64, 17, 0, 0], [128] * 8])
def test_wide_tiles_give_the_bits_of_the_one_cta_kernel(model, encoding, counts, tmp_path):
    """Equal parts of an expert's routes: one tile and a route more, three tiles, many, single routes, none."""
    shape, layer = _layer(model, encoding, 3)
    if sum(counts) > 1300:
        counts = counts + [0] * (len(counts) * 2)                    # the average has to stay in the kernel's range
    gen = torch.Generator(device=DEV).manual_seed(sum(counts))
    expert = torch.cat([torch.full((counts[n % len(counts)],), n, device=DEV) for n in range(shape.experts)])
    expert = expert[torch.randperm(len(expert), device=DEV, generator=gen)][:, None].contiguous()
    x = torch.randn(len(expert), shape.hidden, device=DEV, generator=gen).to(torch.bfloat16)
    w = torch.rand(len(expert), 1, device=DEV, generator=gen) + 0.1
    assert _launched(lambda: _prefill_launch(layer, x, expert, w), tmp_path) == {"grouped_wide_kernel"}
    assert torch.equal(_prefill(layer, x, expert, w), _stagewise(layer, x, expert, w, variant=1)[1])


def _prefill_launch(layer, x, idx, w):
    from uma_qmoe_b200 import ops
    return ops.moe_prefill(layer, x, idx, w, ops.prefill_workspace(layer, x.shape[0], idx.shape[1], None, torch.device(DEV)))


@pytest.mark.parametrize("tokens", [100, 7000])
def test_q4_scales_outside_the_fused_conversion(tokens):
    """Scales of 2^-5 and more, below 2^-100 and zero take the general conversion, group by group, on the transposed, the wide
    and the one-CTA kernel.  Bounds as for the few-routes kernel: two BF16 roundings on either side."""
    shape, layer = _layer("olmoe", "q4_group128", 5)
    gen = torch.Generator(device=DEV).manual_seed(4)
    for scales in (layer.gate_scales, layer.up_scales, layer.down_scales):
        pick = torch.rand(scales.shape, device=DEV, generator=gen)
        scales.copy_(torch.where(pick < 0.002, 0.0, torch.where(pick < 0.004, 0.03125, torch.where(pick < 0.006, 1e-37, scales))))
    expert = torch.randint(64, (tokens, 1), device=DEV, generator=gen)
    x = torch.randn(tokens, 2048, device=DEV, generator=gen).to(torch.bfloat16)
    w = torch.rand(tokens, 1, device=DEV, generator=gen) + 0.1
    want = _reference_layer(layer, x, expert[:, 0], w[:, 0]).float()
    for got in (_prefill(layer, x, expert, w).float(), _stagewise(layer, x, expert, w, variant=1)[1].float().to(DEV)):
        assert (got - want).norm() <= 2.0 ** -8 * want.norm()
        assert (got - want).abs().max() <= 2.0 ** -7 * want.abs().max()


def _exact(layer, x, idx, w):
    """A Q8 layer in 64 bits over the stored codes and scales, without any rounding; one route per token."""
    e, h, i = layer.num_experts, layer.hidden, layer.intermediate
    deq = lambda c, s, n, k: (c.view(torch.int8).double().reshape(-1, 128) * s.double()[:, None]).reshape(e, n, k)
    gate, up = deq(layer.gate, layer.gate_scales, i, h), deq(layer.up, layer.up_scales, i, h)
    down = deq(layer.down, layer.down_scales, h, i)
    out = torch.zeros(len(x), h, dtype=torch.float64, device=DEV)
    for n in range(e):
        r = (idx[:, 0] == n).nonzero().flatten()
        mid = torch.nn.functional.silu(x[r].double() @ gate[n].T) * (x[r].double() @ up[n].T)
        out[r] = mid @ down[n].T * w[r].double()
    return out


@pytest.mark.parametrize("model", ["olmoe", "qwen"])
@pytest.mark.parametrize("where", ["x", "intermediate"])
@pytest.mark.parametrize("factor", [100.0, 3000.0, 1e5])
def test_q8_batch_keeps_small_values_beside_a_large_one(model, where, factor):
    """One channel of every 128 far above the others, under codes that are zero: its neighbours keep their precision.  The BF16
    roundings of weights, intermediate and result (2^-9 each at most) came to 0.0037 in the 2-norm of a layer; 0.006 leaves room for
    single tokens.  The bits are the one-CTA kernel's."""
    shape, layer = _layer(model, "q8_group128", 7)
    e, h, i = shape.experts, shape.hidden, shape.intermediate
    gen = torch.Generator(device=DEV).manual_seed(3)
    x = torch.randn(100, h, device=DEV, generator=gen).to(torch.bfloat16)
    if where == "x":
        x[:, 7::128] *= factor
        for codes in (layer.gate, layer.up):
            codes.view(torch.int8).view(e, i, h)[:, :, 7::128] = 0
    else:
        layer.up_scales.view(e, i, h // 128)[:, 5::128] *= factor
        layer.down.view(torch.int8).view(e, h, i)[:, :, 5::128] = 0
    idx = torch.randint(e, (100, 1), device=DEV, generator=gen)
    w = torch.rand(100, 1, device=DEV, generator=gen) + 0.1
    got, want = _prefill(layer, x, idx, w), _exact(layer, x, idx, w)
    assert ((got.double() - want).norm(dim=1) <= 0.006 * want.norm(dim=1)).all()
    assert torch.equal(got, _stagewise(layer, x, idx, w, variant=1)[1])


def test_q8_batch_gives_an_infinity_where_one_feature_overflows():
    """SwiGLU of one feature overflows: the rows whose down code is not zero are infinite, the others NaN (infinity times zero)."""
    shape, layer = _layer("olmoe", "q8_group128", 9)
    gen = torch.Generator(device=DEV).manual_seed(1)
    row = lambda codes, scales: (codes.view(torch.int8).view(64, 1024, 16, 128)[:, 17].double() *
                                 scales.view(64, 1024, 16, 1)[:, 17].double()).reshape(64, 2048)
    layer.gate_scales.view(64, 1024, 16)[:, 17] *= 100.0
    layer.up_scales.view(64, 1024, 16)[:, 17] *= 1e19
    layer.up_scales.view(64, 1024, 16)[:, 17] *= 1e19                # the sums stay within float32, the product does not
    idx = torch.randint(64, (40, 1), device=DEV, generator=gen)
    x = torch.randn(40, 2048, device=DEV, generator=gen).to(torch.bfloat16)
    got = _prefill(layer, x, idx, torch.ones(40, 1, device=DEV))
    gate, up = ((x.double() * row(c, s)[idx[:, 0]]).sum(1) for c, s in ((layer.gate, layer.gate_scales), (layer.up, layer.up_scales)))
    over = (torch.nn.functional.silu(gate) * up).abs() > 4e38
    zero = (layer.down.view(torch.int8).view(64, 2048, 1024)[idx[:, 0], :, 17] == 0)[over]
    assert over.sum() > 5 and zero.any()
    assert torch.equal(got[over].isnan(), zero) and torch.equal(got[over].isinf(), ~zero)


@pytest.mark.parametrize("model", ["olmoe", "qwen"])
@pytest.mark.parametrize("tokens", [4, 24, 192])
def test_q8_token_has_the_same_bits_in_a_batch_of_any_size(model, tokens):
    shape, layer = _layer(model, "q8_group128", 11)
    gen = torch.Generator(device=DEV).manual_seed(2)
    idx = torch.rand(700, shape.experts, device=DEV, generator=gen).topk(shape.top_k, 1).indices.contiguous()
    x = torch.randn(700, shape.hidden, device=DEV, generator=gen).to(torch.bfloat16)
    w = torch.rand(700, shape.top_k, device=DEV, generator=gen)
    few = _prefill(layer, x[:tokens], idx[:tokens], w[:tokens])
    for more in (193, 700):
        assert torch.equal(_prefill(layer, x[:more], idx[:more], w[:more])[:tokens], few)
    assert torch.equal(_stagewise(layer, x[:tokens], idx[:tokens], w[:tokens], variant=1)[1], few)
