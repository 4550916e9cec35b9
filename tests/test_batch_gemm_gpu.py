"""Grouped GEMMs between few routes and full 256-row tiles: wide transposed tiles (grouped_wide.cu), bit for bit against the
one-CTA kernel."""

import pytest
import torch

from tests.test_prefill_gpu import DEV, _reference_layer, _stagewise
from uma_qmoe_b200 import synthetic as syn

pytestmark = pytest.mark.gpu


def _layer(model, encoding, seed):
    from uma_qmoe_b200.stack import random_layer
    shape = syn.OLMOE if model == "olmoe" else syn.QWEN
    return shape, random_layer(shape, encoding, seed, torch.device(DEV))


def _prefill(layer, x, idx, w, **kw):
    from uma_qmoe_b200 import ops
    ws = ops.prefill_workspace(layer, x.shape[0], idx.shape[1], None, torch.device(DEV))
    y = ops.moe_prefill(layer, x, idx, w, ws, **kw)
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
    return {n for n in ("grouped_gemm_kernel", "grouped_ts_kernel", "grouped_wide_kernel", "grouped_digits_kernel") if n in text}


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
