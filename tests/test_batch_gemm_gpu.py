"""Grouped GEMMs between few routes and full 256-row tiles: wide transposed tiles (grouped_wide.cu), bit for bit against the
one-CTA kernel, and Q8 batches on integer digits (grouped_digits.cu), against 64 bits."""

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


def _exact(layer, x, idx, w):
    """Per-route results in 64 bits over the stored codes and scales, the intermediate and the result rounded to BF16 (as every
    path does) or not at all."""
    e, h, i = layer.num_experts, layer.hidden, layer.intermediate
    deq = lambda c, s, n, k: (c.view(torch.int8).double().reshape(-1, 128) * s.double()[:, None]).reshape(e, n, k)
    gate, up = deq(layer.gate, layer.gate_scales, i, h), deq(layer.up, layer.up_scales, i, h)
    down = deq(layer.down, layer.down_scales, h, i)
    flat, weight, rows = idx.reshape(-1), w.reshape(-1, 1).double(), x.repeat_interleave(idx.shape[1], 0).double()
    rounded, plain = (torch.zeros(len(flat), h, dtype=torch.float64, device=DEV) for _ in range(2))
    for n in range(e):
        r = (flat == n).nonzero().flatten()
        if len(r):
            mid = torch.nn.functional.silu(rows[r] @ gate[n].T) * (rows[r] @ up[n].T)
            plain[r] = mid @ down[n].T * weight[r]
            rounded[r] = (mid.to(torch.bfloat16).double() @ down[n].T * weight[r]).to(torch.bfloat16).double()
    return rounded, plain


@pytest.mark.parametrize("model", ["olmoe", "qwen"])
@pytest.mark.parametrize("counts", [[16, 17, 1, 31, 33, 63], [65, 0, 64, 2], [128, 64], [1] * 40])
def test_digits_of_q8_batches_match_float64(model, counts, tmp_path):
    """Against the same two roundings in 64 bits only values whose sum falls on the other side of a rounding boundary differ: the
    digits are off by 2^-15 of a group's largest value (2^-16 on average over a normal group's 2.7 sigma: 2.4e-5), so one
    value in a hundred, by 2^-8 of itself; 2^-10 in the 2-norm leaves a factor of two.  Against no rounding at all the result is no
    further off than the BF16 kernels'."""
    shape, layer = _layer(model, "q8_group128", 7)
    gen = torch.Generator(device=DEV).manual_seed(sum(counts))
    idx = torch.cat([torch.full((c,), (11 * n) % shape.experts, device=DEV) for n, c in enumerate(counts)])
    idx = idx[torch.randperm(len(idx), device=DEV, generator=gen)][:, None].contiguous()
    x = torch.randn(len(idx), shape.hidden, device=DEV, generator=gen).to(torch.bfloat16)
    x[0] *= 1e15
    x[1] *= 1e-30
    x[2, 5] = 300.0                                                      # one value far above the others of its group
    x[3, 256:512] = 0.0
    w = torch.rand(len(idx), 1, device=DEV, generator=gen) + 0.1
    w[0] *= 1e-30                                                        # SwiGLU squares the 1e15
    assert _launched(lambda: _prefill_launch(layer, x, idx, w), tmp_path) == {"grouped_digits_kernel"}
    got, bf16 = _prefill(layer, x, idx, w).double(), _prefill(layer, x, idx, w, digits=False).double()
    rounded, plain = _exact(layer, x, idx, w)
    rel = lambda a, b: ((a - b).norm(dim=1) / b.norm(dim=1))
    rest = torch.ones(len(idx), dtype=torch.bool, device=DEV)
    rest[1] = False                                                      # its results are below the smallest BF16 number
    assert (rel(got, plain)[rest] <= rel(bf16, plain)[rest]).all()
    assert (got[1] == 0).all()
    rest[2] = False                                                      # its group's rounding is 300 / 2.7 times as coarse
    assert (rel(got, rounded)[rest] <= 2.0 ** -9).all() and rel(got, rounded)[rest].mean() <= 2.0 ** -10


def test_digits_carry_infinities_and_nan_to_their_own_token_only():
    shape, layer = _layer("olmoe", "q8_group128", 9)
    gen = torch.Generator(device=DEV).manual_seed(1)
    idx = torch.rand(32, 64, device=DEV, generator=gen).topk(8, 1).indices.contiguous()
    x = torch.randn(32, 2048, device=DEV, generator=gen).to(torch.bfloat16)
    w = torch.rand(32, 8, device=DEV, generator=gen)
    clean = _prefill(layer, x, idx, w)
    x[3, 100], x[17, 2047] = float("inf"), float("nan")
    dirty = _prefill(layer, x, idx, w)
    keep = torch.ones(32, dtype=torch.bool, device=DEV)
    keep[[3, 17]] = False
    assert torch.equal(dirty[keep], clean[keep]) and dirty[~keep].isnan().all()
    assert _prefill(layer, x, idx, w, digits=False)[~keep].isnan().all()       # as on the BF16 kernels
