"""Prefill path (route sort, tcgen05 grouped GEMMs, ordered combine) and the fused router vs the
CPU oracle and the reference-made golden vectors, through the C ABI."""

import numpy as np
import pytest
import torch

from oracle import moe_oracle as orc
from tests.helpers import SEED, assert_parity, bits_to_bf16, expert_source, stage_layer
from uma_qmoe_b200 import synthetic as syn

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _run_prefill(layer, x, idx, w, shared=None):
    from uma_qmoe_b200 import ops
    ws = ops.prefill_workspace(layer, x.shape[0], idx.shape[1], shared, torch.device(DEV))
    args = (layer, x.to(DEV).contiguous(), idx.to(DEV).contiguous(), w.to(DEV).contiguous(), ws, shared)
    y = ops.moe_prefill(*args)
    y2 = ops.moe_prefill(*args)
    torch.cuda.synchronize()
    assert ops.prefill_status(ws) == 0
    assert torch.equal(y, y2), "two calls must give identical bits"
    return y.cpu()


def test_olmoe_prefill_golden(golden_dir):
    g = np.load(golden_dir / "olmoe_prefill.npz")
    x = bits_to_bf16(g["x_bits"])
    idx, w = torch.from_numpy(g["idx"]), torch.from_numpy(g["w"])
    src = expert_source(SEED, 3, "olmoe", "q4_group128")
    experts = {int(e): src(int(e)) for e in set(idx.reshape(-1).tolist())}
    layer = stage_layer(experts, 64, 2048, 1024, "q4_group128", DEV)
    assert_parity(_run_prefill(layer, x, idx, w), bits_to_bf16(g["y_bits"]))


@pytest.mark.parametrize("layer_index", [0, 1, 2])
def test_qwen_prefill_golden(golden_dir, layer_index):
    from uma_qmoe_b200.ops import DeviceSharedExpert
    g = np.load(golden_dir / "qwen_layers.npz")
    enc = str(g[f"L{layer_index}_encoding"])
    src = expert_source(SEED, layer_index, "qwen", enc)
    x = bits_to_bf16(g["x8_bits"])
    idx = torch.from_numpy(g[f"L{layer_index}_i8"])
    w = torch.from_numpy(g[f"L{layer_index}_w8"])
    experts = {int(e): src(int(e)) for e in set(idx.reshape(-1).tolist())}
    layer = stage_layer(experts, 60, 2048, 1408, enc, DEV)
    assert_parity(_run_prefill(layer, x, idx, w), bits_to_bf16(g[f"L{layer_index}_y8_bits"]))
    sg, su, sd, sgate = (t.to(DEV).contiguous() for t in syn.shared_expert_weights(SEED, layer_index, syn.QWEN))
    b = _run_prefill(layer, x, idx, w, DeviceSharedExpert(sg, su, sd, sgate))
    assert_parity(b, bits_to_bf16(g[f"L{layer_index}_b8_bits"]))


def test_prefill_many_tokens_few_experts_matches_oracle():
    """300 tokens over 4 experts: several 128-route tiles per expert, ragged last tiles, one empty expert."""
    src = expert_source(SEED, 9, "olmoe", "q4_group128")
    tokens = 300
    rng = np.random.default_rng(5)
    idx = torch.from_numpy(np.stack([rng.permutation([0, 1, 2, 4, 5, 6, 7, 8])[:8] for _ in range(tokens)]).astype(np.int64))
    idx[:, 4:] = idx[:, :4]          # every token hits only 4 distinct experts, each twice
    w = torch.from_numpy(rng.random((tokens, 8), dtype=np.float32) / 8)
    used = sorted(set(idx.reshape(-1).tolist()))
    layer = stage_layer({e: src(e) for e in used}, 16, 2048, 1024, "q4_group128", DEV)
    x = syn.activations(SEED + 21, tokens)
    want = orc.moe_forward(x, idx, w, src, num_experts=64, top_k=8, qwen=False)
    assert_parity(_run_prefill(layer, x, idx, w), want)


@pytest.mark.parametrize("tokens", [500, 40, 5, 299])      # tensor-core kernel (ragged last CTA) / cluster kernel: ten
                                                            # clusters, two with a one-token tail, 75 with a ragged tail
@pytest.mark.parametrize("model,renorm", [("olmoe", True), ("olmoe", False), ("qwen", False)])
def test_router_matches_oracle(model, renorm, tokens):
    from uma_qmoe_b200 import ops
    shape = syn.OLMOE if model == "olmoe" else syn.QWEN
    wr = syn.router_weight(SEED, 1, shape, skew=1.5)
    x = syn.activations(SEED + 31, tokens)
    probs, w_ref, idx_ref = orc.router_topk(x, wr, shape.top_k, renorm)
    w, idx, logits = ops.route_topk(x.to(DEV), wr.to(DEV), shape.top_k, renorm, return_logits=True)
    w, idx, logits = w.cpu(), idx.cpu(), logits.cpu()
    ref_logits = torch.nn.functional.linear(x, wr)
    same_logits = (logits == ref_logits).all(dim=1)
    # BF16 logits are coarse, so equal probabilities are common.  Rows whose logits agree with the
    # oracle's and whose k-th and (k+1)-th probabilities differ must select the same expert SET with
    # the same weights; if no two of the top k+1 are equal the order must match too.
    srt = probs.sort(dim=1, descending=True).values
    k = shape.top_k
    boundary_clear = same_logits & (srt[:, k - 1] != srt[:, k])
    all_clear = same_logits & (srt[:, : k + 1].diff(dim=1) != 0).all(dim=1)
    # the kernel rounds an exactly summed dot product; the CPU GEMM of the oracle is off by one BF16 ulp on
    # about 1 logit in 5000, i.e. on 1-2 % of the rows
    if tokens >= 40:                                   # (with a handful of rows these shares are not statistics)
        assert same_logits.float().mean() >= 0.95 and boundary_clear.float().mean() > 0.85 and all_clear.any()
    assert torch.equal(idx[boundary_clear].sort(dim=1).values, idx_ref[boundary_clear].sort(dim=1).values)
    assert torch.allclose(w[boundary_clear].sort(dim=1).values, w_ref[boundary_clear].sort(dim=1).values,
                          rtol=2e-5, atol=1e-8)
    assert torch.equal(idx[all_clear], idx_ref[all_clear])
    assert torch.allclose(w[all_clear], w_ref[all_clear], rtol=2e-5, atol=1e-8)
    # every other row must still pick a valid top-k of its own logits
    own = torch.softmax(logits.float(), dim=1)
    chosen = own.gather(1, idx)
    kth = own.sort(dim=1, descending=True).values[:, shape.top_k - 1]
    assert bool((chosen >= kth[:, None] - 1e-9).all())
    assert int((~same_logits).sum()) <= max(1, 0.05 * x.shape[0])


@pytest.mark.parametrize("tokens,top_k,experts,dtype", [(8192, 8, 64, torch.int64), (5000, 4, 60, torch.int32),
                                                        (3, 8, 64, torch.int64)])
def test_route_sort_is_the_stable_sort_by_expert(tokens, top_k, experts, dtype):
    """Single-CTA and many-CTA sorts both equal a stable argsort; the tile list covers every route once."""
    from uma_qmoe_b200 import ops
    gen = torch.Generator().manual_seed(SEED + tokens)
    popularity = 1.0 / torch.arange(1, experts + 1, dtype=torch.float64) ** 1.2
    idx = torch.multinomial(popularity.expand(tokens, experts), top_k, replacement=False, generator=gen).to(dtype)
    w = torch.rand((tokens, top_k), generator=gen, dtype=torch.float32)
    r = ops.route_sort(idx.to(DEV), w.to(DEV), experts)
    torch.cuda.synchronize()
    assert int(r.status.item()) == 0
    flat = idx.reshape(-1).long()
    order = torch.argsort(flat, stable=True)
    counts = torch.bincount(flat, minlength=experts)
    assert torch.equal(r.sorted_route.cpu().long(), order)
    assert torch.equal(r.counts.cpu().long(), counts)
    assert torch.equal(r.offsets.cpu().long(), torch.cat([torch.zeros(1, dtype=torch.long), counts.cumsum(0)]))
    assert torch.equal(r.route_pos.cpu().long()[order], torch.arange(flat.numel()))
    assert torch.equal(r.sorted_weight.cpu(), w.reshape(-1)[order])
    tiles = int(r.num_tiles.item())
    table = r.tile_table.cpu().view(3, r.max_tiles)[:, :tiles]
    covered = torch.zeros(flat.numel(), dtype=torch.int32)
    for e, row0, rows in table.t().tolist():
        assert (flat[order[row0:row0 + rows]] == e).all()
        covered[row0:row0 + rows] += 1
    assert (covered == 1).all()


def _stagewise(layer, x, idx, w, variant):
    """Prefill assembled from the exported stages, with the grouped GEMM kernel chosen explicitly."""
    from uma_qmoe_b200 import ops
    quant = layer.encoding != "bf16_le"
    r = ops.route_sort(idx, w, layer.num_experts)
    xs = ops.gather_rows(x, r.sorted_route, idx.shape[1], permute=quant)
    inter = ops.grouped_gemm(layer, 0, xs, r, permute_out=quant, variant=variant)
    yw = ops.grouped_gemm(layer, 1, inter, r, route_weight=r.sorted_weight, variant=variant)
    y = ops.combine_routes(yw, idx, r.route_pos)
    torch.cuda.synchronize()
    assert int(r.status.item()) == 0
    return inter, y


@pytest.mark.parametrize("encoding", ["q4_group128", "q8_group128", "bf16_le"])
def test_pair_kernel_matches_single_cta_kernel_and_oracle(encoding):
    """The persistent CTA-pair GEMM (cta_group::2) against the one-CTA-per-tile GEMM and the oracle: 700 tokens
    over 5 experts give full 256-route tiles, ragged tiles above and below 128 routes, and enough (tile, column)
    items that every cluster walks several of them with both accumulators in use."""
    src = expert_source(SEED, 3, "olmoe", encoding)
    tokens = 700
    rng = np.random.default_rng(11)
    pool = np.array([0, 2, 3, 5, 9])
    prob = np.array([0.45, 0.3, 0.15, 0.07, 0.03])
    idx = torch.from_numpy(np.stack([rng.choice(pool, size=2, replace=False, p=prob) for _ in range(tokens)]).astype(np.int64))
    w = torch.from_numpy(rng.random((tokens, 2), dtype=np.float32) / 2)
    layer = stage_layer({int(e): src(int(e)) for e in pool}, 16, 2048, 1024, encoding, DEV)
    x = syn.activations(SEED + 33, tokens)
    args = (layer, x.to(DEV), idx.to(DEV), w.to(DEV))
    inter1, y1 = _stagewise(*args, variant=1)
    inter2, y2 = _stagewise(*args, variant=2)
    inter2b, y2b = _stagewise(*args, variant=2)
    assert torch.equal(y2, y2b) and torch.equal(inter2, inter2b), "two calls must give identical bits"
    assert_parity(y2.cpu(), y1.cpu(), max_abs=4e-3)
    mismatch = (inter1 != inter2).float().mean().item()
    assert mismatch < 1e-3, f"intermediates differ in {mismatch:.2%} of the elements"
    want = orc.moe_forward(x, idx, w, src, num_experts=64, top_k=2, qwen=False)
    assert_parity(y2.cpu(), want)


def test_large_batch_prefill_matches_the_pair_kernel_and_the_oracle():
    """4096 tokens x top-8 (32768 routes: every persistent CTA walks many tiles) through umaq_moe_prefill vs the
    stages run on the CTA-pair kernel; a sample of tokens is checked against the oracle."""
    src = expert_source(SEED, 5, "olmoe", "q4_group128")
    tokens, experts = 4096, 16
    gen = torch.Generator().manual_seed(SEED + 77)
    popularity = 1.0 / torch.arange(1, experts + 1, dtype=torch.float64) ** 1.1
    idx = torch.multinomial(popularity.expand(tokens, experts), 8, replacement=False, generator=gen)
    w = torch.rand((tokens, 8), generator=gen, dtype=torch.float32) / 8
    layer = stage_layer({e: src(e) for e in range(experts)}, experts, 2048, 1024, "q4_group128", DEV)
    x = syn.activations(SEED + 34, tokens)
    y = _run_prefill(layer, x, idx, w)
    _, y2 = _stagewise(layer, x.to(DEV), idx.to(DEV), w.to(DEV), variant=2)
    assert_parity(y, y2.cpu(), max_abs=4e-3)
    sample = torch.arange(0, tokens, 512)
    want = orc.moe_forward(x[sample], idx[sample], w[sample], src, num_experts=experts, top_k=8, qwen=False)
    assert_parity(y[sample], want)


@pytest.mark.parametrize("encoding", ["q4_group128", "q8_group128", "bf16_le"])
def test_gate_up_gemm_by_index_equals_the_gemm_on_gathered_rows(encoding):
    """The gate/up GEMM that fetches its activation rows itself (cp.async producers writing the swizzled tile) must
    give the bits of the same GEMM on a gathered copy: full, ragged and half tiles, and an expert without routes."""
    from uma_qmoe_b200 import ops
    src = expert_source(SEED, 7, "olmoe", encoding)
    tokens = 777
    rng = np.random.default_rng(12)
    pool = np.array([0, 1, 3, 4, 7, 8, 11])
    idx = torch.from_numpy(np.stack([rng.choice(pool, 2, replace=False, p=[.5, .2, .1, .1, .05, .03, .02]) for _ in range(tokens)]))
    w = torch.rand((tokens, 2), generator=torch.Generator().manual_seed(3)) / 2
    layer = stage_layer({int(e): src(int(e)) for e in pool}, 16, 2048, 1024, encoding, DEV)
    x = syn.activations(SEED + 36, tokens).to(DEV)
    quant = encoding != "bf16_le"
    r = ops.route_sort(idx.to(DEV), w.to(DEV), layer.num_experts)
    xs = ops.gather_rows(x, r.sorted_route, 2, permute=quant)
    want = ops.grouped_gemm(layer, 0, xs, r, permute_out=quant, variant=1)
    source = ops.gather_rows(x, None, 1, permute=True) if quant else x
    got = ops.grouped_gemm_by_index(layer, source, r, 2, permute_out=quant)
    again = ops.grouped_gemm_by_index(layer, source, r, 2, permute_out=quant)
    torch.cuda.synchronize()
    assert int(r.status.item()) == 0
    assert torch.equal(got, want) and torch.equal(got, again)


def test_bf16_large_batch_takes_the_pair_kernel_by_default_and_matches_the_one_cta_kernel():
    """BF16 layers on 16,384 routes or more run on the CTA-pair kernel unless the caller picks one; the whole
    operator must agree with the stages run explicitly on the one-CTA kernel and with the oracle on a sample."""
    src = expert_source(SEED, 6, "olmoe", "bf16_le")
    tokens, experts = 2048, 16
    gen = torch.Generator().manual_seed(SEED + 78)
    idx = torch.stack([torch.randperm(experts, generator=gen)[:8] for _ in range(tokens)])
    w = torch.rand((tokens, 8), generator=gen, dtype=torch.float32) / 8
    layer = stage_layer({e: src(e) for e in range(experts)}, experts, 2048, 1024, "bf16_le", DEV)
    x = syn.activations(SEED + 35, tokens)
    y = _run_prefill(layer, x, idx, w)                                        # 16,384 routes: variant 0 -> pairs
    _, y1 = _stagewise(layer, x.to(DEV), idx.to(DEV), w.to(DEV), variant=1)
    _, y2 = _stagewise(layer, x.to(DEV), idx.to(DEV), w.to(DEV), variant=2)
    assert torch.equal(y, y2.cpu())
    assert_parity(y, y1.cpu(), max_abs=4e-3)
    sample = torch.arange(0, tokens, 256)
    want = orc.moe_forward(x[sample], idx[sample], w[sample], src, num_experts=experts, top_k=8, qwen=False)
    assert_parity(y[sample], want)


def test_operator_edge_shapes_through_the_registered_backend():
    """The public operator on an empty batch, on one token (decode kernels) and on two tokens (prefill kernels):
    same pack, results consistent with each other."""
    from uma_qmoe_b200 import custom_op, native_backend
    from uma_qmoe_b200.packs import InMemoryPack, expert_tensor_name
    from uma_qmoe_b200.formats import encode
    pack = InMemoryPack({0: "q4_group128"})
    packed = {}                                      # 8 distinct experts, repeated to fill the layer's 64
    for e in range(8):
        for proj, m in zip(("gate_proj", "up_proj", "down_proj"), syn.expert_weights(SEED, 0, e, syn.OLMOE)):
            packed[e, proj] = encode(m, "q4_group128")
    for e in range(64):
        for proj in ("gate_proj", "up_proj", "down_proj"):
            pack.add_packed(expert_tensor_name(0, e, proj), packed[e % 8, proj])
    native_backend.install_mixed_target_backend()
    handle = custom_op.register_expert_pack(pack)
    try:
        x = syn.activations(SEED + 3, 2).to(DEV)
        idx = torch.tensor([[0, 1, 2, 3, 4, 5, 6, 7], [7, 6, 5, 4, 3, 2, 1, 0]], device=DEV)
        w = torch.full((2, 8), 0.125, device=DEV)
        both = torch.ops.uma_qmoe.moe_forward(x, idx, w, 0, handle, True)
        one = torch.ops.uma_qmoe.moe_forward(x[:1], idx[:1], w[:1], 0, handle, True)
        none = torch.ops.uma_qmoe.moe_forward(x[:0], idx[:0], w[:0], 0, handle, True)
        assert none.shape == (0, 2048) and none.dtype == torch.bfloat16
        assert_parity(one.cpu(), both[:1].cpu(), max_abs=4e-3)
        three_d = torch.ops.uma_qmoe.moe_forward(x.reshape(1, 2, 2048), idx, w, 0, handle, True)
        assert three_d.shape == (1, 2, 2048) and torch.equal(three_d.reshape(2, 2048), both)
        with pytest.raises(RuntimeError, match=r"requires \[tokens, 8\] routes"):
            torch.ops.uma_qmoe.moe_forward(x, idx[:, :4], w[:, :4], 0, handle, True)
        with pytest.raises(RuntimeError, match="layer_index must be in"):
            torch.ops.uma_qmoe.moe_forward(x, idx, w, 16, handle, True)
    finally:
        custom_op.unregister_expert_pack(handle)


def test_reference_validator_and_route_trace_prefill(golden_dir):
    """The reference validator's 32-token case and the 128-token prefill event of layer 0 of its frozen route
    trace (32 of 64 experts hit, 53 routes on the busiest, un-normalised weights), against the reference's CPU
    outputs."""
    g = np.load(golden_dir / "reference_cases.npz")
    src = expert_source(SEED, int(g["layer"]), "olmoe", "q4_group128")
    layer = stage_layer({int(e): src(int(e)) for e in g["hit"]}, 64, 2048, 1024, "q4_group128", DEV)
    idx = torch.from_numpy(g["val_idx"]).repeat(32, 1)
    w = bits_to_bf16(g["val_w_bits"]).float().repeat(32, 1)
    assert_parity(_run_prefill(layer, bits_to_bf16(g["val_x32_bits"]), idx, w), bits_to_bf16(g["val_y32_bits"]))
    y = _run_prefill(layer, bits_to_bf16(g["trace_prefill_x_bits"]), torch.from_numpy(g["trace_prefill_idx"]),
                     torch.from_numpy(g["trace_prefill_w"]))
    assert_parity(y, bits_to_bf16(g["trace_prefill_y_bits"]))


def test_baseline_prefill_512_tokens_skewed_router():
    """The 512-token prefill configuration exactly: all 64 experts staged, routes from the skewed seeded router
    through the router kernel (some experts get no token, the busiest at least three times the mean), result
    against the CPU oracle."""
    from uma_qmoe_b200 import ops
    shape = syn.OLMOE
    src = expert_source(SEED, 2, "olmoe", "q4_group128")
    layer = stage_layer({e: src(e) for e in range(64)}, 64, 2048, 1024, "q4_group128", DEV)
    x = syn.activations(SEED + 51, 512)
    wr = syn.router_weight(SEED, 2, shape, skew=1.5)
    w, idx = ops.route_topk(x.to(DEV), wr.to(DEV), shape.top_k, True)
    w, idx = w.cpu(), idx.cpu()
    counts = torch.bincount(idx.reshape(-1), minlength=64)
    assert int(counts.min()) == 0 and int(counts.max()) >= 3 * counts.float().mean(), counts.tolist()
    want = orc.moe_forward(x, idx, w, src, num_experts=64, top_k=8, qwen=False)
    assert_parity(_run_prefill(layer, x, idx, w), want)


def test_stack_shape_8192_tokens_sampled_rows():
    """The expert-parallel stack's shape (8192 tokens x 64 experts x top-8, layer 0 of the benchmark stack) on one
    GPU; 64 sampled token rows against the CPU oracle, which dequantises the staged bytes of the experts they hit."""
    from uma_qmoe_b200 import ops
    from uma_qmoe_b200.stack import random_layer
    shape = syn.OLMOE
    dev = torch.device(DEV)
    layer = random_layer(shape, "q4_group128", SEED, dev)
    x = syn.activations(SEED, 8192)
    wr = syn.router_weight(SEED, 0, shape, skew=1.0)
    w, idx = ops.route_topk(x.to(dev), wr.to(dev), shape.top_k, True)
    y = _run_prefill(layer, x, idx.cpu(), w.cpu())
    rows = torch.arange(0, 8192, 128)
    idx_s, w_s = idx.cpu()[rows], w.cpu()[rows]

    def staged(e: int):
        def take(t, s, n, k):
            per = n * k // 2
            data = t[e * per:(e + 1) * per].cpu().numpy()
            scales = s[e * (n * k // 128):(e + 1) * (n * k // 128)].cpu().numpy()
            return orc.EncodedMatrix("q4_group128", (n, k), data, scales)
        return (take(layer.gate, layer.gate_scales, 1024, 2048), take(layer.up, layer.up_scales, 1024, 2048),
                take(layer.down, layer.down_scales, 2048, 1024))
    cache = {}
    src = lambda e: cache.setdefault(e, staged(e))
    want = orc.moe_forward(x[rows], idx_s, w_s, src, num_experts=64, top_k=8, qwen=False)
    assert_parity(y[rows], want)


# ---- few routes per expert: the transposed kernel (grouped_ts.cu) ------------------------------------------------

def _dequantised(codes, scales, encoding, experts, rows, k):
    """The BF16 weights the tensor cores multiply, from the staged bytes."""
    if encoding == "bf16_le":
        return codes.view(torch.bfloat16).reshape(experts, rows, k).float()
    raw = codes.view(torch.uint8).reshape(-1)
    if encoding == "q4_group128":
        q = torch.stack((raw & 15, raw >> 4), dim=1).reshape(-1).to(torch.int16)
        scales = scales.to(torch.bfloat16).float()                      # the kernels multiply by the BF16 scale
    else:
        q = raw.to(torch.int16)
    half, full = (8, 16) if encoding == "q4_group128" else (128, 256)
    q = torch.where(q >= half, q - full, q).float().reshape(-1, 128)
    return (q * scales.reshape(-1, 1)).to(torch.bfloat16).float().reshape(experts, rows, k)


def _reference_layer(layer, x, expert, weight):
    """float32 sums over the same BF16 operands, with the kernels' two roundings; one route per token."""
    e, h, i = layer.num_experts, layer.hidden, layer.intermediate
    gate = _dequantised(layer.gate, layer.gate_scales, layer.encoding, e, i, h)
    up = _dequantised(layer.up, layer.up_scales, layer.encoding, e, i, h)
    down = _dequantised(layer.down, layer.down_scales, layer.encoding, e, h, i)
    out = torch.zeros(x.shape, dtype=torch.bfloat16, device=x.device)
    for n in range(e):
        rows = (expert == n).nonzero().flatten()
        if len(rows):
            xr = x[rows].double()
            inter = (torch.nn.functional.silu(xr @ gate[n].double().T) * (xr @ up[n].double().T)).to(torch.bfloat16)
            out[rows] = ((inter.double() @ down[n].double().T) * weight[rows, None]).to(torch.bfloat16)
    return out


@pytest.mark.parametrize("model", ["olmoe", "qwen"])
@pytest.mark.parametrize("encoding", ["q4_group128", "q8_group128", "bf16_le"])
@pytest.mark.parametrize("counts", [[1], [2, 0, 15], [16, 17, 1, 31, 33, 63, 64, 65], [129, 0, 7] * 4, [300, 1, 192]])
def test_few_routes_per_expert_at_tile_edges(model, encoding, counts):
    """Route counts around the MMA's N steps (16) and the tile (64), absent experts, experts with several tiles.  Both sides
    round the intermediate and the output to BF16 once: they differ where a float32 sum falls on the other side of a
    rounding boundary, by 2^-8 of the value, and by 2^-8 of single terms of a sum; a misplaced row or column is off by
    the whole value."""
    from uma_qmoe_b200.stack import random_layer
    shape = syn.OLMOE if model == "olmoe" else syn.QWEN
    layer = random_layer(shape, encoding, 3, torch.device(DEV))
    gen = torch.Generator(device=DEV).manual_seed(sum(counts))
    expert = torch.cat([torch.full((c,), (11 * n) % shape.experts, device=DEV) for n, c in enumerate(counts)])
    expert = expert[torch.randperm(len(expert), device=DEV, generator=gen)]
    x = torch.randn(len(expert), shape.hidden, device=DEV, generator=gen).to(torch.bfloat16)
    w = torch.rand(len(expert), 1, device=DEV, generator=gen) + 0.1
    got = _run_prefill(layer, x, expert[:, None], w).float()
    want = _reference_layer(layer, x, expert, w[:, 0]).cpu().float()
    assert (got - want).norm() <= 2.0 ** -8 * want.norm()
    assert (got - want).abs().max() <= 2.0 ** -7 * want.abs().max()


@pytest.mark.parametrize("encoding,tokens", [("q4_group128", 520), ("q4_group128", 704), ("q4_group128", 705),
                                             ("q8_group128", 608), ("q8_group128", 609)])
def test_top_8_prompts_around_the_line_match_float64(encoding, tokens):
    """Prompts whose routes are sorted by several CTAs into a table of 64-route tiles (and just above the line of 256-route
    ones), with a skewed choice of experts, absent routes and real weights.  Against :func:`_reference_layer` per route and the
    ordered BF16 sum: 16 roundings per value, each off by one at the rare sum on a boundary; a misplaced row is off by itself."""
    from uma_qmoe_b200.stack import random_layer
    layer = random_layer(syn.OLMOE, encoding, 9, torch.device(DEV))
    gen = torch.Generator(device=DEV).manual_seed(tokens)
    popularity = 1.0 / torch.arange(1, 65, device=DEV, dtype=torch.float32) ** 0.5
    idx = torch.multinomial(popularity.expand(tokens, 64), 8, generator=gen)
    idx[torch.rand(tokens, 8, device=DEV, generator=gen) < 0.02] = -1
    x = torch.randn(tokens, 2048, device=DEV, generator=gen).to(torch.bfloat16)
    w = torch.rand(tokens, 8, device=DEV, generator=gen) + 0.1
    got = _run_prefill(layer, x, idx, w).float()
    per_route = _reference_layer(layer, x.repeat_interleave(8, 0), idx.reshape(-1), w.reshape(-1)).reshape(tokens, 8, 2048)
    order = torch.where(idx < 0, 64, idx).argsort(1)                        # ascending expert; absent routes are zero rows
    want = torch.zeros(tokens, 2048, device=DEV, dtype=torch.bfloat16)
    for slot in range(8):
        want = want + per_route[torch.arange(tokens, device=DEV), order[:, slot]]
    want = want.cpu().float()
    assert (got - want).norm() <= 2.0 ** -7 * want.norm()
    assert (got - want).abs().max() <= 2.0 ** -5 * want.abs().max()


def test_few_routes_kernel_takes_tables_of_wider_tiles():
    """The exported stage calls hand the transposed kernel tables of up to 256 routes per entry: it cuts them itself, and a
    gathered copy of the rows gives the bits that rows fetched by index give."""
    from uma_qmoe_b200 import ops
    from uma_qmoe_b200.stack import random_layer
    layer = random_layer(syn.OLMOE, "q4_group128", 4, torch.device(DEV))
    gen = torch.Generator(device=DEV).manual_seed(2)
    counts = [256, 257, 100, 64, 1, 80]
    idx = torch.cat([torch.full((c, 1), 5 * n, device=DEV) for n, c in enumerate(counts)])
    x = torch.randn(len(idx), 2048, device=DEV, generator=gen).to(torch.bfloat16)
    w = torch.rand(len(idx), 1, device=DEV, generator=gen)
    routes = ops.route_sort(idx, w, 64)
    xp = ops.gather_rows(x, None, 1, permute=True)
    xs = ops.gather_rows(x, routes.sorted_route, 1, permute=True)
    inter = ops.grouped_gemm_by_index(layer, xp, routes, 1, permute_out=True)
    assert torch.equal(inter, ops.grouped_gemm(layer, 0, xs, routes, permute_out=True))
    y = ops.grouped_gemm(layer, 1, inter, routes, routes.sorted_weight)
    assert torch.equal(ops.combine_routes(y, idx, routes.route_pos).cpu(), _run_prefill(layer, x, idx, w))


@pytest.mark.parametrize("tokens", [1, 5, 63, 192, 193, 448, 449, 600, 1030])
def test_shared_expert_in_parts_of_its_contraction(tokens):
    """The shared expert's down GEMM cut along k: eight parts, an uneven last part (600 tokens: 88 steps in six), the
    transposed kernel and the wide one.  The routes weigh nothing, so the result is the shared expert's; rounding as above
    and once more for the gate."""
    from uma_qmoe_b200.stack import random_layer, random_shared_expert
    dev = torch.device(DEV)
    layer, sh = random_layer(syn.QWEN, "q4_group128", 6, dev), random_shared_expert(syn.QWEN, 6, dev)
    gen = torch.Generator(device=DEV).manual_seed(tokens)
    x = torch.randn(tokens, 2048, device=DEV, generator=gen).to(torch.bfloat16)
    idx = torch.arange(tokens * 4, device=DEV).reshape(tokens, 4) % 60
    got = _run_prefill(layer, x, idx, torch.zeros(tokens, 4, device=DEV), sh).float()
    xd = x.double()
    inter = (torch.nn.functional.silu(xd @ sh.gate.double().T) * (xd @ sh.up.double().T)).to(torch.bfloat16)
    y = (inter.double() @ sh.down.double().T).to(torch.bfloat16)
    gate = torch.sigmoid((xd @ sh.gate_vec.reshape(-1).double()).to(torch.bfloat16).float()).to(torch.bfloat16)
    want = (gate[:, None] * y).cpu().float()
    assert (got - want).norm() <= 2.0 ** -7 * want.norm()
    assert (got - want).abs().max() <= 2.0 ** -6 * want.abs().max()


@pytest.mark.parametrize("hidden,encoding,tokens", [(1024, "q4_group128", 1400), (1024, "q4_group128", 449), (512, "q8_group128", 2100),
                                                    (4096, "bf16_le", 5), (4096, "bf16_le", 300)])
def test_shared_expert_in_parts_at_other_hidden_sizes(hidden, encoding, tokens):
    """As above where the parts' room is another: six parts of 1400 tokens at hidden 1024, eight of 2100 at 512, eight of 5 and
    one of 300 at 4096.  The bounds are those of :func:`test_shared_expert_in_parts_of_its_contraction`: the same roundings."""
    from dataclasses import replace
    from uma_qmoe_b200.stack import random_layer, random_shared_expert
    dev, shape = torch.device(DEV), replace(syn.QWEN, hidden=hidden, experts=6)
    layer, sh = random_layer(shape, encoding, 7, dev), random_shared_expert(shape, 7, dev)
    gen = torch.Generator(device=DEV).manual_seed(tokens)
    x = torch.randn(tokens, hidden, device=DEV, generator=gen).to(torch.bfloat16)
    idx = torch.arange(tokens * 4, device=DEV).reshape(tokens, 4) % 6
    got = _run_prefill(layer, x, idx, torch.zeros(tokens, 4, device=DEV), sh).float()
    xd = x.double()
    inter = (torch.nn.functional.silu(xd @ sh.gate.double().T) * (xd @ sh.up.double().T)).to(torch.bfloat16)
    y = (inter.double() @ sh.down.double().T).to(torch.bfloat16)
    gate = torch.sigmoid((xd @ sh.gate_vec.reshape(-1).double()).to(torch.bfloat16).float()).to(torch.bfloat16)
    want = (gate[:, None] * y).cpu().float()
    assert (got - want).norm() <= 2.0 ** -7 * want.norm()
    assert (got - want).abs().max() <= 2.0 ** -6 * want.abs().max()


def _kernels(call, tmp_path):
    """Which grouped GEMM kernels a call launches, from the nodes of a graph it is captured into."""
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        call()                                                   # whatever a first call sets up, outside the capture
        graph = torch.cuda.CUDAGraph(keep_graph=True)
        graph.enable_debug_mode()
        with torch.cuda.graph(graph, stream=stream):
            call()
    graph.debug_dump(str(tmp_path / "graph.dot"))
    text = (tmp_path / "graph.dot").read_text()
    names = ("grouped_gemm_kernel", "grouped_pair_kernel", "grouped_ts_kernel")
    assert any(name in text for name in names), text[:2000]
    return {name for name in names if name in text}


@pytest.mark.parametrize("encoding,line", [("q4_group128", 88), ("q8_group128", 76), ("bf16_le", 64)])
def test_variants_name_their_kernels_on_both_sides_of_the_line(encoding, line, tmp_path):
    """Variants 1, 2 and 3 run the kernel they name at any size, variant 0 changes over at `line` routes per expert.  One-CTA
    and transposed tiles multiply the same BF16 operands and add the same 16-k steps in the same order: equal bits."""
    from uma_qmoe_b200 import ops
    from uma_qmoe_b200.stack import random_layer
    layer = random_layer(syn.OLMOE, encoding, 8, torch.device(DEV), experts=range(16))
    gen = torch.Generator(device=DEV).manual_seed(line)
    quant = encoding != "bf16_le"
    for routes in (16 * line, 16 * line + 1):
        idx = (torch.arange(routes, device=DEV) % 16)[:, None]
        x = torch.randn(routes, 2048, device=DEV, generator=gen).to(torch.bfloat16)
        w = torch.rand(routes, 1, device=DEV, generator=gen)
        inter1, y1 = _stagewise(layer, x, idx, w, variant=1)
        inter3, y3 = _stagewise(layer, x, idx, w, variant=3)
        assert torch.equal(inter1, inter3) and torch.equal(y1, y3)
        one_cta, pair, transposed = {"grouped_gemm_kernel"}, {"grouped_pair_kernel"}, {"grouped_ts_kernel"}
        by_size = one_cta | transposed if routes == 16 * line else one_cta        # below the line the counts decide
        for variant, want in enumerate((by_size, one_cta, pair, transposed)):
            assert _kernels(lambda: _stagewise_launches(layer, x, idx, w, variant), tmp_path) == want, (routes, variant)
        source = ops.gather_rows(x, None, 1, permute=True) if quant else x
        table = ops.route_sort(idx, w, layer.num_experts)
        assert _kernels(lambda: ops.grouped_gemm_by_index(layer, source, table, 1, permute_out=quant), tmp_path) == by_size


def _stagewise_launches(layer, x, idx, w, variant):
    """:func:`_stagewise` without its checks, so that it can be captured."""
    from uma_qmoe_b200 import ops
    r = ops.route_sort(idx, w, layer.num_experts)
    xs = ops.gather_rows(x, r.sorted_route, idx.shape[1], permute=layer.encoding != "bf16_le")
    inter = ops.grouped_gemm(layer, 0, xs, r, permute_out=layer.encoding != "bf16_le", variant=variant)
    return ops.grouped_gemm(layer, 1, inter, r, route_weight=r.sorted_weight, variant=variant)


@pytest.mark.parametrize("model,encoding,tokens", [("olmoe", "q4_group128", 384), ("olmoe", "q4_group128", 704),
                                                   ("olmoe", "q8_group128", 512), ("olmoe", "bf16_le", 224), ("olmoe", "bf16_le", 512),
                                                   ("qwen", "q8_group128", 960), ("qwen", "bf16_le", 900)])
def test_concentrated_routes_take_the_one_cta_kernel(model, encoding, tokens):
    """Below the line of routes per expert the kernel is picked from the counts on the device: few experts in use -> one-CTA
    tiles, all of them -> transposed ones.  Either way and through the exported stages (which pick from the table), the bits are
    those of the stages run on the one-CTA kernel; an absent route counts like one that weighs nothing."""
    from uma_qmoe_b200 import ops
    from uma_qmoe_b200.stack import random_layer
    shape = syn.OLMOE if model == "olmoe" else syn.QWEN
    layer = random_layer(shape, encoding, 5, torch.device(DEV))
    gen = torch.Generator(device=DEV).manual_seed(tokens)
    k = shape.top_k
    x = torch.randn(tokens, shape.hidden, device=DEV, generator=gen).to(torch.bfloat16)
    w = torch.rand(tokens, k, device=DEV, generator=gen)
    spread = (torch.arange(tokens * k, device=DEV) % shape.experts).reshape(tokens, k)     # as even as routes can be
    narrow = (torch.arange(tokens * k, device=DEV) % (k + k // 2)).reshape(tokens, k)
    absent = spread.clone()
    absent[::3, 1] = -1
    present = torch.where(absent >= 0, w, 0.0)
    for idx, routes, weights, transposed in ((narrow, narrow, w, 0), (spread, spread, w, 1), (absent, spread, present, None)):
        ws = ops.prefill_workspace(layer, tokens, k, None, torch.device(DEV))
        y = ops.moe_prefill(layer, x, idx, w, ws)
        assert ops.prefill_status(ws) == 0
        if transposed is not None:
            assert int(ws[64:68].view(torch.int32).item()) == transposed
        _, want = _stagewise(layer, x, routes, weights, variant=1)       # the gather stage takes present routes only
        assert torch.equal(y, want)
        _, picked = _stagewise(layer, x, routes, weights, variant=0)
        assert torch.equal(picked, want)


def test_a_failed_launch_is_reported_once():
    """A launch that the runtime refuses (into the legacy stream while a blocking stream is being captured: an error on the host,
    nothing runs) fails its own call and no later one."""
    import ctypes as C
    from uma_qmoe_b200 import _native, ops
    runtime = C.CDLL("libcudart.so.12")
    x = torch.zeros(1, 2048, dtype=torch.bfloat16, device=DEV)
    idx = torch.zeros(1, 1, dtype=torch.int32, device=DEV)
    pos, out = torch.zeros(1, dtype=torch.int32, device=DEV), torch.empty_like(x)
    combine = lambda: _native.lib().umaq_combine_routes(x.data_ptr(), idx.data_ptr(), 0, pos.data_ptr(), 1, 1, 2048,
                                                        out.data_ptr(), None)
    torch.cuda.synchronize()
    stream, graph = C.c_void_p(), C.c_void_p()
    assert runtime.cudaStreamCreate(C.byref(stream)) == 0
    try:
        assert runtime.cudaStreamBeginCapture(stream, 2) == 0
        refused = combine()
        runtime.cudaStreamEndCapture(stream, C.byref(graph))         # invalidated by the refused launch
    finally:
        runtime.cudaStreamDestroy(stream)
        runtime.cudaGetLastError()
    assert refused != 0
    ops.quantize_groups(x.reshape(-1), "q4_group128")
    assert combine() == 0
    torch.cuda.synchronize()


@pytest.mark.parametrize("encoding", ["q4_group128", "q8_group128"])
def test_wide_packed_linear_takes_the_one_cta_kernel_above_one_tile(encoding, tmp_path):
    """A single matrix of many columns: two transposed tiles would take twice the waves of a one-CTA tile.  Narrow ones and
    64 rows keep the transposed kernel; the bits are the same."""
    from uma_qmoe_b200 import ops
    from uma_qmoe_b200.ops import DeviceLayer
    gen = torch.Generator(device=DEV).manual_seed(4)
    for out, rows, want in ((32768, 64, "grouped_ts_kernel"), (32768, 65, "grouped_gemm_kernel"), (2048, 65, "grouped_ts_kernel")):
        codes, scales = ops.quantize_groups((torch.randn(out * 256, device=DEV, generator=gen) * 0.02).to(torch.bfloat16), encoding)
        layer = DeviceLayer(encoding, 1, out, 256, codes, codes, codes, scales, scales, scales)
        x = torch.randn(rows, 256, device=DEV, generator=gen).to(torch.bfloat16)
        routes = ops.route_sort(torch.zeros(rows, 1, dtype=torch.int32, device=DEV), torch.ones(rows, 1, device=DEV), 1)
        assert _kernels(lambda: ops.grouped_gemm(layer, 1, x, routes), tmp_path) == {want}
        assert torch.equal(ops.grouped_gemm(layer, 1, x, routes), ops.grouped_gemm(layer, 1, x, routes, variant=1))
