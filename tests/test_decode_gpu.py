"""Batch-1 decode kernel vs the CPU oracle and the reference-made golden vectors (through the C ABI)."""

import numpy as np
import pytest
import torch

from oracle import moe_oracle as orc
from tests.helpers import SEED, assert_parity, bits_to_bf16, expert_source, stage_layer
from uma_qmoe_b200 import synthetic as syn

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _ops():
    from uma_qmoe_b200 import ops
    return ops


def _run_decode(layer, x, idx, w, shared=None):
    ops = _ops()
    ws = ops.decode_workspace(layer, idx.numel(), shared, torch.device(DEV))
    y = ops.moe_decode(layer, x.to(DEV).contiguous(), idx.to(DEV).contiguous(), w.to(DEV).contiguous(), ws, shared)
    y2 = ops.moe_decode(layer, x.to(DEV).contiguous(), idx.to(DEV).contiguous(), w.to(DEV).contiguous(), ws, shared)
    torch.cuda.synchronize()
    assert ops.workspace_status(ws) == 0
    assert torch.equal(y, y2), "two calls on one workspace must give identical bits"
    return y.cpu()


def test_device_packer_bit_exact():
    ops = _ops()
    v = torch.from_numpy(syn.normal_bf16((SEED, 77), (64, 1024), 0.02))
    v[3, :128] = 0.0
    v[5, 128:256] = 1e-30
    vb = v.to(torch.bfloat16)
    for enc, ref in (("q4_group128", orc.quantize_q4), ("q8_group128", orc.quantize_q8)):
        codes, scales = ops.quantize_groups(vb.to(DEV), enc)
        want_codes, want_scales = ref(vb.float().numpy())
        assert np.array_equal(codes.cpu().numpy().view(np.uint8), np.asarray(want_codes).view(np.uint8)), enc
        assert np.array_equal(scales.cpu().numpy(), want_scales), enc


@pytest.mark.parametrize("enc", ["q4_group128", "q8_group128"])
@pytest.mark.parametrize("groups,offset", [(1, 0), (7, 4), (64, 8), (131, 0), (1029, 4)])
def test_device_packer_rounding_boundaries_and_layouts(enc, groups, offset):
    """Ties and their neighbours, subnormal groups and chunks of a fused tensor; 8- and 16-byte aligned sources, group
    counts around a block's 64: bit-exact against the oracle, which divides."""
    ops = _ops()
    quant, qmax = (orc.quantize_q4, 7) if enc == "q4_group128" else (orc.quantize_q8, 127)
    rng = np.random.default_rng(groups)
    n = groups * 128
    v = torch.from_numpy(rng.standard_normal((2, n)).astype(np.float32)).to(torch.bfloat16)
    flat = v.reshape(-1, 128)
    for g in range(0, len(flat), 3):                         # scale a power of two: (k + 1/2) * scale is a tie
        half = torch.from_numpy((rng.integers(-2 * qmax, 2 * qmax + 1, 128) / 2).astype(np.float32))
        half[5] = qmax
        flat[g] = (half * 2.0 ** int(rng.integers(-20, 20))).to(torch.bfloat16)
    flat[1] = (flat[1].float() * 2.0 ** -127).to(torch.bfloat16)        # subnormal weights and scale
    want = [quant(part.float().numpy()) for part in v]
    store = torch.zeros(offset + 2 * (n + 128), dtype=torch.bfloat16, device=DEV)
    chunks = torch.as_strided(store, (2, groups, 128), (n + 128, 128, 1), offset)
    chunks.copy_(v.reshape(2, groups, 128))
    for codes, scales in (ops.quantize_chunks(chunks, enc), ops.quantize_groups(chunks.contiguous(), enc)):
        got = codes.cpu().numpy().view(np.uint8)
        assert np.array_equal(got, np.concatenate([np.asarray(c).view(np.uint8).reshape(-1) for c, _ in want]))
        assert np.array_equal(scales.cpu().numpy(), np.concatenate([s for _, s in want]))


@pytest.mark.parametrize("enc", ["q4_group128", "q8_group128"])
@pytest.mark.parametrize("experts,offset,pad", [(3, 1, 0), (3, 2, 0), (3, 0, 1), (2, 3, 6), (1, 1, 0)])
def test_encode_experts_takes_any_offset_and_expert_stride(enc, experts, offset, pad):
    """A fused gate/up tensor that starts off an 8-byte boundary, or whose experts are padded to an odd stride, packs to the
    bytes of an aligned copy of it."""
    from uma_qmoe_b200.host import encode_experts
    hidden, inter = 256, 128
    gen = torch.Generator(device=DEV).manual_seed(offset + 8 * pad)
    def view(rows, k):
        store = torch.randn(offset + experts * (rows * k + pad), device=DEV, generator=gen).to(torch.bfloat16)
        return torch.as_strided(store, (experts, rows, k), (rows * k + pad, k, 1), offset)
    gate_up, down = view(2 * inter, hidden), view(hidden, inter)
    got = encode_experts(gate_up, down, enc)
    want = encode_experts(gate_up.clone(memory_format=torch.contiguous_format), down.clone(memory_format=torch.contiguous_format), enc)
    assert got.tensors and all(torch.equal(a, b) for a, b in zip(got.tensors, want.tensors))


@pytest.mark.parametrize("enc", ["q4_group128", "q8_group128"])
def test_device_packer_values_that_divide(enc):
    """Groups the quantiser divides for: an infinity, a NaN (fmax passes over it, its code is -qmax), maxima near the largest
    BF16 value, scales around 2^-100 and with the largest mantissas, next to ordinary groups in the other half of their warp."""
    ops, qmax = _ops(), 7 if enc == "q4_group128" else 127
    rng = np.random.default_rng(3)
    g = rng.standard_normal((64, 128)).astype(np.float32)
    g[1, 5], g[4, 0], g[4, 127], g[7, 9], g[8, :] = np.inf, -np.inf, np.inf, np.nan, np.nan
    g[10, 3], g[10, 4], g[13, 64] = np.nan, np.inf, -np.nan
    g[16] *= np.float32(3.3e38 / 4)
    g[19, 77] = np.float32(3.3895e38)                                       # the largest finite BF16 value
    for n, e in enumerate(range(-106, -94)):
        g[20 + 2 * n] *= np.float32(2.0 ** e)
    top = (1 + np.arange(128, dtype=np.float32) / 128) * 4                  # of every mantissa of the maximum, those with these scales
    for n in range(16):
        g[46 + n] = np.clip(g[46 + n], -3.9, 3.9)
        g[46 + n, n] = top[np.argsort((top / np.float32(qmax)).view(np.uint32) & 0x7fffff)[-1 - n]]
    v = torch.from_numpy(g).to(torch.bfloat16)
    f = v.float().numpy()
    with np.errstate(all="ignore"):
        am = np.where(np.isnan(f), np.float32(0), np.abs(f)).max(axis=1)
        scale = am / np.float32(qmax)
        scale[scale == 0] = 1
        q = np.rint(f / scale[:, None])
    q = np.clip(np.where(np.isnan(q), -qmax, q), -qmax, qmax).astype(np.int8)
    codes, scales = ops.quantize_groups(v.reshape(-1).to(DEV), enc)
    want = q.reshape(-1).view(np.uint8)
    if enc == "q4_group128":
        want = (want[0::2] & 15) | (want[1::2] << 4)
    assert np.array_equal(scales.cpu().numpy(), scale)
    assert np.array_equal(codes.cpu().numpy().view(np.uint8), want)


@pytest.mark.parametrize("enc", ["q4_group128", "q8_group128"])
def test_device_packer_every_ratio_of_bf16_mantissas(enc):
    """Every BF16 mantissa against every BF16 maximum over the exponents whose codes are not all zero: every quotient a group
    of normal weights can have, exact ties between two codes among them."""
    ops = _ops()
    quant = orc.quantize_q4 if enc == "q4_group128" else orc.quantize_q8
    m = 1 + np.arange(128, dtype=np.float32) / 128
    rows = []
    for am in m:
        for e in range(10):
            g = m * np.float32(2.0 ** -e)
            g[g > am] /= 2
            rows.append(np.concatenate(([am], g[1:])).astype(np.float32))
            rows.append(np.concatenate(([am], -g[:-1])).astype(np.float32))
    v = torch.from_numpy(np.stack(rows)).to(torch.bfloat16)
    assert np.array_equal(v.float().numpy(), np.stack(rows))
    codes, scales = ops.quantize_groups((v * 2.0 ** -7).to(DEV), enc)
    want_codes, want_scales = quant(v.float().numpy() * np.float32(2.0 ** -7))
    assert np.array_equal(codes.cpu().numpy().view(np.uint8), np.asarray(want_codes).view(np.uint8).reshape(-1))
    assert np.array_equal(scales.cpu().numpy(), want_scales)


def test_olmoe_decode_golden(golden_dir):
    g = np.load(golden_dir / "olmoe_decode.npz")
    x = bits_to_bf16(g["x_bits"])
    idx = torch.from_numpy(g["idx"])
    src = expert_source(SEED, 0, "olmoe", "q4_group128")
    experts = {int(e): src(int(e)) for e in set(idx.reshape(-1).tolist())}
    layer = stage_layer(experts, 64, 2048, 1024, "q4_group128", DEV)
    for wkey, ykey in (("w_norm", "y_norm_bits"), ("w_raw", "y_raw_bits")):
        y = _run_decode(layer, x, idx, torch.from_numpy(g[wkey]))
        m = assert_parity(y, bits_to_bf16(g[ykey]))
        assert m["max_abs"] <= 4e-3, m          # the kernel keeps the oracle's rounding points


def test_olmoe_decode_int32_duplicate_and_order():
    src = expert_source(SEED, 5, "olmoe", "q4_group128")
    idx = torch.tensor([[9, 2, 2, 7, 0, 11, 4, 1]], dtype=torch.int32)
    w = torch.tensor([[0.3, 0.05, 0.1, 0.2, 0.05, 0.1, 0.15, 0.05]])
    experts = {int(e): src(int(e)) for e in set(idx.reshape(-1).tolist())}
    layer = stage_layer(experts, 16, 2048, 1024, "q4_group128", DEV)
    x = syn.activations(SEED + 11, 1)
    want = orc.moe_forward(x, idx.long(), w, src, num_experts=64, top_k=8, qwen=False)
    assert_parity(_run_decode(layer, x, idx, w), want)


@pytest.mark.parametrize("encoding", ["q8_group128", "bf16_le"])
def test_olmoe_shape_other_encodings(encoding):
    src = expert_source(SEED, 6, "olmoe", encoding)
    idx = torch.tensor([[3, 1, 0, 2, 5, 4, 7, 6]])
    w = torch.full((1, 8), 0.125)
    layer = stage_layer({e: src(e) for e in range(8)}, 8, 2048, 1024, encoding, DEV)
    x = syn.activations(SEED + 12, 1)
    want = orc.moe_forward(x, idx, w, src, num_experts=64, top_k=8, qwen=False)
    assert_parity(_run_decode(layer, x, idx, w), want)


def test_large_activations_do_not_overflow():
    src = expert_source(SEED, 6, "olmoe", "q4_group128")
    idx = torch.tensor([[3, 1, 0, 2, 5, 4, 7, 6]])
    w = torch.full((1, 8), 0.125)
    layer = stage_layer({e: src(e) for e in range(8)}, 8, 2048, 1024, "q4_group128", DEV)
    x = (syn.activations(SEED + 13, 1).float() * 3000.0).to(torch.bfloat16)
    want = orc.moe_forward(x, idx, w, src, num_experts=64, top_k=8, qwen=False)
    got = _run_decode(layer, x, idx, w)
    m = orc.compare(got, want)
    assert m["cosine"] >= 0.9999 and torch.isfinite(got.float()).all(), m


@pytest.mark.parametrize("layer_index", [0, 1, 2])
def test_qwen_decode_golden(golden_dir, layer_index):
    from uma_qmoe_b200.ops import DeviceSharedExpert
    g = np.load(golden_dir / "qwen_layers.npz")
    enc = str(g[f"L{layer_index}_encoding"])
    src = expert_source(SEED, layer_index, "qwen", enc)
    x = bits_to_bf16(g["x1_bits"])
    idx = torch.from_numpy(g[f"L{layer_index}_i1"])
    w = torch.from_numpy(g[f"L{layer_index}_w1"])
    experts = {int(e): src(int(e)) for e in set(idx.reshape(-1).tolist())}
    layer = stage_layer(experts, 60, 2048, 1408, enc, DEV)
    y = _run_decode(layer, x, idx, w)
    assert_parity(y, bits_to_bf16(g[f"L{layer_index}_y1_bits"]))
    sg, su, sd, sgate = (t.to(DEV).contiguous() for t in syn.shared_expert_weights(SEED, layer_index, syn.QWEN))
    shared = DeviceSharedExpert(sg, su, sd, sgate)
    b = _run_decode(layer, x, idx, w, shared)
    assert_parity(b, bits_to_bf16(g[f"L{layer_index}_b1_bits"]))


def test_bad_expert_index_sets_status_and_does_not_hang():
    ops = _ops()
    src = expert_source(SEED, 6, "olmoe", "q4_group128")
    layer = stage_layer({0: src(0)}, 4, 2048, 1024, "q4_group128", DEV)
    ws = ops.decode_workspace(layer, 8, None, torch.device(DEV))
    idx = torch.tensor([[0, 1, 2, 3, 0, 1, 2, 99]], device=DEV)
    ops.moe_decode(layer, syn.activations(1, 1).to(DEV), idx, torch.full((1, 8), 0.125, device=DEV), ws)
    torch.cuda.synchronize()
    assert ops.workspace_status(ws) == -1


def test_rejects_cpu_tensors_and_bad_shapes():
    ops = _ops()
    src = expert_source(SEED, 6, "olmoe", "q4_group128")
    layer = stage_layer({0: src(0)}, 1, 2048, 1024, "q4_group128", DEV)
    ws = ops.decode_workspace(layer, 8, None, torch.device(DEV))
    idx = torch.zeros((1, 8), dtype=torch.int64, device=DEV)
    w = torch.full((1, 8), 0.125, device=DEV)
    with pytest.raises(RuntimeError):
        ops.moe_decode(layer, syn.activations(1, 1), idx, w, ws)               # CPU tensor: no fallback
    with pytest.raises(RuntimeError):
        ops.moe_decode(layer, syn.activations(1, 2).to(DEV), idx, w, ws)       # two tokens
    with pytest.raises(RuntimeError):
        ops.moe_decode(layer, syn.activations(1, 1).to(DEV), idx, w, ws[:64])  # workspace too small


def test_reference_validator_and_route_trace_decode(golden_dir):
    """One token of the reference validator's inputs (linspace hidden state, experts 0..7, weights 0.125) and the
    first decode event of layer 0 of the reference's frozen route trace, against the reference's CPU outputs."""
    g = np.load(golden_dir / "reference_cases.npz")
    src = expert_source(SEED, int(g["layer"]), "olmoe", "q4_group128")
    layer = stage_layer({int(e): src(int(e)) for e in g["hit"]}, 64, 2048, 1024, "q4_group128", DEV)
    y = _run_decode(layer, bits_to_bf16(g["val_x1_bits"]), torch.from_numpy(g["val_idx"]),
                    bits_to_bf16(g["val_w_bits"]).float())
    assert_parity(y, bits_to_bf16(g["val_y1_bits"]))
    y = _run_decode(layer, bits_to_bf16(g["trace_decode_x_bits"]), torch.from_numpy(g["trace_decode_idx"]),
                    torch.from_numpy(g["trace_decode_w"]))
    assert_parity(y, bits_to_bf16(g["trace_decode_y_bits"]))


def test_bad_expert_index_is_skipped_like_the_reference():
    """An out-of-range index contributes nothing (the reference's kernels skip it,
    src/uma_qmoe/native/packed_q4_kernel.cu:176); the other routes still produce the complete output."""
    ops = _ops()
    src = expert_source(SEED, 6, "olmoe", "q4_group128")
    layer = stage_layer({e: src(e) for e in range(4)}, 4, 2048, 1024, "q4_group128", DEV)
    x = syn.activations(SEED + 14, 1)
    idx = torch.tensor([[0, 1, 2, 3, 0, 1, 2, 99]])
    w = torch.full((1, 8), 0.125)
    ws = ops.decode_workspace(layer, 8, None, torch.device(DEV))
    y = ops.moe_decode(layer, x.to(DEV), idx.to(DEV), w.to(DEV), ws).cpu()
    torch.cuda.synchronize()
    assert ops.workspace_status(ws) == -1
    want = orc.moe_forward(x, idx[:, :7].contiguous(), w[:, :7].contiguous(), src, num_experts=64, top_k=7, qwen=False)
    assert_parity(y, want)
