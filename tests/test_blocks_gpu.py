"""The blocks' one native call against the router and the operator called one after the other."""

from types import SimpleNamespace

import pytest
import torch

from uma_qmoe_b200 import custom_op, native_backend, ops, synthetic as syn
from uma_qmoe_b200.blocks import QuantizedMoEBlock, QuantizedQwenMoEBlock
from uma_qmoe_b200.packs import InMemoryPack
from uma_qmoe_b200.stack import random_layer, random_shared_expert

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("model", ["olmoe", "qwen"])
@pytest.mark.parametrize("tokens", [1, 9, 300])
def test_block_gives_the_bits_of_router_and_operator(model, tokens):
    """Also on a stream of its own, in a graph, and after a larger call on the same workspace."""
    shape = syn.OLMOE if model == "olmoe" else syn.QWEN
    backend = native_backend.install_mixed_target_backend()
    handle = custom_op.register_target_pack(InMemoryPack({0: "q8_group128"}))
    try:
        backend.preload_layer(handle, 0, DEV, random_layer(shape, "q8_group128", 3, DEV))
        gate = SimpleNamespace(weight=syn.router_weight(1, 0, shape, skew=1.0).to(DEV), top_k=shape.top_k, norm_topk_prob=False)
        args = dict(layer_index=0, pack_handle=handle, performance_mode=True)
        if model == "olmoe":
            block = QuantizedMoEBlock(gate, **args)
        else:
            w = random_shared_expert(shape, 5, DEV)
            linear = lambda t: SimpleNamespace(weight=t)
            shared = SimpleNamespace(gate_proj=linear(w.gate), up_proj=linear(w.up), down_proj=linear(w.down))
            block = QuantizedQwenMoEBlock(gate, shared, linear(w.gate_vec), **args)
        x = torch.randn(1, tokens, shape.hidden, device=DEV).to(torch.bfloat16)
        weights, selected = ops.route_topk(x.reshape(tokens, -1), gate.weight, shape.top_k, False)
        if model == "olmoe":
            want = torch.ops.uma_qmoe.moe_forward(x, selected, weights, 0, handle, True)
        else:
            want = backend.qwen_block_forward(x.reshape(tokens, -1), selected, weights, 0, handle, block._shared()).view(x.shape)
        block(torch.randn(1, 400, shape.hidden, device=DEV).to(torch.bfloat16))
        assert torch.equal(block(x), want)
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            assert torch.equal(block(x), want)
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=side):
                captured = block(x)
            graph.replay()
        side.synchronize()
        assert torch.equal(captured, want)
        with pytest.raises(RuntimeError):
            block(x[:, :0])
        backend.check_device_status()
    finally:
        custom_op.unregister_expert_pack(handle)
    with pytest.raises(RuntimeError, match="unknown or closed ExpertPack handle"):
        block(x)


@pytest.mark.parametrize("tokens", [1, 9])
def test_block_shows_its_operator_to_modes_profilers_and_autograd(tokens):
    from torch.utils._python_dispatch import TorchDispatchMode

    class Seen(TorchDispatchMode):
        def __init__(self):
            super().__init__()
            self.names = []

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            self.names.append(str(func))
            return func(*args, **(kwargs or {}))

    shape = syn.OLMOE
    backend = native_backend.install_mixed_target_backend()
    handle = custom_op.register_target_pack(InMemoryPack({0: "q4_group128"}))
    try:
        backend.preload_layer(handle, 0, DEV, random_layer(shape, "q4_group128", 3, DEV))
        gate = SimpleNamespace(weight=syn.router_weight(1, 0, shape, skew=1.0).to(DEV), top_k=8, norm_topk_prob=False)
        block = QuantizedMoEBlock(gate, layer_index=0, pack_handle=handle, performance_mode=True)
        x = torch.randn(1, tokens, shape.hidden, device=DEV).to(torch.bfloat16)
        want = block(x)
        with Seen() as seen:
            assert torch.equal(block(x), want)
        assert any(name.startswith("uma_qmoe.moe_forward") for name in seen.names)
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as profile:
            block(x)
        assert any(event.key == "uma_qmoe::moe_forward" for event in profile.key_averages())
        leaf = x.clone().requires_grad_()
        out = block(leaf)
        assert out.requires_grad and torch.equal(out.detach(), want)
        with torch.no_grad():
            assert not block(leaf).requires_grad
    finally:
        custom_op.unregister_expert_pack(handle)


@pytest.mark.parametrize("tokens", [1, 9, 300])
def test_block_takes_activations_that_start_anywhere(tokens):
    shape = syn.OLMOE
    backend = native_backend.install_mixed_target_backend()
    handle = custom_op.register_target_pack(InMemoryPack({0: "q4_group128"}))
    try:
        backend.preload_layer(handle, 0, DEV, random_layer(shape, "q4_group128", 3, DEV))
        gate = SimpleNamespace(weight=syn.router_weight(1, 0, shape, skew=1.0).to(DEV), top_k=8, norm_topk_prob=False)
        block = QuantizedMoEBlock(gate, layer_index=0, pack_handle=handle, performance_mode=True)
        x = torch.randn(1, tokens, shape.hidden, device=DEV).to(torch.bfloat16)
        want = block(x)
        shifted = torch.empty(x.numel() + 1, dtype=torch.bfloat16, device=DEV)[1:].view(x.shape).copy_(x)
        assert torch.equal(block(shifted), want)
        weights, selected = ops.route_topk(shifted.view(tokens, -1), gate.weight, 8, False)
        assert torch.equal(torch.ops.uma_qmoe.moe_forward(shifted, selected, weights, 0, handle, True), want)
    finally:
        custom_op.unregister_expert_pack(handle)
