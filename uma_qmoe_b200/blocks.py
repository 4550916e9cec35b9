"""Drop-in MoE blocks with the constructor signatures of the reference's
``QuantizedMoEBlock`` (``src/uma_qmoe/compressed_loader.py:41-67``) and
``QuantizedQwenMoEBlock`` (``src/uma_qmoe/qwen_compressed_loader.py:46-86``).

They run what the ``torch.ops.uma_qmoe`` operators run, with the path around it fused: the router
(softmax / top-k / renormalisation) is one kernel, for Qwen the shared expert, its sigmoid gate and the
final add run inside the expert kernels instead of as separate cuBLAS and element-wise launches, and the
back end issues all of it from one native call.  Where the OLMoE operator would be seen (dispatch modes,
profilers, autograd) the block calls the router and the operator one after the other, with the same bits.
"""

from __future__ import annotations

from typing import Any

import torch

from . import ops
from .custom_op import _backend_for, acquire_expert_pack, platform_of
from .ops import DeviceSharedExpert


def _router_params(gate: Any) -> tuple[torch.Tensor, int, bool]:
    return gate.weight, int(gate.top_k), bool(getattr(gate, "norm_topk_prob", False))


def _unobserved(hidden: torch.Tensor) -> bool:
    """Nobody looks at the operators of this call: no dispatch mode or tensor subclass, no profiler, no autograd history to keep."""
    return (type(hidden) is torch.Tensor and not torch._C._len_torch_dispatch_stack()
            and not torch.autograd._profiler_enabled() and not (hidden.requires_grad and torch.is_grad_enabled()))


class QuantizedMoEBlock(torch.nn.Module):
    """OLMoE router plus the compressed routed experts."""

    def __init__(self, gate: Any, *, layer_index: int, pack_handle: int, performance_mode: bool) -> None:
        super().__init__()
        self.gate = gate
        self.layer_index = layer_index
        self.pack_handle = pack_handle
        self.performance_mode = performance_mode

    def forward(self, hidden_states: torch.Tensor) -> torch.Tensor:
        weight, top_k, renorm = _router_params(self.gate)
        flat = hidden_states.reshape(-1, hidden_states.shape[-1])
        whole = getattr(_backend_for(platform_of(torch, flat)), "block_forward", None)
        if callable(whole) and _unobserved(flat):             # router and experts in one native call
            with acquire_expert_pack(self.pack_handle):
                return whole("olmoe", flat, weight, top_k, renorm, self.layer_index, self.pack_handle).view(hidden_states.shape)
        routing_weights, selected = ops.route_topk(flat, weight, top_k, renorm)
        return torch.ops.uma_qmoe.moe_forward(hidden_states, selected, routing_weights, self.layer_index,
                                              self.pack_handle, self.performance_mode)


class QuantizedQwenMoEBlock(torch.nn.Module):
    """Qwen router, shared expert and sigmoid gate fused around the packed routed experts."""

    def __init__(self, gate: Any, shared_expert: Any, shared_expert_gate: Any, *, layer_index: int,
                 pack_handle: int, performance_mode: bool) -> None:
        super().__init__()
        self.gate = gate
        self.shared_expert = shared_expert
        self.shared_expert_gate = shared_expert_gate
        self.layer_index = layer_index
        self.pack_handle = pack_handle
        self.performance_mode = performance_mode

    def _shared(self) -> DeviceSharedExpert:
        se = self.shared_expert
        return DeviceSharedExpert(se.gate_proj.weight, se.up_proj.weight, se.down_proj.weight,
                                  self.shared_expert_gate.weight)

    def forward(self, hidden_states: torch.Tensor) -> torch.Tensor:
        batch, seq, hidden = hidden_states.shape
        flat = hidden_states.reshape(-1, hidden)
        weight, top_k, renorm = _router_params(self.gate)
        backend = _backend_for(platform_of(torch, flat))
        whole = getattr(backend, "block_forward", None)
        if callable(whole):                       # router, experts and shared expert in one native call
            with acquire_expert_pack(self.pack_handle):
                return whole("qwen", flat, weight, top_k, renorm, self.layer_index, self.pack_handle,
                             self._shared()).view(batch, seq, hidden)
        routing_weights, selected = ops.route_topk(flat, weight, top_k, renorm)
        fused = getattr(backend, "qwen_block_forward", None)
        if not callable(fused):
            raise RuntimeError("performance mode has no Qwen-capable backend with a fused shared expert; "
                               "silent reference fallback is forbidden")
        with acquire_expert_pack(self.pack_handle):
            out = fused(flat, selected, routing_weights, self.layer_index, self.pack_handle, self._shared())
        return out.reshape(batch, seq, hidden)
