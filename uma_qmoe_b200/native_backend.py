"""The sm_100a performance backend behind ``uma_qmoe::moe_forward`` /
``uma_qmoe::qwen_moe_forward``.

Same public surface as the reference's ``src/uma_qmoe/native_backend.py``
(``PackedQ4NativeBackend``, ``MixedTargetNativeBackend``,
``install_packed_q4_backend``, ``install_mixed_target_backend``,
``load_native_extension``, ``native_kernel_source_sha256``,
``observed_native_platform``; ``cache_summary()`` keys ``:457-467``;
``release_pack`` ``:469-480``), but the native side is ``libumaq_b200.so``
called through its C ABI, one fused kernel per decode call and a tcgen05
grouped-GEMM pipeline per prefill call, for every layer encoding.

Staging (``_device_layer``, reference ``:374-455`` / ``:769-956``): the first
call on a (pack handle, layer, device) copies every expert's canonical bytes,
projection by projection, through a pinned host buffer into one device tensor
per projection; nothing is dequantised, ``dequantized_weight_bytes`` stays 0.
"""

from __future__ import annotations

import contextlib
import threading
import warnings
from pathlib import Path
from typing import Any, Optional

from . import _native, build as _build
from .custom_op import PLATFORM, acquire_expert_pack, register_moe_forward, register_performance_backend
from .formats import ContractError, row_bytes
from .packs import expert_tensor_name

_MODELS = {
    # op name -> (layers, experts, top_k, hidden, intermediate)    src/uma_qmoe/fixed_models.py:32-55
    "olmoe": (16, 64, 8, 2048, 1024),
    "qwen": (24, 60, 4, 2048, 1408),
}
_LABELS = {"olmoe": "OLMoE", "qwen": "Qwen"}


def native_kernel_source_sha256() -> str:
    return _build.source_sha256()


def observed_native_platform(torch: Any, device: Any = 0) -> str:
    if not torch.cuda.is_available():
        raise ContractError("the native backend requires a CUDA device")
    capability = torch.cuda.get_device_capability(device)
    if torch.version.hip or capability != (10, 0):
        raise ContractError(f"the native backend requires SM100 (B200), got sm_{capability[0]}{capability[1]}")
    return PLATFORM


def load_native_extension(*, build_directory: str | Path | None = None, verbose: bool = False) -> tuple[str, Any]:
    """Build (if stale) and load ``libumaq_b200.so``; returns (platform, library).

    ``build_directory`` is accepted for signature compatibility; the library is
    always built in-tree next to its sources."""
    import torch

    platform = observed_native_platform(torch)
    _build.build(verbose=verbose)
    return platform, _native.lib()


class _LayerCache:
    def __init__(self) -> None:
        self.layers: dict[tuple[int, int, str], Any] = {}
        self.lock = threading.Lock()


class _Workspace:
    """A kernel workspace owned by one (shape, device, stream), room for the routes of a call that routes itself, and the host's
    view of the workspace's sticky status word.

    The last kernel of a call copies the word to mapped host memory if it is set, and an event is recorded behind the call.
    The next call on this workspace looks at the host's copy; `cache_summary()` and `release_pack()` wait for the event and
    then look at the word itself as well, which every CTA of the call has written by then.  Nothing on the hot path waits for
    the device."""

    __slots__ = ("kind", "buffer", "host", "word", "event", "used", "tokens", "indices", "weights", "lock", "captured",
                 "outgrown")

    def __init__(self, kind: str, buffer: Any, tokens: int, top_k: int, stream: Any) -> None:
        import torch

        self.kind, self.buffer, self.tokens = kind, buffer, tokens
        self.host = torch.zeros(4, dtype=torch.int32).pin_memory()
        self.word = self.host.numpy()
        self.event = torch.cuda.Event()
        if not torch.cuda.is_current_stream_capturing():
            self.event.record(stream)                # creates it
        self.used = False
        self.captured: set[int] = set()              # packs with a captured call, whose graph holds this slot's addresses
        self.outgrown = False                        # a larger slot has taken its place: no further call
        self.lock = threading.Lock()                 # the launches of a call stay together on the stream
        self.indices = torch.empty((tokens, top_k), dtype=torch.int64, device=buffer.device)
        self.weights = torch.empty((tokens, top_k), dtype=torch.float32, device=buffer.device)

    def report(self, device: Any, pack_handle: int) -> tuple[Optional[int], Optional[int]]:
        """Where a call leaves its status and which event it records; a captured call reports through the workspace only."""
        import torch

        if torch.cuda.is_current_stream_capturing():
            self.captured.add(pack_handle)
            return None, None
        if not self.event.cuda_event:                # made during a capture
            self.event.record(torch.cuda.current_stream(device))
        self.used = True
        return self.host.data_ptr(), self.event.cuda_event

    def raise_if_failed(self, wait: bool) -> None:
        if not self.used or not (wait or self.word[0]):
            return
        import torch

        if torch.cuda.is_current_stream_capturing():
            return
        self.event.synchronize()                     # all work on the buffer has finished
        code = int(self.word[0])
        if wait and code == 0:
            code = int(self.buffer[:16].view(torch.int32)[0 if self.kind == "prefill" else 2])
        if code == 0:
            return
        # sticky on the device: clear it so that the error is reported once
        self.word[0] = 0
        self.used = False
        if code == -1:                               # UMAQ_ERR_BAD_ARGUMENT: the kernels skipped a route
            self.buffer[:16].zero_()
            raise RuntimeError("expert_indices contains an invalid expert")
        self.buffer[:1024].zero_()                   # a timeout leaves stale counters behind
        raise RuntimeError(f"an earlier uma_qmoe::moe_forward call failed on the device ({_native.ERRORS.get(code, code)})")


class MixedTargetNativeBackend:
    """Executes Q4, Q8 and BF16 layers of an ExpertPack or TargetPack."""

    allowed_encodings = ("q4_group128", "q8_group128", "bf16_le")

    def __init__(self, platform: str, extension: Any) -> None:
        if platform != PLATFORM:
            raise ContractError(f"unsupported native platform {platform!r}")
        for name in _native.SIGNATURES:
            if not hasattr(extension, name):
                raise ContractError(f"native library does not export {name}")
        self.platform = platform
        self.extension = extension
        self._cache = _LayerCache()
        self._workspaces: dict[tuple, _Workspace] = {}
        self._outgrown: list[_Workspace] = []                    # replaced by larger ones, but captured graphs use them
        self._pending: dict[tuple[int, int, str], Any] = {}      # layers being staged: (DeviceLayer, wait)
        self._linear_cache: dict[tuple[int, str, str], Any] = {}  # single tensors staged for q4_linear / q8_linear
        self._workspace_lock = threading.Lock()

    # ---- construction ---------------------------------------------------------------------
    @classmethod
    def build_and_register(cls, *, build_directory: str | Path | None = None, verbose: bool = False):
        platform, extension = load_native_extension(build_directory=build_directory, verbose=verbose)
        backend = cls(platform, extension)
        register_moe_forward()
        register_performance_backend(platform, backend)
        return backend

    # ---- staging --------------------------------------------------------------------------
    @staticmethod
    def _encoding_of(reader: Any, layer_index: int) -> str:
        if hasattr(reader, "layer_encoding"):
            return reader.layer_encoding(layer_index)
        group = int(reader.header["quantization"]["group_size"])
        if group != 128:
            raise RuntimeError(f"the native backend requires group size 128, got {group}")
        return "q4_group128"

    def _device_layer(self, pack_handle: int, layer_index: int, device: Any, reader: Any, model: str):
        import torch

        from .ops import DeviceLayer

        key = (pack_handle, layer_index, str(device))
        with self._cache.lock:
            hit = self._cache.layers.get(key)
        if hit is not None:
            return hit
        layers, experts, _k, hidden, inter = _MODELS[model]
        if not 0 <= layer_index < layers:
            name = "OLMoE" if model == "olmoe" else "Qwen"
            raise RuntimeError(f"{name} layer_index must be in [0, {layers - 1}]")
        encoding = self._encoding_of(reader, layer_index)
        if encoding not in self.allowed_encodings:
            raise RuntimeError(f"this backend cannot execute layer {layer_index} encoded as {encoding}; "
                               "install the mixed backend")
        quantised = encoding != "bf16_le"
        if hasattr(reader, "stage_layer_async"):
            # the native reader stages by itself: a worker thread, pinned chunks, copies on a stream of its own;
            # a prefetch may already be under way
            with self._cache.lock:
                pending = self._pending.pop(key, None)
            layer, wait = pending if pending is not None else self._start_staging(reader, layer_index, device, model)
            wait(torch.cuda.current_stream(device))
            with self._cache.lock:
                return self._cache.layers.setdefault(key, layer)
        staged = {}
        for proj, (rows, k) in (("gate_proj", (inter, hidden)), ("up_proj", (inter, hidden)),
                                ("down_proj", (hidden, inter))):
            nbytes = rows * row_bytes(encoding, k)
            host = torch.empty((experts, nbytes), dtype=torch.uint8).pin_memory()
            host_s = torch.empty((experts, rows * k // 128), dtype=torch.float32).pin_memory() if quantised else None
            for e in range(experts):
                data, scales, meta = reader.tensor_views(expert_tensor_name(layer_index, e, proj))
                try:
                    if tuple(meta["shape"]) != (rows, k):
                        raise RuntimeError(f"tensor {meta.get('name', proj)!r} has unexpected shape {tuple(meta['shape'])!r}")
                    if meta.get("encoding", encoding) != encoding:
                        raise RuntimeError(f"tensor of layer {layer_index} is not {encoding}")
                    if len(data) != nbytes:
                        raise RuntimeError("pack tensor byte count does not match its shape")
                    with warnings.catch_warnings():       # the mapping is read-only and is only read here
                        warnings.filterwarnings("ignore", message="The given buffer is not writable")
                        host[e].copy_(torch.frombuffer(data, dtype=torch.uint8))
                        if quantised:
                            host_s[e].copy_(torch.frombuffer(scales, dtype=torch.float32))
                finally:
                    data.release()
                    scales.release()
            staged[proj] = (host.to(device, non_blocking=True),
                            host_s.to(device, non_blocking=True) if quantised else None)
        torch.cuda.current_stream(device).synchronize()      # the pinned buffers go away after this
        layer = DeviceLayer(encoding, experts, hidden, inter, staged["gate_proj"][0], staged["up_proj"][0],
                            staged["down_proj"][0], staged["gate_proj"][1], staged["up_proj"][1],
                            staged["down_proj"][1])
        with self._cache.lock:
            return self._cache.layers.setdefault(key, layer)

    def _start_staging(self, reader: Any, layer_index: int, device: Any, model: str):
        import torch

        from .ops import DeviceLayer
        layers, experts, _k, hidden, inter = _MODELS[model]
        if not 0 <= layer_index < layers:
            raise RuntimeError(f"{'OLMoE' if model == 'olmoe' else 'Qwen'} layer_index must be in [0, {layers - 1}]")
        encoding = self._encoding_of(reader, layer_index)
        if encoding not in self.allowed_encodings:
            raise RuntimeError(f"this backend cannot execute layer {layer_index} encoded as {encoding}; "
                               "install the mixed backend")
        quantised = encoding != "bf16_le"
        codes = lambda rows, k: torch.empty(experts * rows * row_bytes(encoding, k), dtype=torch.uint8, device=device)
        scales = lambda rows, k: torch.empty(experts * rows * k // 128, dtype=torch.float32, device=device) if quantised else None
        layer = DeviceLayer(encoding, experts, hidden, inter, codes(inter, hidden), codes(inter, hidden), codes(hidden, inter),
                            scales(inter, hidden), scales(inter, hidden), scales(hidden, inter))
        # the copies run on the reader's own stream: whatever used this memory before must have finished
        torch.cuda.current_stream(device).synchronize()
        return layer, reader.stage_layer_async(layer_index, layer, device)

    def prefetch_layer(self, pack_handle: int, layer_index: int, device: Any, model: str = "olmoe") -> None:
        """Start staging a layer of a pack opened with the native reader and return at once; the first call that
        needs the layer waits for what is left.  (Nothing to do for the Python readers, which stage on demand.)"""
        import torch
        device = torch.device(device)
        key = (pack_handle, layer_index, str(device))
        with acquire_expert_pack(pack_handle) as reader:
            if not hasattr(reader, "stage_layer_async"):
                return
            with self._cache.lock:
                if key in self._cache.layers or key in self._pending:
                    return
            started = self._start_staging(reader, layer_index, device, model)
            with self._cache.lock:
                self._pending[key] = started

    def preload_layer(self, pack_handle: int, layer_index: int, device: Any, layer: Any) -> None:
        """Adopt a layer that already sits on the device in the staged layout (synthetic weights
        built with the device-side packer), instead of staging it from the pack's host bytes."""
        with self._cache.lock:
            self._cache.layers[(pack_handle, layer_index, str(device))] = layer

    def check_device_status(self) -> None:
        """Wait for the calls submitted so far and raise if one of them recorded a device-side error."""
        with self._workspace_lock:
            slots = [*self._workspaces.values(), *self._outgrown]
        for slot in slots:
            slot.raise_if_failed(wait=True)

    def cache_summary(self) -> dict[str, int]:
        self.check_device_status()
        with self._cache.lock:
            layers = list(self._cache.layers.values())
        return {
            "tensor_count": sum(3 * layer.num_experts for layer in layers),
            "device_storage_bytes": sum(layer.device_storage_bytes for layer in layers),
            "dequantized_weight_bytes": 0,
        }

    def release_pack(self, pack_handle: int) -> None:
        """Drop every device copy that belongs to a closed pack handle."""
        try:
            self.check_device_status()
        finally:
            self._drop_layers(pack_handle)

    def _drop_layers(self, pack_handle: int) -> None:
        import torch
        with self._cache.lock:
            unfinished = [self._pending.pop(k) for k in [k for k in self._pending if k[0] == pack_handle]]
        for layer, wait in unfinished:              # the worker threads must be done before the mapping goes away
            wait(torch.cuda.current_stream(layer.gate.device))
        with self._cache.lock:
            for key in [k for k in self._cache.layers if k[0] == pack_handle]:
                del self._cache.layers[key]
            for key in [k for k in self._linear_cache if k[0] == pack_handle]:
                del self._linear_cache[key]
        with self._workspace_lock:
            for slot in [*self._workspaces.values(), *self._outgrown]:
                slot.captured.discard(pack_handle)
            self._outgrown = [slot for slot in self._outgrown if slot.captured]

    # ---- execution ------------------------------------------------------------------------
    def _workspace(self, kind: str, layer: Any, tokens: int, top_k: int, shared: Any, device: Any, stream: int) -> _Workspace:
        """The workspace of this shape on this stream.  Calls on different streams (or threads, which have their own
        current stream only if they set one) never share a workspace, so they may overlap on the device; a stream
        keeps one prefill workspace per layer shape, grown to the largest token count seen.  One that a graph has captured
        stays until the packs of the captured calls are released: without their weights no such graph can run."""
        from . import ops

        family = (kind, device.index, stream, layer.hidden, layer.intermediate, layer.num_experts, top_k,
                  0 if shared is None else shared.gate.shape[0])
        while True:
            with self._workspace_lock:
                slot = self._workspaces.get(family)
                if slot is not None and (kind == "decode" or slot.tokens >= tokens):
                    return slot
            import torch
            with contextlib.nullcontext() if slot is None else slot.lock:    # no call is being issued on it meanwhile
                if slot is not None:
                    slot.raise_if_failed(wait=True)  # the smaller buffer is about to be dropped
                if kind == "decode":
                    buffer, room = ops.decode_workspace(layer, top_k, shared, device), 1
                else:
                    buffer, room = ops.prefill_workspace(layer, tokens, top_k, shared, device), tokens
                fresh = _Workspace(kind, buffer, room, top_k, torch.cuda.current_stream(device))
                with self._workspace_lock:
                    if self._workspaces.get(family) is not slot:             # another thread was quicker
                        continue
                    self._workspaces[family] = fresh
                    if slot is not None:
                        slot.outgrown = True
                        # (under a capture nobody has waited for the calls that may still write to the host's copy)
                        if slot.captured or torch.cuda.is_current_stream_capturing():
                            self._outgrown.append(slot)
                return fresh

    def _run(self, model: str, hidden_states: Any, expert_indices: Any, routing_weights: Any, layer_index: int,
             pack_handle: int, shared: Optional[Any] = None, router: Optional[tuple] = None):
        """`router`: (weight, top_k, renormalise) of a call that routes itself; its routes stay in the workspace."""
        import torch

        from . import ops

        _layers, _experts, top_k, hidden, _inter = _MODELS[model]
        if hidden_states.dtype != torch.bfloat16:
            raise RuntimeError(f"{_LABELS[model]} native backend requires BF16 hidden states")
        flat = hidden_states.reshape(-1, hidden_states.shape[-1])
        tokens = flat.shape[0]
        if flat.shape[1] != hidden:
            raise RuntimeError(f"{_LABELS[model]} native backend requires hidden size {hidden}")
        if router is not None:
            ops._require_cuda_bf16(flat, "hidden_states")
            ops._require_cuda_bf16(router[0], "router weight")
            if router[1] != top_k or router[0].ndim != 2 or router[0].shape[1] != hidden:
                raise RuntimeError(f"{_LABELS[model]} native backend requires [tokens, {top_k}] routes")
        else:
            if tuple(expert_indices.shape) != (tokens, top_k):
                raise RuntimeError(f"{_LABELS[model]} native backend requires [tokens, {top_k}] routes")
            if expert_indices.dtype not in (torch.int32, torch.int64):
                raise RuntimeError("expert_indices must use int32 or int64")
            if tuple(routing_weights.shape) != tuple(expert_indices.shape):
                raise RuntimeError("expert_indices and routing_weights shapes must match")
            if expert_indices.device != flat.device or routing_weights.device != flat.device:
                raise RuntimeError("expert_indices and routing_weights must be on the device of hidden_states")
        device = flat.device
        with acquire_expert_pack(pack_handle) as reader:
            layer = self._device_layer(pack_handle, layer_index, device, reader, model)
        stream = torch._C._cuda_getCurrentRawStream(device.index)
        layer.used_on(stream, device)
        flat = flat.contiguous()
        if flat.data_ptr() & 15:              # the kernels read 16 bytes at a time
            flat = flat.clone()
        out = torch.empty_like(flat)
        if tokens == 0 and router is not None:
            ops.route_topk(flat, *router)     # refuses it: a router has no empty result
        if tokens == 0:                       # an empty batch has an empty result; there is nothing to launch
            return out.reshape(hidden_states.shape)
        if router is None:
            indices = expert_indices.contiguous()
            weights = routing_weights.to(dtype=torch.float32).contiguous()     # float32 routing weights, no BF16 rounding
        while True:
            slot = self._workspace("decode" if tokens == 1 else "prefill", layer, tokens, top_k, shared, device, stream)
            slot.raise_if_failed(wait=False)  # an error an earlier call on this workspace left behind, if already known
            with slot.lock:
                if slot.outgrown:             # by another thread on this stream, between the two lines above
                    continue
                if router is not None:
                    indices, weights = slot.indices, slot.weights
                    if slot.tokens != tokens:
                        indices, weights = indices[:tokens], weights[:tokens]
                host, event = slot.report(device, pack_handle)
                ops.moe_step(layer, flat, indices, weights, out, slot.buffer, shared, None if router is None else router[0],
                             router is not None and router[2], host, event, stream)
                break
        return out.reshape(hidden_states.shape)

    # ---- one projection as a linear layer -----------------------------------------------------
    def _linear(self, input_tensor: Any, pack_handle: int, tensor_name: str, encoding: str):
        """``bf16(input . W^T)`` for one packed tensor of a registered pack (the reference backend's ``q4_linear`` /
        ``q8_linear``, ``src/uma_qmoe/native_backend.py:319-372``; there a GEMV kernel per call, here the grouped GEMM's
        down mode on a one-expert layer: rows of any count, out features a multiple of 256, in features of 128)."""
        import torch

        from . import ops
        from .ops import DeviceLayer
        if input_tensor.dtype != torch.bfloat16 or input_tensor.ndim != 2 or not input_tensor.is_cuda:
            raise RuntimeError("the native backend requires a 2-D BF16 CUDA input")
        device = input_tensor.device
        key = (pack_handle, tensor_name, str(device))
        with self._cache.lock:
            hit = self._linear_cache.get(key)
        if hit is None:
            with acquire_expert_pack(pack_handle) as reader:
                data, scales, meta = reader.tensor_views(tensor_name)
                try:
                    if meta.get("encoding", "q4_group128") != encoding:
                        raise RuntimeError(f"tensor {tensor_name!r} is not {encoding}")
                    rows, k = (int(d) for d in meta["shape"])
                    with warnings.catch_warnings():
                        warnings.filterwarnings("ignore", message="The given buffer is not writable")
                        codes = torch.frombuffer(data, dtype=torch.uint8).to(device)
                        sc = torch.frombuffer(scales, dtype=torch.float32).to(device)
                finally:
                    data.release()
                    scales.release()
            if rows % 256 or k % 128:
                raise RuntimeError(f"tensor {tensor_name!r} has a shape the linear path does not take: {(rows, k)}")
            # a one-expert layer whose "down" projection is this tensor: hidden = out features, intermediate = in
            hit = DeviceLayer(encoding, 1, rows, k, codes, codes, codes, sc, sc, sc)
            with self._cache.lock:
                hit = self._linear_cache.setdefault(key, hit)
        if input_tensor.shape[1] != hit.intermediate:
            raise RuntimeError(f"input has {input_tensor.shape[1]} features, the tensor takes {hit.intermediate}")
        n = input_tensor.shape[0]
        if n == 0:
            return input_tensor.new_empty((0, hit.hidden))
        ones = torch.ones((n, 1), dtype=torch.float32, device=device)
        routes = ops.route_sort(torch.zeros((n, 1), dtype=torch.int32, device=device), ones, 1)
        act = ops.gather_rows(input_tensor.contiguous(), None, 1, permute=True)      # the k order of the quantised GEMM
        return ops.grouped_gemm(hit, 1, act, routes)

    def q4_linear(self, input_tensor: Any, pack_handle: int, tensor_name: str):
        return self._linear(input_tensor, pack_handle, tensor_name, "q4_group128")

    def q8_linear(self, input_tensor: Any, pack_handle: int, tensor_name: str):
        return self._linear(input_tensor, pack_handle, tensor_name, "q8_group128")

    def __call__(self, hidden_states, expert_indices, routing_weights, layer_index: int, pack_handle: int):
        return self._run("olmoe", hidden_states, expert_indices, routing_weights, layer_index, pack_handle)

    def qwen_forward(self, hidden_states, expert_indices, routing_weights, layer_index: int, pack_handle: int):
        return self._run("qwen", hidden_states, expert_indices, routing_weights, layer_index, pack_handle)

    def qwen_block_forward(self, hidden_states, expert_indices, routing_weights, layer_index: int, pack_handle: int,
                           shared: Any):
        """Routed experts plus the shared expert and its sigmoid gate in the same kernels."""
        return self._run("qwen", hidden_states, expert_indices, routing_weights, layer_index, pack_handle, shared)

    def block_forward(self, model: str, hidden_states, router_weight, top_k: int, renormalize: bool, layer_index: int,
                      pack_handle: int, shared: Any = None):
        """A whole MoE block: router, routed experts and (Qwen) the shared expert with its gate, in one native call."""
        return self._run(model, hidden_states, None, None, layer_index, pack_handle, shared, (router_weight, top_k, renormalize))


class PackedQ4NativeBackend(MixedTargetNativeBackend):
    """The Q4-only backend of the reference's first milestone; other encodings are refused with the
    reference's hint to install the mixed backend (``native_backend.py:421-427``)."""

    allowed_encodings = ("q4_group128",)


def install_packed_q4_backend(*, build_directory: str | Path | None = None, verbose: bool = False):
    return PackedQ4NativeBackend.build_and_register(build_directory=build_directory, verbose=verbose)


def install_mixed_target_backend(*, build_directory: str | Path | None = None, verbose: bool = False):
    return MixedTargetNativeBackend.build_and_register(build_directory=build_directory, verbose=verbose)


__all__ = [
    "PackedQ4NativeBackend",
    "MixedTargetNativeBackend",
    "install_mixed_target_backend",
    "install_packed_q4_backend",
    "load_native_extension",
    "native_kernel_source_sha256",
    "observed_native_platform",
]
