"""What a user of this package runs, as cases that can be timed.

A case is one pass of a program through the package's public entry points: a decode step or a prompt through the MoE
blocks of a fixed-shape model (``blocks.QuantizedMoEBlock`` / ``QuantizedQwenMoEBlock``: router, routed experts and, for
Qwen, the shared expert), or the encoding of a layer's dense experts into the packed layout
(``host.encode_experts``).  The shapes are the two fixed models of ``synthetic.py``; weights are random with their
distribution, activations are N(0, 1), the scale of what an RMS norm hands to the block.

Between two MoE blocks a real model has attention and a norm; here every layer gets an input of its own, so that a
case's outputs are comparable layer by layer.  ``graph`` cases replay the step from a CUDA graph captured once, as
``host.GraphedDecoder`` does; the others call the blocks eagerly, as a prefill of a Hugging Face model does.
"""

from __future__ import annotations

import functools
import math
import random
import weakref
from types import SimpleNamespace
from typing import Any

import numpy as np
import torch

from uma_qmoe_b200 import custom_op, host, native_backend
from uma_qmoe_b200.blocks import QuantizedMoEBlock, QuantizedQwenMoEBlock
from uma_qmoe_b200.packs import InMemoryPack
from uma_qmoe_b200.stack import random_layer, random_shared_expert
from uma_qmoe_b200.synthetic import OLMOE, QWEN, router_weight

_SHAPES = {"olmoe": OLMOE, "qwen": QWEN}
_BYTES_PER_WEIGHT = {"q4_group128": 0.5 + 4 / 128, "q8_group128": 1 + 4 / 128, "bf16_le": 2.0}

# Layer policies.  "mixed" is the published Qwen TargetPack policy (two BF16 layers for every Q8 layer).
_POLICIES = {
    "q4": lambda layer, layers: "q4_group128",
    "q8": lambda layer, layers: "q8_group128",
    "bf16": lambda layer, layers: "bf16_le",
    "mixed": lambda layer, layers: "bf16_le" if 3 * layer < 2 * layers else "q8_group128",
}


def _blocks(name: str, model: str, policy: str, tokens: int, layers: int, graph: bool, skew: float) -> dict:
    return {"name": name, "kind": "blocks", "model": model, "policy": policy, "tokens": tokens, "layers": layers,
            "graph": graph, "skew": skew}


def listed() -> list[dict]:
    return [
        # one user generating: a token through all 16 layers of the Q4 model, the step replayed from a graph
        _blocks("olmoe_q4_token_graph", "olmoe", "q4", 1, 16, True, 1.0),
        # the same step issued eagerly, as a host without graph capture runs it: the smallest calls there are
        _blocks("olmoe_q4_token_eager", "olmoe", "q4", 1, 16, False, 1.0),
        # one user generating with the mixed BF16 / Q8 Qwen model and its shared expert
        _blocks("qwen_mixed_token_graph", "qwen", "mixed", 1, 6, True, 1.0),
        # a few users at once: one token of each of 7 sequences
        _blocks("olmoe_q4_batch7_graph", "olmoe", "q4", 7, 8, True, 0.0),
        # a serving batch of the mixed model
        _blocks("qwen_mixed_batch24_graph", "qwen", "mixed", 24, 6, True, 0.0),
        # a large serving batch in the higher-precision encoding
        _blocks("olmoe_q8_batch96_graph", "olmoe", "q8", 96, 4, True, 0.0),
        # the 128-token prompt of the model host's measurement loop, eager, mixed model
        _blocks("qwen_mixed_prompt128", "qwen", "mixed", 128, 6, False, 1.0),
        # the 512-token prompt with a skewed router (some experts without a token)
        _blocks("olmoe_q4_prompt512", "olmoe", "q4", 512, 4, False, 1.0),
        # a prompt of odd length in the quantised Qwen encoding
        _blocks("qwen_q8_prompt1531", "qwen", "q8", 1531, 4, False, 1.0),
        # a batch of prompts through BF16 layers
        _blocks("qwen_bf16_prompt4096", "qwen", "bf16", 4096, 2, False, 1.0),
        # the package's headline: 8192 tokens through Q4 layers
        _blocks("olmoe_q4_prompt8192", "olmoe", "q4", 8192, 4, False, 1.0),
        # loading: a layer's dense BF16 experts encoded on the device
        {"name": "olmoe_q4_encode", "kind": "encode", "model": "olmoe", "policy": "q4"},
    ]


def draw(rng: random.Random) -> dict:
    pick = rng.random()
    model = rng.choice(["olmoe", "qwen"])
    if pick < 0.08:
        return {"kind": "encode", "model": model, "policy": rng.choice(["q4", "q8"])}
    policy = rng.choice(["q4", "q4", "q8", "bf16"] if model == "olmoe" else ["mixed", "q8", "q4", "bf16"])
    skew = rng.choice([0.0, 1.0])
    if pick < 0.2:                                                        # one token, either way of issuing it
        case = _blocks("", model, policy, 1, rng.choice([6, 9, 12]), rng.random() < 0.5, skew)
    elif pick < 0.55:                                                     # a decode step of a batch
        tokens = int(round(2 * math.exp(rng.random() * math.log(64))))    # 2 .. 128
        case = _blocks("", model, policy, tokens, rng.choice([3, 6]), True, skew)
    else:                                                                 # a prompt, or several
        tokens = int(round(16 * math.exp(rng.random() * math.log(512))))  # 16 .. 8192
        case = _blocks("", model, policy, tokens, 2, False, skew)
    del case["name"]
    return case


@functools.lru_cache(maxsize=None)
def _active_experts(model: str, tokens: int, skew: float) -> float:
    """Expected number of experts that get a token, by simulating the router (logits N(0, row norm)).  Beyond 2048
    tokens it no longer changes by anything that matters."""
    shape = _SHAPES[model]
    rng = np.random.default_rng(7)
    found = []
    for _ in range(8):
        norm = np.exp(skew * rng.standard_normal(shape.experts)) * 0.02 * math.sqrt(shape.hidden)
        logits = rng.standard_normal((min(tokens, 2048), shape.experts)) * norm
        found.append(len(np.unique(np.argpartition(-logits, shape.top_k, axis=1)[:, :shape.top_k])))
    return float(np.mean(found))


def _encodings(case: dict) -> list[str]:
    return [_POLICIES[case["policy"]](l, case["layers"]) for l in range(case["layers"])]


def work(case: dict) -> dict:
    shape = _SHAPES[case["model"]]
    h, i, s, e = shape.hidden, shape.intermediate, shape.shared_intermediate, shape.experts
    if case["kind"] == "encode":
        weights = 3 * e * h * i
        return {"bytes": weights * (2 + _BYTES_PER_WEIGHT[_POLICIES[case["policy"]](0, 1)]), "flops": 0}
    t = case["tokens"]
    per_token = 2 * e * h + 6 * h * i * shape.top_k + 6 * h * s           # router, routed experts, shared expert
    nbytes = sum(_active_experts(case["model"], t, case["skew"]) * 3 * h * i * _BYTES_PER_WEIGHT[enc]
                 + 2 * (3 * h * s + e * h) + 4 * t * h for enc in _encodings(case))
    return {"bytes": nbytes, "flops": case["layers"] * t * per_token}


def tolerance(case: dict) -> Any:
    if case["kind"] == "encode":
        return "exact"                                                    # codes and scales are defined bit for bit
    # BF16 results.  Measured against float64 with the same routes: rel 0.0035 (one token) to 0.006, largest
    # difference 0.012 to 0.029 of the root mean square
    return {"rel": 0.02, "max": 0.12}


class _State:
    """What a program keeps: the blocks with their packed layers, the layer inputs and, if it has one, its graph."""

    def __init__(self) -> None:
        self.blocks: list[Any] = []
        self.inputs: list[torch.Tensor] = []
        self.graph: Any = None
        self.outputs: Any = None
        self.dense: Any = None


@functools.lru_cache(maxsize=None)
def _backend() -> Any:
    """Installed once per process: the back end owns the staged layers and the workspaces of every pack registered."""
    return native_backend.install_mixed_target_backend()


def _step(state: _State) -> list[torch.Tensor]:
    return [block(x) for block, x in zip(state.blocks, state.inputs)]


@torch.no_grad()
def prepare(case: dict, seed: int) -> _State:
    device = torch.device("cuda", torch.cuda.current_device())
    shape = _SHAPES[case["model"]]
    gen = torch.Generator(device=device)
    gen.manual_seed(seed * 9176 + 11)
    state = _State()
    if case["kind"] == "encode":
        mk = lambda *dims: torch.randn(*dims, device=device, dtype=torch.bfloat16, generator=gen).mul_(0.02)
        e, h, i = shape.experts, shape.hidden, shape.intermediate
        state.dense = (mk(e, 2 * i, h), mk(e, h, i), _POLICIES[case["policy"]](0, 1))
        return state
    backend = _backend()
    encodings = _encodings(case)
    handle = custom_op.register_target_pack(InMemoryPack(dict(enumerate(encodings))))
    weakref.finalize(state, custom_op.unregister_expert_pack, handle)
    for l, encoding in enumerate(encodings):
        backend.preload_layer(handle, l, device, random_layer(shape, encoding, seed * 64 + l, device))
        gate = SimpleNamespace(weight=router_weight(seed, l, shape, skew=case["skew"]).to(device), top_k=shape.top_k,
                               norm_topk_prob=False)
        if shape.qwen:
            w = random_shared_expert(shape, seed * 64 + l, device)
            linear = lambda t: SimpleNamespace(weight=t)
            shared = SimpleNamespace(gate_proj=linear(w.gate), up_proj=linear(w.up), down_proj=linear(w.down))
            block = QuantizedQwenMoEBlock(gate, shared, linear(w.gate_vec), layer_index=l, pack_handle=handle,
                                          performance_mode=True)
        else:
            block = QuantizedMoEBlock(gate, layer_index=l, pack_handle=handle, performance_mode=True)
        state.blocks.append(block)
        # a decode step is [sequences, 1, hidden], a prompt [1, tokens, hidden]
        dims = (case["tokens"], 1) if case["graph"] else (1, case["tokens"])
        state.inputs.append(torch.randn(*dims, shape.hidden, device=device, generator=gen).to(torch.bfloat16))
    if case["graph"]:
        side = torch.cuda.Stream(device=device)
        side.wait_stream(torch.cuda.current_stream(device))
        with torch.cuda.stream(side):
            _step(state)
            state.graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(state.graph, stream=side):
                state.outputs = _step(state)
        torch.cuda.current_stream(device).wait_stream(side)
    return state


@torch.no_grad()
def run(state: _State) -> Any:
    if state.dense is not None:
        layer = host.encode_experts(*state.dense)
        return list(layer.tensors)
    if state.graph is not None:
        state.graph.replay()
        return state.outputs
    return _step(state)
