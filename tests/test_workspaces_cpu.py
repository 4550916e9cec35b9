"""How the back end keeps the workspaces of its calls, with the device calls replaced."""

import contextlib
import gc
import weakref
from types import SimpleNamespace

import pytest
import torch

from uma_qmoe_b200 import _native, native_backend, ops


class _Buffer(torch.Tensor):
    """A workspace that can be watched going away."""


@pytest.fixture
def world(monkeypatch):
    state = SimpleNamespace(capturing=False, calls=[], made=[], on_step=None)
    backend = native_backend.MixedTargetNativeBackend(native_backend.PLATFORM, _native.lib())
    layer = SimpleNamespace(hidden=2048, intermediate=1024, num_experts=64, used_on=lambda *_: None)
    monkeypatch.setattr(backend, "_device_layer", lambda *_: layer)
    monkeypatch.setattr(native_backend, "acquire_expert_pack", lambda handle: contextlib.nullcontext())
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda index: 7, raising=False)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: state.capturing)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: None)
    event = lambda: SimpleNamespace(cuda_event=1, record=lambda stream=None: None, synchronize=lambda: None)
    monkeypatch.setattr(torch.cuda, "Event", event)
    monkeypatch.setattr(torch.Tensor, "pin_memory", lambda self: self)

    def workspace(layer, tokens, *_):
        buffer = torch.zeros(4096, dtype=torch.uint8).as_subclass(_Buffer)
        state.made.append(weakref.ref(buffer))
        return buffer

    def step(layer, hidden, indices, weights, out, buffer, shared, router, renormalize, host, event, stream):
        if state.on_step:
            state.on_step(buffer)
        state.calls.append((buffer.data_ptr(), host, hidden.data_ptr()))

    monkeypatch.setattr(ops, "prefill_workspace", workspace)
    monkeypatch.setattr(ops, "decode_workspace", lambda layer, top_k, *_: workspace(layer, 1))
    monkeypatch.setattr(ops, "moe_step", step)
    state.backend = backend
    state.run = lambda tokens, pack=1: backend._run(
        "olmoe", torch.zeros(tokens, 2048, dtype=torch.bfloat16), torch.zeros(tokens, 8, dtype=torch.int64),
        torch.zeros(tokens, 8), 0, pack)
    return state


@pytest.mark.parametrize("tokens,word", [(1, 2), (4, 0)])
def test_a_waiting_check_sees_an_error_that_the_hosts_copy_missed(world, tokens, word):
    """The last kernel's first CTA may have copied the status word before another CTA of it gave up."""
    world.run(tokens)
    world.made[0]()[:16].view(torch.int32)[word] = -4         # UMAQ_ERR_DEVICE_TIMEOUT
    with pytest.raises(RuntimeError, match="failed on the device"):
        world.backend.check_device_status()
    world.backend.check_device_status()                       # reported once
    world.run(tokens)


def test_a_captured_workspace_outlives_its_replacement(world):
    """Capture at 7 tokens, then an eager prompt of 300 on the same stream: the graph still holds the first buffer's address."""
    world.run(7)
    world.capturing = True
    world.run(7)
    world.capturing = False
    world.run(300)
    gc.collect()
    assert len(world.made) == 2 and world.made[0]() is not None
    world.run(600)                                            # the one for 300 was not captured: it goes
    gc.collect()
    assert world.made[0]() is not None and world.made[1]() is None
    world.backend._drop_layers(2)                             # another pack
    assert world.made[0]() is not None
    world.backend._drop_layers(1)                             # the graph's weights go as well now
    gc.collect()
    assert world.made[0]() is None


@pytest.mark.parametrize("before", [None, 4])
def test_no_call_runs_on_a_workspace_that_another_thread_has_replaced(world, before):
    """Its host copy of the status would be given back while the call may still write to it, and nobody would look there."""
    if before:
        world.run(before)
    find, pending = world.backend._workspace, [True]

    def find_and_be_overtaken(*args):
        slot = find(*args)
        if pending:
            pending.clear()
            world.run(300)                                    # the other thread's call, on the same stream
        return slot

    world.backend._workspace = find_and_be_overtaken
    world.run(4)
    kept = {slot.buffer.data_ptr() for slot in world.backend._workspaces.values()}
    assert world.calls[-1][0] in kept and world.calls[-2][0] in kept


def test_two_threads_first_calls_share_one_workspace(world, monkeypatch):
    make, pending = ops.prefill_workspace, [True]

    def make_and_be_overtaken(*args):
        if pending:
            pending.clear()
            world.run(4)
        return make(*args)

    monkeypatch.setattr(ops, "prefill_workspace", make_and_be_overtaken)
    world.run(4)
    kept = {slot.buffer.data_ptr() for slot in world.backend._workspaces.values()}
    assert {call[0] for call in world.calls} == kept


@pytest.mark.parametrize("tokens", [1, 4])
@pytest.mark.parametrize("which", ["indices", "weights"])
def test_routes_on_another_device_are_refused(world, tokens, which):
    """The kernels would follow a host pointer."""
    indices, weights = torch.zeros(tokens, 8, dtype=torch.int64), torch.zeros(tokens, 8)
    if which == "indices":
        indices = indices.to("meta")
    else:
        weights = weights.to("meta")
    with pytest.raises(RuntimeError, match="must be on the device of hidden_states"):
        world.backend._run("olmoe", torch.zeros(tokens, 2048, dtype=torch.bfloat16), indices, weights, 0, 1)
    assert not world.calls


@pytest.mark.parametrize("tokens", [1, 4])
@pytest.mark.parametrize("offset", [1, 4, 8])
def test_activations_reach_the_kernels_on_a_16_byte_boundary(world, tokens, offset):
    """A contiguous view may start anywhere in its storage."""
    hidden = torch.zeros(tokens * 2048 + offset, dtype=torch.bfloat16)[offset:].view(tokens, 2048)
    world.backend._run("olmoe", hidden, torch.zeros(tokens, 8, dtype=torch.int64), torch.zeros(tokens, 8), 0, 1)
    assert world.calls[-1][2] % 16 == 0
