"""What the modules keep beside their buffers (re-ordered indices, scaled codebook): when it is read, waited for, rebuilt."""

from __future__ import annotations

import copy
import pickle
import types

import pytest
import torch

from dimq_b200 import _lib, modules, ops
from dimq_b200.modules import DIMQConv2d, DIMQLinear


class _Gpu:
    """A stand-in for the CUDA calls around a kept tensor: which stream is current, what it was told to wait for."""

    def __init__(self, monkeypatch):
        self.current, self.capturing, self.done, self.log, self.built = 1, False, False, [], 0
        gpu = self

        def record(device):
            gpu.log.append(("record", gpu.current))
            return "event"

        def prepack(pw, *args):
            gpu.built += 1
            return pw.clone()

        monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: types.SimpleNamespace(cuda_stream=gpu.current))
        monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda d: gpu.current, raising=False)
        monkeypatch.setattr(_lib, "host", lambda: types.SimpleNamespace(
            record_event=record, event_done=lambda e: gpu.done, capturing=lambda d: gpu.capturing,
            wait_event=lambda e, d: gpu.log.append(("wait", gpu.current))))
        monkeypatch.setattr(torch.Tensor, "record_stream", lambda t, s: gpu.log.append(("uses", s.cuda_stream)))
        monkeypatch.setattr(ops, "conv_prepack", prepack)


@pytest.fixture()
def gpu(monkeypatch):
    return _Gpu(monkeypatch)


def _conv():
    return DIMQConv2d(torch.arange(8 * 64 // 2, dtype=torch.uint8), torch.zeros(16), None, None, (8, 64, 1, 1))


def test_a_second_stream_waits_for_the_copy(gpu):
    layer = _conv()
    first = layer._prepacked()
    assert layer._prepacked() is first and gpu.log == [("record", 1)]      # the building stream needs no wait
    gpu.current = 2
    assert layer._prepacked() is first
    assert gpu.log[1:] == [("wait", 2), ("uses", 2)]                       # before this: read without waiting
    assert layer._prepacked() is first and gpu.log[3:] == [("wait", 2)]    # every call, until it is known to be written
    gpu.done = True
    del gpu.log[:]
    assert layer._prepacked() is first and gpu.log == []
    gpu.current = 3
    assert layer._prepacked() is first and gpu.log == [("uses", 3)]
    assert gpu.built == 1


def test_a_capture_keeps_nothing_and_reads_nothing_unwritten(gpu):
    layer = _conv()
    gpu.capturing = True
    assert layer._prepacked() is not None and layer._khwc is None          # a replay writes that one
    gpu.capturing = False
    first = layer._prepacked()
    gpu.capturing, gpu.current = True, 2
    assert layer._prepacked() is not first and gpu.built == 3              # not written yet: a replay would not wait
    gpu.done = True
    assert layer._prepacked() is first


def test_rebuilt_with_every_new_buffer(gpu):
    layer = _conv()
    gpu.done = True
    for i in range(50):                        # a freed buffer's address comes back at once
        layer.packed_weight = torch.full((256,), i, dtype=torch.uint8)
        assert int(layer._prepacked()[0]) == i
    layer.packed_weight.add_(1)
    assert int(layer._prepacked()[0]) == 50
    built = gpu.built
    layer.float()                              # nothing moved
    assert int(layer._prepacked()[0]) == 50 and gpu.built == built
    layer._apply(lambda t: t.clone())
    assert layer._khwc is None


def test_inference_tensors_are_taken(gpu):
    with torch.inference_mode():
        layer = _conv()
    assert torch.equal(layer._prepacked(), layer.packed_weight) and layer._khwc is None


def test_modules_are_copied_and_saved_without_it(gpu):
    layer = _conv()
    layer._prepacked()
    for twin in (copy.deepcopy(layer), pickle.loads(pickle.dumps(layer))):
        assert twin._khwc is None and torch.equal(twin.packed_weight, layer.packed_weight)


def test_buffers_may_have_become_parameters(monkeypatch):
    seen = []
    monkeypatch.setattr(ops, "dimq_linear_wq", lambda x, pw, cb, bias, *a, **k: seen.append((pw, cb, bias)))
    monkeypatch.setattr(ops, "dimq_conv2d_wq", lambda x, pw, cb, bias, *a, **k: seen.append((pw, cb, bias)))
    monkeypatch.setattr(modules._PackedBase, "_refuse", lambda self: None)
    monkeypatch.setattr(DIMQConv2d, "_prepacked", lambda self: None)
    for layer in (DIMQLinear(torch.zeros(32, dtype=torch.uint8), torch.zeros(16), None, None, 8, 8, torch.zeros(8)),
                  DIMQConv2d(torch.zeros(32, dtype=torch.uint8), torch.zeros(16), None, None, (8, 8, 1, 1), torch.zeros(8))):
        layer.codebook = torch.nn.Parameter(torch.ones(16))              # trained on top of the export
        layer.bias = torch.nn.Parameter(torch.ones(8))
        layer.packed_weight = torch.nn.Parameter(layer.packed_weight, requires_grad=False)
        layer(torch.zeros(1, 8, 1, 8))
        assert seen[-1][0] is layer.packed_weight and seen[-1][1] is layer.codebook and seen[-1][2] is layer.bias


def test_the_registered_operator_is_bypassed_in_plain_eager_calls_only():
    from torch.overrides import TorchFunctionMode
    from torch.utils._python_dispatch import TorchDispatchMode

    class Function(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    class Dispatch(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    x, p = torch.zeros(2), torch.nn.Parameter(torch.zeros(2))
    assert modules._eager(x, x, None) and modules._eager(x, x, x)
    assert not modules._eager(x, p, None) and not modules._eager(x, x, p) and not modules._eager(x.clone().requires_grad_(), x, None)
    with torch.no_grad():
        assert modules._eager(x, p, p)
    for mode in (Function(), Dispatch()):
        with mode:
            seen = modules._eager(x, x, None)
        assert not seen


# ---- on the GPU ----------------------------------------------------------------------------------

def _a4_conv(seed=0):
    gen = torch.Generator().manual_seed(seed)
    packed = torch.randint(0, 256, (64 * 64 * 9 // 2,), dtype=torch.uint8, generator=gen)
    return DIMQConv2d(packed, torch.randn(16, generator=gen), 0.25, 7, (64, 64, 3, 3), padding=1).cuda()


def _linear(seed=0):
    gen = torch.Generator().manual_seed(seed)
    packed = torch.randint(0, 256, (1024 * 4096 // 2,), dtype=torch.uint8, generator=gen)
    return DIMQLinear(packed, torch.randn(16, generator=gen).half(), None, None, 1024, 4096, out_dtype=torch.float16).cuda()


def _inputs(layer):
    return torch.randn(2, 64, 9, 9, device="cuda") if isinstance(layer, DIMQConv2d) else torch.randn(4, 4096, device="cuda").half()


@pytest.mark.gpu
@pytest.mark.parametrize("make", [_a4_conv, _linear])
def test_first_call_on_a_busy_stream_then_another_stream(cuda_device, make):
    layer, twin = make(), make()
    x = _inputs(layer)
    want = twin(x)
    torch.cuda.synchronize()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(a):
        torch.cuda._sleep(50_000_000)          # the copy is written some 25 ms after the call has returned
        layer(x)
    with torch.cuda.stream(b):
        y = layer(x)
    torch.cuda.synchronize()
    assert torch.equal(y, want)


@pytest.mark.gpu
@pytest.mark.parametrize("make", [_a4_conv, _linear])
@pytest.mark.parametrize("warm", [False, True])
def test_captured_calls(cuda_device, make, warm):
    layer, twin = make(), make()
    x = _inputs(layer)
    want = twin(x)
    if warm:
        layer(x)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = layer(x)
    assert torch.equal(layer(x), want)         # an eager call before the first replay
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want)
    if make is _a4_conv:                       # replays follow the buffer itself
        layer.packed_weight.copy_(make(1).packed_weight)
        twin.packed_weight.copy_(layer.packed_weight)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, twin(x))
