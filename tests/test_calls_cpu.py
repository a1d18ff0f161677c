"""CPU tests of the native call path (csrc/python_calls.cpp) and of the passes that ConvChain records through it: a recording
holds plan handles and pointers, so whatever they were taken from may not be replaced, moved or closed unnoticed.  No GPU is
touched: launches either go to a stand-in or fail on the null plan before anything is launched."""
import gc

import pytest


class FakePlan:
    def __init__(self, handle):
        self._plan = handle


class FakeCalls:
    """Stands in for the extension module: a recording is the list of calls, running it hands that list back."""

    def __init__(self):
        self.ran = []

    def record(self, steps):
        return list(steps)

    def run_sequence(self, steps, stream):
        self.ran.append(list(steps))


def small_chain(pkg, ops=None):
    """A ConvChain of two convolutions and an add over host tensors, without its constructor's device work."""
    import torch
    from cuda_inference_b200 import chain as chain_module
    from cuda_inference_b200.workloads import ChainOp, ConvShape
    c = chain_module.ConvChain.__new__(chain_module.ConvChain)
    shape = ConvShape(1, 16, 4, 4, 16, 1, 1, 0, pkg.FP16)
    c.ops = [ChainOp("conv", 0, 1, shape, True, layer=0), ChainOp("conv", 1, 2, shape, False, layer=1), ChainOp("add", 2, 3, relu=True, other=0)]
    c.slots = {i: torch.zeros(256, dtype=torch.float16) for i in range(4)}
    c.convs = [(op, FakePlan(0x1000 + 16 * i), torch.zeros(256, dtype=torch.float16), torch.zeros(16, dtype=torch.float16))
               for i, op in enumerate(c.ops[:2])]
    c.precision, c.batch, c.layout, c.fused = pkg.FP16, 1, "nchw", False
    c._ws = torch.zeros(1024, dtype=torch.uint8)
    c.ws_ptr, c.ws_bytes = c._ws.data_ptr(), 512
    return c


@pytest.fixture
def fake(pkg, monkeypatch):
    from cuda_inference_b200 import chain as chain_module
    f = FakeCalls()
    monkeypatch.setattr(chain_module, "calls", lambda: f)
    return f


def close(c):
    c.convs[0][1]._plan = None


def replace_plan(c):
    op, _, w, b = c.convs[0]
    c.convs[0] = (op, FakePlan(0x2000), w, b)


def replace_weights_in_place(c):
    import torch
    c.convs[0][2].set_(torch.ones(512, dtype=torch.float16).untyped_storage(), 256, (256,))


def replace_bias(c):
    import torch
    op, plan, w, _ = c.convs[1]
    c.convs[1] = (op, plan, w, torch.ones(16, dtype=torch.float16))


def replace_slot(c):
    import torch
    c.slots[2] = torch.ones(256, dtype=torch.float16)


def shrink_slot(c):
    c.slots[3] = c.slots[3][:128]


def replace_workspace(c):
    import torch
    c._ws = torch.zeros(4096, dtype=torch.uint8)
    c.ws_ptr = c._ws.data_ptr()


def grow_workspace(c):
    c.ws_bytes = 1024


def drop_relu(c):
    from dataclasses import replace
    c.ops[2] = replace(c.ops[2], relu=False)


@pytest.mark.parametrize("change", [close, replace_plan, replace_weights_in_place, replace_bias, replace_slot, shrink_slot, replace_workspace,
                                    grow_workspace, drop_relu])
def test_recorded_pass_follows_what_it_was_made_from(pkg, fake, change):
    c = small_chain(pkg)
    c._steps = c._record()
    c.enqueue(7)
    assert fake.ran[-1] == c._steps
    change(c)
    c.enqueue(7)
    want = small_chain_steps(c)
    assert fake.ran[-1] == want and fake.ran[-1] != fake.ran[0]


def small_chain_steps(c):
    """The calls of a pass, from what the chain holds now."""
    (_, p0, w0, b0), (_, p1, w1, b1) = c.convs
    s = {i: t.data_ptr() for i, t in c.slots.items()}
    return [("conv_launch", p0._plan, s[0], w0.data_ptr(), b0.data_ptr(), s[1], c.ws_ptr, c.ws_bytes),
            ("conv_launch", p1._plan, s[1], w1.data_ptr(), b1.data_ptr(), s[2], c.ws_ptr, c.ws_bytes),
            ("add_relu_launch", c.precision, int(c.ops[2].relu), s[2], s[0], s[3], c.slots[3].numel())]


def test_replaced_twice_between_passes(pkg, fake):
    """The second tuple may lie where the first one lay."""
    c = small_chain(pkg)
    c._steps = c._record()
    for handle in (0x3000, 0x4000, 0x5000):
        for h in (handle + 1, handle):
            op, _, w, b = c.convs[0]
            c.convs[0] = None
            gc.collect()
            c.convs[0] = (op, FakePlan(h), w, b)
        c.enqueue(7)
        assert fake.ran[-1] == small_chain_steps(c)


def test_recording_keeps_what_it_points_to(pkg, fake):
    import weakref
    c = small_chain(pkg)
    c._steps = c._record()
    plan, slot = weakref.ref(c.convs[0][1]), weakref.ref(c.slots[2])
    c.convs.clear()
    c.slots.clear()
    gc.collect()
    assert plan() is not None and slot() is not None


def test_closed_plan_in_a_recorded_pass_is_an_error(pkg):
    """Through the extension module itself: the null plan is refused before anything is launched."""
    c = small_chain(pkg)
    for _, plan, _, _ in c.convs:
        plan._plan = None
    c._steps = c._record()
    with pytest.raises(pkg.GieError) as e:
        c.enqueue(0)
    assert e.value.code == pkg.INVALID_ARGUMENT


class Stream:
    """What torch.cuda.Stream is to a foreign-function call."""

    def __init__(self, value):
        import ctypes
        self._as_parameter_ = ctypes.c_void_p(value)


def entry_points(pkg):
    """Every call of the extension module through its wrapper, with one argument left open and one fault that the C side reports
    before it touches a device (a null plan, no rows, a null tensor)."""
    closed = pkg.ConvPlan.__new__(pkg.ConvPlan)
    import ctypes
    closed._h, closed._plan = ctypes.c_void_p(), None
    return {
        "launch": lambda v: closed.launch(v, 256, None, 256, None, 0, 0),
        "launch stream": lambda v: closed.launch(256, 256, None, 256, None, 0, v),
        "launch_fused": lambda v: closed.launch_fused(256, 256, None, v, 256, None, 0, 0),
        "rmsnorm": lambda v: pkg.rmsnorm_forward(0, 64, 1e-6, 2, v, 256, 256, stream=0),
        "rmsnorm stream": lambda v: pkg.rmsnorm_forward(0, 64, 1e-6, 2, 256, 256, 256, stream=v),
        "bias_act": lambda v: pkg.bias_act(pkg.FP16, 0, 4, 4, v, True, 256, 0),
        "maxpool2d": lambda v: pkg.maxpool2d(pkg.FP16, 0, 4, 8, 8, 3, 2, 1, v, 256, 0),
        "maxpool2d_nhwc": lambda v: pkg.maxpool2d_nhwc(pkg.FP16, 0, 8, 8, 8, 3, 2, 1, v, 256, 0),
        "add_relu": lambda v: pkg.add_relu(pkg.FP16, True, v, 256, 256, -1, 0),
    }


NAMES = ["launch", "launch stream", "launch_fused", "rmsnorm", "rmsnorm stream", "bias_act", "maxpool2d", "maxpool2d_nhwc", "add_relu"]


@pytest.mark.parametrize("name", NAMES)
def test_pointer_arguments_are_those_of_ctypes(pkg, name):
    """Accepted: ints, None, objects with _as_parameter_, c_void_p.  Refused: floats, numpy integers, other objects."""
    import ctypes

    import numpy as np
    call = entry_points(pkg)[name]
    for v in (256, True, None, Stream(256), Stream(None), ctypes.c_void_p(256), ctypes.c_void_p()):
        with pytest.raises(pkg.GieError) as e:
            call(v)
        assert e.value.code == pkg.INVALID_ARGUMENT, (name, v)
    for v in (1.0, np.int64(256), object(), [256]):
        with pytest.raises(ctypes.ArgumentError):
            call(v)


def test_counts_are_those_of_ctypes(pkg):
    import ctypes

    import numpy as np
    for rows in (0, np.int32(0), False):
        with pytest.raises(pkg.GieError) as e:
            pkg.rmsnorm_forward(rows, 64, np.float32(1e-6), 2, 256, 256, 256)
        assert e.value.code == pkg.INVALID_ARGUMENT
    for rows in (1.0, None, "1"):
        with pytest.raises(TypeError):
            pkg.rmsnorm_forward(rows, 64, 1e-6, 2, 256, 256, 256)
    with pytest.raises(TypeError):
        pkg.rmsnorm_forward(0, 64, "eps", 2, 256, 256, 256)
    with pytest.raises(ctypes.ArgumentError):
        pkg.add_relu(pkg.FP16, True, 256, 256, 256, 1.5)


def test_recorded_pass_takes_stream_objects(pkg, fake):
    import ctypes
    c = small_chain(pkg)
    c._steps = c._record()
    streams = []
    fake.run_sequence = lambda steps, stream: streams.append(stream)
    for s in (512, Stream(512), ctypes.c_void_p(512), None, Stream(None)):
        c.enqueue(s)
    assert streams == [512, 512, 512, None, None]
    with pytest.raises(ctypes.ArgumentError):
        c.enqueue(1.5)


def test_extension_module_reports_its_own_errors(pkg):
    calls = pkg.calls()
    with pytest.raises(TypeError, match="8 arguments, got 2"):
        calls.conv_launch(None, 1)
    with pytest.raises(TypeError, match="device pointer"):
        calls.conv_launch(None, 1.5, None, None, None, None, 0, None)
    with pytest.raises(TypeError, match="an int"):
        calls.conv_launch(None, None, None, None, None, None, None, None)
    assert calls.conv_launch(None, None, None, None, None, None, 0, None) == pkg.INVALID_ARGUMENT and pkg.last_error()
    with pytest.raises(ValueError, match="unknown call gemm"):
        calls.record([("gemm", 1)])
    with pytest.raises(TypeError, match="arguments"):
        calls.record([("add_relu_launch", 1, 1)])
    for bad in ([()], [(7, 1)], [("add_relu_launch", 1, 1, 1.5, 1, 1, 1)]):
        with pytest.raises((TypeError, ValueError)):
            calls.record(bad)
    for bad in (5, None):
        with pytest.raises(TypeError):
            calls.record(bad)
    with pytest.raises(TypeError, match="2 arguments"):
        calls.run_sequence(calls.record([]))
    with pytest.raises(ValueError):
        calls.run_sequence(object(), 0)
    assert calls.run_sequence(calls.record([]), 0) is None
    # the first failing step ends the pass with its own status: a null tensor, then a precision that does not exist
    null_add = ("add_relu_launch", pkg.FP16, 1, None, None, None, 16)
    null_plan = ("conv_launch", None, 256, 256, None, 256, None, 0)
    assert calls.run_sequence(calls.record([null_add, null_plan]), 0) == pkg.INVALID_ARGUMENT
    first = pkg.last_error()
    assert calls.run_sequence(calls.record([null_plan, null_add]), 0) == pkg.INVALID_ARGUMENT
    assert pkg.last_error() != first
