"""A recorded step list that runs without arguments of its own, after a call whose argument was read in place: it reads
the tensors' own values, not the earlier caller's memory."""
import types

import numpy as np
import pytest

import ngraph_python_b200 as ng
from ngraph_python_b200 import transformers


@pytest.mark.parametrize("taken, in_place, sets", [(True, True, 0), (False, True, 1), (False, False, 0)])
def test_addresses_are_set_unless_the_call_has(taken, in_place, sets):
    io = transformers._CallIO.__new__(transformers._CallIO)
    io.args = [(0, None, types.SimpleNamespace(src=None), False), (1, None, types.SimpleNamespace(src=None), in_place)]
    io.in_front, io.taken, calls = True, taken, []

    def take():
        assert all(arg.src is None for _, _, arg, _ in io.args)
        calls.append(True)
        io.taken = True
    io.take = take
    io.before_replay()
    assert len(calls) == sets and not io.taken
    io.before_replay()                                       # the next one is no call either
    assert len(calls) == sets + in_place


@pytest.mark.gpu
@pytest.mark.parametrize("flex", [False, True])
def test_replays_after_a_call_in_place(flex):
    import torch
    rows, cols = 512, 516
    A, B = ng.make_axis(rows, name="A"), ng.make_axis(cols, name="B")
    x = ng.placeholder([A, B])
    t = ng.transformers.make_transformer_factory("b200", flex=flex)()
    comp = t.computation(ng.max(x * 2.0, reduction_axes=[B]), x)
    g = torch.Generator(device="cuda").manual_seed(1)
    first, second = [torch.rand((rows, cols), device="cuda", generator=g) + 0.25 for _ in range(2)]
    host = np.random.RandomState(2).rand(rows, cols).astype(np.float32) + 0.25

    def right(got, v):
        v = v.cpu().numpy() if isinstance(v, torch.Tensor) else v
        np.testing.assert_allclose(got, 2 * v.max(axis=1), atol=2.0 ** -11 if flex else 0)
    comp(first)
    comp.capture()
    assert [s for s in comp.steps if getattr(s, "stores_argument", ())]
    right(comp(first), first)
    # the argument's range has to be found again: the values are placed step by step, the step list is replayed
    if flex:
        t._view_of(x).buffer.entry.reset_entry()
        right(comp(host), host)
        right(comp(second), second)
        t._view_of(x).buffer.entry.initialized = False
        right(comp(first), first)
    # the step list alone: what the last call stored
    right(comp(second), second)
    was = second.clone()
    second.zero_()
    for _ in range(2):
        t._begin_call(comp)
        comp.executor()
        result = t._device_to_host_async(comp.return_views[0])
        t._end_call(comp)
        right(t._finish_host(result), was)
    right(comp(first), first)
    t.close()
