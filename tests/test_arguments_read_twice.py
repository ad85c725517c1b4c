"""Large arguments that one kernel, or a copy in front of it, reads through several views: a recorded call
must not read the argument's own memory while the kernel stores the argument there."""
import numpy as np
import pytest

import ngraph_python_b200 as ng

# (above the size from which arguments are read in place, in fp32 bytes)
SQUARE, TURNED = (768, 768), (24, 40, 40, 24)


def _column(x, axes):
    """The argument and one column of it."""
    return x - ng.tensor_slice(x, (slice(None), 0))


def _transposed(x, axes):
    """Both views over the whole argument."""
    return x + ng.cast_axes(ng.axes_with_order(x, axes[::-1]), axes)


def _beside(x, axes):
    """The argument once more, in a later kernel; nothing stands in the way of reading it in place."""
    return ng.tanh(x) * 2.0 + ng.sum(x, reduction_axes=[axes[0]])


# (four axes in reverse are laid out dense by a copy that runs in front of the kernel)
CASES = {"column": (_column, SQUARE, []), "transposed": (_transposed, SQUARE, []),
         "copied": (_transposed, TURNED, []), "beside": (_beside, SQUARE, [0])}


def _graph(name):
    build, lengths, taken = CASES[name]
    axes = [ng.make_axis(n, name=c) for n, c in zip(lengths, "ABCD")]
    x = ng.placeholder(axes)
    return x, build(x, axes), taken


@pytest.mark.parametrize("flex", [False, True])
@pytest.mark.parametrize("name", sorted(CASES))
def test_which_arguments_are_read_in_place(name, flex):
    x, y, taken = _graph(name)
    t = ng.transformers.allocate_transformer("b200", plan_only=True, flex=flex)
    comp = t.computation(y, x)
    t.initialize()
    assert any(s.kind == "dimshuffle" for s in comp.steps) == (name == "copied")
    buf, stored = t._view_of(x).buffer, False
    for s in comp.steps:
        mine = [i for i, v in enumerate(s.in_views) if v.buffer is buf]
        at = list(getattr(s, "stores_argument", ()))
        if at:
            assert not stored and mine == at
        stored = stored or bool(mine)
    assert [i for s in comp.steps for i in getattr(s, "stores_argument", ())] == taken


@pytest.mark.gpu
@pytest.mark.parametrize("flex", [False, True])
@pytest.mark.parametrize("name", sorted(CASES))
def test_recorded_calls_are_those_step_by_step(name, flex):
    import torch

    def run(capture):
        x, y, _ = _graph(name)
        t = ng.transformers.allocate_transformer("b200", flex=flex)
        comp = t.computation(y, x)
        out = []
        for i in range(6):
            g = torch.Generator(device="cuda").manual_seed(i)
            out.append(np.array(comp(torch.randn(CASES[name][1], device="cuda", generator=g)), copy=True))
            out.append(np.array(t.get_tensor_view_value(x)))
            if capture and i == 0:
                comp.capture()
        t.close()
        return out
    for i, (a, b) in enumerate(zip(run(False), run(True))):
        assert np.array_equal(a, b), i
