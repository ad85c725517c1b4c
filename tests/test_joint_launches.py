"""Updates of one form share a launch: more tensors than one launch takes, sizes that take the vector and
the scalar kernel, one block and several; a tensor that another one depends on stays in order."""
import numpy as np
import pytest

import ngraph_python_b200 as ng
from ngraph_python_b200 import lib


@pytest.mark.gpu
@pytest.mark.parametrize("flex", [False, True])
def test_joint_updates(flex):
    sizes = [8 * k for k in range(1, 40)] + [1, 3, 10, 17, 4099, 65536, 40000]
    rng = np.random.RandomState(1)
    start = [rng.uniform(-1, 1, n).astype(np.float32) for n in sizes]
    ws = [ng.variable([ng.make_axis(n, name="A%d" % i)], initial_value=v)
          for i, (n, v) in enumerate(zip(sizes, start))]
    steps = [ng.assign(w, w * 0.5 + 0.25) for w in ws]
    total = ng.sum(ws[3], reduction_axes=ws[3].axes)         # reads a tensor before and after ...
    last = ng.assign(ws[3], ws[3] * 0.5 + 0.25)              # ... it is written once more
    t = ng.transformers.allocate_transformer("b200", flex=flex)
    comp = t.computation(ng.sequential(steps + [total, last, total * 1.0]))
    t.initialize()
    comp()
    comp.capture()
    leaders = [s for s in comp.steps if getattr(s, "joint", ())]
    assert sum(len(s.joint) for s in leaders) >= 40
    before = t.kernel_launches
    comp()
    assert t.kernel_launches - before <= 16
    for i, (w, v) in enumerate(zip(ws, start)):
        for _ in range(4 if i == 3 else 2):
            v = v * np.float32(0.5) + np.float32(0.25)
        got = np.asarray(t.get_tensor_view_value(w))
        if flex:
            np.testing.assert_allclose(got, v, rtol=0, atol=4 * 2.0 ** -14)
        else:
            np.testing.assert_array_equal(got, v)
    t.close()


def _beside_a_copy():
    """Two kernels of one form, the second over what a copy between them lays out."""
    A = ng.make_axis(2880, name="A")
    turned = [ng.make_axis(n, name=c) for n, c in zip((6, 8, 6, 10), "PQST")]
    a, b = ng.placeholder([A]), ng.placeholder(turned)
    return [a * 0.5, ng.axes_with_order(b, turned[::-1]) * 0.5], [a, b]


def _beside_a_pooling():
    axes = [ng.make_axis(n, name=c) for n, c in zip((3, 1, 8, 8, 16), "CDHWN")]
    half = [axes[0], axes[1], ng.make_axis(4, name="H"), ng.make_axis(4, name="W"), axes[4]]
    a, b = ng.placeholder(half), ng.placeholder(axes)
    params = dict(op="max", pad_d=0, pad_h=0, pad_w=0, pad_c=0, str_d=1, str_h=2, str_w=2, str_c=1, T=1, R=2, S=2, J=1)
    return [a * 0.5, ng.pooling(params, b, half) * 0.5], [a, b]


BETWEEN = [_beside_a_copy, _beside_a_pooling]


@pytest.mark.parametrize("graph", BETWEEN)
@pytest.mark.parametrize("flex", [False, True])
def test_a_kernel_stays_behind_what_it_reads(flex, graph, monkeypatch):
    """Steps without exponents of their own (copies, pooling) count as writers where launches are joined."""
    monkeypatch.setattr(lib.PlannedKernel, "joint_source", lambda self: b"one form")
    monkeypatch.setattr(lib.PlannedKernel, "prepare_joint", lambda self: None, raising=False)
    outs, params = graph()
    t = ng.transformers.allocate_transformer("b200", plan_only=True, flex=flex)
    comp = t.computation(outs, *params)
    t.initialize()
    for s in comp.steps:
        for follower in getattr(s, "joint", ())[1:]:
            between = comp.steps[comp.steps.index(s):comp.steps.index(follower)]
            written = set(v.buffer for step in between for v in step.out_views)
            assert not written & set(v.buffer for v in follower.in_views)


@pytest.mark.gpu
@pytest.mark.parametrize("graph", BETWEEN)
@pytest.mark.parametrize("flex", [False, True])
def test_values_behind_a_copy_or_a_pooling(flex, graph):
    outs, params = graph()
    t = ng.transformers.allocate_transformer("b200", flex=flex)
    comp = t.computation(outs, *params)
    rng = np.random.RandomState(2)
    for i in range(4):
        a, b = [rng.uniform(-1, 1, [x.length for x in p.axes]).astype(np.float32) for p in params]
        got = comp(a, b)
        want = b.transpose(3, 2, 1, 0) if graph is _beside_a_copy else \
            b.reshape(3, 1, 4, 2, 4, 2, 16).max(axis=(3, 5))
        for x, y in zip(got, (a, want)):
            np.testing.assert_allclose(x, y * 0.5, rtol=0, atol=2.0 ** -13 if flex else 0)
        if i == 1:
            comp.capture()
    t.close()
