"""Convolutions whose filters the computation makes itself -- an elementwise result, a dense copy of a view --
or whose variable another computation overwrites with a copy: every call, recorded or not, uses the filters as
they are then.  Against torch in double precision."""
import numpy as np
import pytest

import ngraph_python_b200 as ng
from ngraph_python_b200 import configs, kernels

KINDS = ["computed", "turned", "overwritten"]


def _net(kind):
    """Four layers with ReLU tails: (results, the last one that of the layers, input, the variables, what a layer's
    filters are of its variable, assignments that copy the variables into the filters)."""
    ax = lambda length, name: ng.make_axis(length, name=name)   # noqa: E731
    N, D, T, M = ax(20, "N"), ax(1, "D"), ax(1, "T"), ax(1, "M")
    H, W, R, S = ax(16, "H"), ax(16, "W"), ax(3, "R"), ax(3, "S")
    x = ng.placeholder([ax(16, "C"), D, H, W, N])
    shapes = []
    for i in range(4):
        shapes.append([shapes[-1][-1] if shapes else x.axes[0], T, R, S, ax(16, "K%d" % i)])
    # (turned views are laid out dense by a copy)
    store = [s if kind == "computed" else s[::-1] for s in shapes]
    variables = [ng.variable(s, initial_value=np.zeros([a.length for a in s], np.float32)) for s in store]
    outside, writes = variables, []
    if kind == "computed":
        filters = [ng.tanh(v) for v in variables]
    elif kind == "turned":
        filters = [ng.axes_with_order(v, s) for v, s in zip(variables, shapes)]
    else:
        filters = [ng.variable(s, initial_value=np.zeros([a.length for a in s], np.float32)) for s in shapes]
        writes = [ng.assign(f, ng.axes_with_order(v, s)) for f, v, s in zip(filters, variables, shapes)]
    cur = x
    for i, f in enumerate(filters):
        o = ng.convolution(configs._conv_params(1, 1), cur, f, axes=[f.axes[-1], M, H, W, N])
        cur = ng.maximum(ng.cast_axes(o, [f.axes[-1], D, H, W, N]), 0.0)
    of = np.tanh if kind == "computed" else lambda v: v.transpose(4, 3, 2, 1, 0)
    # (computed filters first, so that the layers are neighbours)
    return (filters if kind == "computed" else []) + [cur], x, outside, of, writes


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("flex", [False, True])
def test_plans(flex, kind):
    outs, x, variables, _, writes = _net(kind)
    t = ng.transformers.allocate_transformer("b200", plan_only=True, flex=flex)
    comp = t.computation(outs, x)
    writer = t.computation(ng.sequential(writes)) if writes else None
    t.initialize()
    convs = [s for s in comp.steps if s.kind == "conv"]
    bufs = [s.in_views[1].buffer for s in convs]
    assert len(convs) == 4 and all(s.filters_change == (not writes) for s in convs)
    assert set(bufs) <= set((writer or comp).touched)
    # layers whose filters stay as they are make a run
    run = kernels.chain_convolutions(comp.steps, set(v.buffer for v in comp.return_views), t)
    assert any(s.kind == "conv_chain" for s in run) == (flex and bool(writes))
    for b, s in zip(bufs, convs):
        if s.use_planes or s.tiles:
            assert b.watched


@pytest.mark.gpu
@pytest.mark.parametrize("capture", [False, True])
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("flex", [False, True])
def test_every_call_uses_the_filters_of_then(flex, kind, capture):
    import torch
    outs, x, variables, of, writes = _net(kind)
    t = ng.transformers.allocate_transformer("b200", flex=flex)
    comp = t.computation(outs, x)
    writer = t.computation(ng.sequential(writes)) if writes else None
    t.initialize()
    rng = np.random.RandomState(5)
    value = rng.uniform(-1, 1, [a.length for a in x.axes]).astype(np.float32)
    # (the first call has the largest values: later ones fit the exponents that it chose)
    for i, scale in enumerate((0.3, 0.2, 0.25, 0.2, 0.25)):
        want = torch.from_numpy(value[:, 0]).double().permute(3, 0, 1, 2)
        for v in variables:
            new = rng.uniform(-scale, scale, [a.length for a in v.axes]).astype(np.float32)
            t.device_tensor(v)[...] = new
            f = torch.from_numpy(of(new).astype(np.float64)[:, 0]).permute(3, 0, 1, 2).contiguous()
            want = torch.nn.functional.conv2d(want, f, padding=1).clamp(min=0)
        if writer is not None:
            writer()
        got = np.asarray(comp(value)[-1])[:, 0]
        want = want.permute(1, 2, 3, 0).numpy()
        # fp32: sums of 144 products; flex16: four layers, each rounded to 16 bits
        assert np.abs(got - want).max() <= (2e-3 if flex else 1e-5) * np.abs(want).max(), i
        if capture and i == 1:
            comp.capture()
    t.close()
