"""Convolutions whose filters change between calls -- arguments, and variables that another computation
writes, made before or after the one that reads them: a recorded call gives what the steps give."""
import numpy as np
import pytest

import ngraph_python_b200 as ng
from ngraph_python_b200 import configs

pytestmark = pytest.mark.gpu


def _net(filters_are, n):
    """Two layers with ReLU tails: (result, arguments, the filters)."""
    ax = lambda length, name: ng.make_axis(length, name=name)   # noqa: E731
    N, D, T, M = ax(n, "N"), ax(1, "D"), ax(1, "T"), ax(1, "M")
    H, W, R, S = ax(8, "H"), ax(8, "W"), ax(3, "R"), ax(3, "S")
    x = ng.placeholder([ax(16, "C"), D, H, W, N])
    rng = np.random.RandomState(3)
    cur, filters = x, []
    for i, k in enumerate((16, 32)):
        axes = [cur.axes[0], T, R, S, ax(k, "K%d" % i)]
        lengths = [a.length for a in axes]
        f = ng.placeholder(axes) if filters_are == "arguments" else \
            ng.variable(axes, initial_value=(0.1 * rng.standard_normal(lengths)).astype(np.float32))
        filters.append(f)
        o = ng.convolution(configs._conv_params(1, 1), cur, f, axes=[axes[-1], M, H, W, N])
        cur = ng.maximum(ng.cast_axes(o, [axes[-1], D, H, W, N]), 0.0)
    return cur, [x] + (filters if filters_are == "arguments" else []), filters


@pytest.mark.parametrize("n", [16, 20])
@pytest.mark.parametrize("flex", [False, True])
def test_filters_as_arguments(flex, n):
    rng = np.random.RandomState(n)
    out, args, _ = _net("arguments", n)
    calls = [[(s * rng.standard_normal([a.length for a in p.axes])).astype(np.float32) for p in args]
             for s in (0.5, 0.5, 0.4, 0.3)]
    got = []
    for capture in (False, True):
        t = ng.transformers.allocate_transformer("b200", flex=flex)
        comp = t.computation(out, *args)
        res = []
        for i, values in enumerate(calls):
            if capture and i == 1:
                comp.capture()
            res.append(np.array(comp(*values)))
        got.append(res)
        t.close()
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("flex", [False, True])
@pytest.mark.parametrize("writer_first", [False, True])
def test_filters_written_by_another_computation(flex, writer_first):
    rng = np.random.RandomState(1)
    out, (x,), filters = _net("variables", 16)
    value = rng.standard_normal([a.length for a in x.axes]).astype(np.float32)
    got = []
    for capture in (False, True):
        t = ng.transformers.allocate_transformer("b200", flex=flex)
        halve = lambda: t.computation([ng.assign(f, f * 0.5) for f in filters])   # noqa: E731
        write = halve() if writer_first else None
        read = t.computation(out, x)
        write = write or halve()
        res = []
        for i in range(4):
            if capture and i == 1:
                read.capture()
            res.append(np.array(read(value)))
            write()
        got.append(res)
        t.close()
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)
    assert not np.array_equal(got[0][0], got[0][1])
