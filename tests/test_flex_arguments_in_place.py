"""Large flex16 arguments of recorded calls: the kernel that reads one first takes the caller's fp32 values
as a host write would store them, and stores them.  Against the same call made step by step, where a kernel
of its own has stored them before: every mantissa, maximum and exponent alike."""
import re

import numpy as np
import pytest

import ngraph_python_b200 as ng
from ngraph_python_b200 import lib


@pytest.mark.parametrize("vec", (0, 1))
@pytest.mark.parametrize("mode", (lib.REDUCE_NONE, lib.REDUCE_C, lib.REDUCE_B))
def test_generated_kernel(mode, vec):
    A, B, Cn = 2, 6, 64
    full = (B * Cn, Cn, 1)
    ins = [dict(dtype=lib.FLEX16_AT, slot=3, strides=full), dict(dtype=lib.FLEX16, slot=1, strides=full)]
    outs = [dict(dtype=lib.FLEX16, slot=2, strides=full, reg=2), dict(dtype=lib.FLEX16, slot=3, strides=full, reg=0)]
    red = {lib.REDUCE_NONE: [], lib.REDUCE_C: [(B, 1, 0)], lib.REDUCE_B: [(Cn, 0, 1)]}[mode]
    reds = [dict(dtype=lib.FLEX16, slot=4, strides=st, reg=2, redop="sum") for st in red]
    prog = lib.make_program((A, B, Cn), ins, [], [("mul", 0, 1)], outs, reds, mode)
    src = lib.ew_check(prog, vec=bool(vec), want_source=True)
    body = src[src.index("b2_ew_main"):]
    assert body.count("const bool fp0 = at0 != (const float*)p.out[1];") == 1
    assert re.findall(r"if \(put(\d)\)", body) == ["1"]
    assert ("b2_mantissas(" in body) == bool(vec) and ("b2_as_stored(" in body) == (not vec)
    # a result that stores it has to be there, with the same exponent and layout
    for bad in (dict(outs[1], slot=5), dict(outs[1], strides=(Cn, A * Cn, 1)), dict(outs[1], reg=1)):
        with pytest.raises(lib.B200Error, match="no result that stores it"):
            lib.ew_check(lib.make_program((A, B, Cn), ins, [], [("mul", 0, 1)], [outs[0], bad], reds, mode), vec=bool(vec))


def test_only_the_recorded_program_takes_arguments_in_place():
    R, C = ng.make_axis(512, name="R"), ng.make_axis(1024, name="C")
    x, b = ng.placeholder([R, C]), ng.placeholder([R])
    t = ng.transformers.allocate_transformer("b200", plan_only=True, flex=True)
    comp = t.computation(ng.sum(ng.tanh(x) * b, reduction_axes=[C]), x, b)
    t.initialize()
    step, = comp.steps
    assert [d.dtype for d in step.kernel.prog.inp[:2]] == [lib.FLEX16, lib.FLEX16]
    recorded = step.recorded_program
    at = [i for i in range(2) if recorded.inp[i].dtype == lib.FLEX16_AT]
    assert at == list(step.stores_argument) and step.in_views[at[0]].buffer is t._view_of(x).buffer
    lib.ew_check(recorded)


@pytest.mark.gpu
@pytest.mark.parametrize("rows, cols", [(512, 512), (300, 1001), (1, 262144), (64, 4100), (1200, 1024), (4096, 72)])
def test_device_arguments_in_place(rows, cols):
    import torch
    A, B = ng.make_axis(rows, name="A"), ng.make_axis(cols, name="B")

    def values(seed, scale=1.0, extra=0):
        g = torch.Generator(device="cuda").manual_seed(seed)
        flat = torch.randn((rows * cols + extra,), device="cuda", generator=g) * scale
        special = torch.tensor([0.0, -0.0, -1e-9, 1e9, -1e9, float("inf"), float("-inf"), float("nan")], device="cuda")
        if seed % 2:
            flat[extra:extra + 8] = special
        return flat[extra:].reshape(rows, cols)

    def run(capture):
        x, w = ng.placeholder([A, B]), ng.variable([B], initial_value=np.linspace(-1, 1, cols).astype(np.float32))
        y = ng.tanh(x) * w + x
        t = ng.transformers.allocate_transformer("b200", flex=True)
        comp = t.computation([ng.sum(y, reduction_axes=[B]), ng.max(x, reduction_axes=[A]), y], x)
        out = []
        seq = [values(2), values(4), values(4, 2.5), values(3), values(6, extra=1), values(8).double(),
               values(10).cpu().numpy(), values(12), values(14, 0.1), values(14, 0.1)]
        for i, v in enumerate(seq):
            if capture and i == 1:
                comp.capture()
                assert [s for s in comp.steps if s.kind == "ew" and s.stores_argument]
            out.append([np.array(r, copy=True) for r in comp(v)])
            out[-1].append(np.array(t.get_tensor_view_value(x)))
            out[-1].append(np.array([b.entry.dec for b in list(comp.written) + list(comp.param_buffers)]))
            out[-1].append(t._stats_host.numpy()[:-2].copy())
        t.close()
        return out
    for i, (a, b) in enumerate(zip(run(False), run(True))):
        for k, (u, v) in enumerate(zip(a, b)):
            assert np.array_equal(u, v, equal_nan=True), "call %d, item %d" % (i, k)
