"""The exponent bookkeeping of a call's arguments goes with that of the tensors it writes in one native
pass; every entry makes the choice of the rule applied to it alone."""
import numpy as np

from ngraph_python_b200 import flex as F
from tests.golden import cases
from tests.test_flex_manager_cpu import _bookkeeping_transformer


def test_arguments_follow_the_rule_entry_by_entry():
    import ngraph_python_b200 as ng
    t, comp = _bookkeeping_transformer(ng, cases.resnet8_small)
    inputs = list(comp.param_buffers)
    assert inputs and not set(map(id, inputs)) & set(map(id, comp.written))
    mirror = {id(b): F.FlexEntry(k) for k, b in enumerate(inputs)}
    rng = np.random.RandomState(6)
    level = {id(b): rng.uniform(0.05, 50.0) for b in inputs}
    for call in range(60):
        # the last argument is not written in every call
        given = inputs[:-1] if len(inputs) > 1 and call % 7 == 3 else inputs
        t._begin_call_flex(comp)
        t._inputs_written = list(given)
        stats = t._stats_host.numpy()
        stats[:] = 100
        for b in inputs:
            want = mirror[id(b)].begin_write()
            assert b.entry.dec == want, "call %d, %s" % (call, b.name)
        for b in given:
            if call < 25:
                level[id(b)] *= rng.uniform(0.8, 1.3)        # a drifting range, then a fixed one
            m = int(min(np.rint(level[id(b)] * 2.0 ** b.entry.dec), 32768))
            stats[b.slot] = m
            mirror[id(b)].end_write(m)
        steady = comp._steady
        t._end_call_flex(comp)
        if steady is None or comp._steady is not steady:
            for b in inputs:
                assert b.entry.pending_dec == mirror[id(b)].pending_dec, "call %d, %s" % (call, b.name)
    t.close()
