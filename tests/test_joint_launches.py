"""Updates of one form share a launch: more tensors than one launch takes, sizes that take the vector and
the scalar kernel, one block and several; a tensor that another one depends on stays in order."""
import numpy as np
import pytest

import ngraph_python_b200 as ng

pytestmark = pytest.mark.gpu


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
