"""flex16 tensors that one computation writes in place and another one reads: the reader takes them with the
exponent of the last write, also when that write has moved it."""
import numpy as np
import pytest

import ngraph_python_b200 as ng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("capture", [False, True])
@pytest.mark.parametrize("factor", [0.25, 0.5])
def test_exponents_that_move(factor, capture):
    A, B = ng.make_axis(40, name="A"), ng.make_axis(70, name="B")
    rng = np.random.RandomState(1)
    w0 = rng.uniform(0.5, 1.0, (40, 70)).astype(np.float32)
    x0 = rng.uniform(0.5, 1.0, (70, 16)).astype(np.float32)
    x, w = ng.placeholder([B, ng.make_axis(16, name="N")]), ng.variable([A, B], initial_value=w0)
    t = ng.transformers.allocate_transformer("b200", flex=True)
    read = t.computation([ng.dot(w, x), ng.absolute(w)], x)
    write = t.computation(ng.assign(w, w * factor))
    seen = set()
    for i in range(8):
        got = read(x0)
        held, argument = [np.asarray(t.get_tensor_view_value(v)) for v in (w, x)]
        seen.add(t.device_tensor(w).view.buffer.entry.dec)
        for y, want, view in zip(got, (held @ argument, np.abs(held)), read.return_views):
            assert np.abs(y - want).max() <= view.buffer.entry.scale, i      # (one step of what is stored)
        if capture and i == 1:
            read.capture(), write.capture()
        write()
    assert len(seen) > 1
    t.close()
