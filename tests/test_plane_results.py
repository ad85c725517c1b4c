"""flex16 results that only convolutions read exist as byte planes alone: read from outside they are what a
computation that returns them stores.  Whole and padded rows of images, planes written by convolutions and by
elementwise kernels, layer by layer and in a run of layers."""
import numpy as np
import pytest

import ngraph_python_b200 as ng
from ngraph_python_b200 import configs

pytestmark = pytest.mark.gpu


def _net(n):
    ax = lambda length, name: ng.make_axis(length, name=name)   # noqa: E731
    N, D, H, W, M, T = ax(n, "N"), ax(1, "D"), ax(16, "H"), ax(16, "W"), ax(1, "M"), ax(1, "T")
    r = np.random.RandomState(n)
    x = ng.placeholder([ax(16, "C"), D, H, W, N])
    cur = ng.tanh(x)
    mids = [cur]
    for i in range(4):
        f = ng.variable([cur.axes[0], T, ax(3, "R"), ax(3, "S"), ax(16, "K%d" % i)],
                        initial_value=r.standard_normal((16, 1, 3, 3, 16)) * 0.12)
        o = ng.convolution(configs._conv_params(1, 1), cur, f, axes=[f.axes[-1], M, H, W, N])
        cur = ng.cast_axes(o, [f.axes[-1], D, H, W, N])
        cur = ng.maximum(cur, 0.0) if i != 1 else cur          # (one result with negative values)
        mids.append(cur)
    values = [r.uniform(-1, 1, [a.length for a in x.axes]).astype(np.float32) * s for s in (1.0, 0.5, 0.7)]
    return x, mids, values


@pytest.mark.parametrize("capture", [False, True])
@pytest.mark.parametrize("n", [16, 20, 32])
def test_read_from_outside(n, capture):
    x, mids, values = _net(n)
    got = []
    for returned in (mids[-1:], mids):
        t = ng.transformers.allocate_transformer("b200", flex=True)
        comp = t.computation(returned, x)
        res = []
        for i, v in enumerate(values):
            out = comp(v)
            res.append([t.device_tensor(m).get() for m in mids] if i and returned is not mids else list(out))
            if capture and i == 0:
                comp.capture()
        alone = [t._view_of(m).buffer in comp.bytes_only for m in mids]
        assert any(alone) == (returned is not mids)
        got.append(res[1:])
        t.close()
    for a, b in zip(*got):
        for k, (u, v) in enumerate(zip(a, b)):
            assert np.abs(v).max() > 0 and np.array_equal(u, v), k
