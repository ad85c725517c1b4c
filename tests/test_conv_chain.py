"""Runs of convolution layers in one launch (b2_conv_chain_*): what makes a chain, and that recorded
calls, which use it, give bit for bit what the layers give one by one."""
import numpy as np
import pytest

import ngraph_python_b200 as ng
from ngraph_python_b200 import configs, lib


def _layer(x, res, C, H, K, R, stride, N, W=None, dil=1):
    d = lib.ConvDims()
    W = W or H
    d.C, d.H, d.W, d.N, d.K, d.R, d.S = C, H, W, N, K, R, R
    d.D = d.T = d.M = d.str_d = d.dil_d = 1
    d.pad_h = d.pad_w = R // 2
    d.str_h = d.str_w = stride
    d.dil_h = d.dil_w = dil
    d.P, d.Q = [(n + 2 * (R // 2) - dil * (R - 1) - 1) // stride + 1 for n in (H, W)]
    return lib.ConvChainLayer(dims=d, input=x, residual=res, relu=1)


NONE = lib.CHAIN_NONE


@pytest.mark.parametrize("layers,ok", [
    ([_layer(-1, NONE, 3, 32, 16, 3, 1, 256), _layer(0, NONE, 16, 32, 16, 3, 1, 256)], True),
    ([_layer(-1, NONE, 3, 32, 16, 3, 1, 256), _layer(0, -1, 16, 32, 16, 3, 1, 256)], False),   # 3 + 16
    ([_layer(-1, NONE, 16, 32, 16, 3, 1, 256), _layer(0, -1, 16, 32, 16, 3, 1, 256)], True),
    ([_layer(-1, NONE, 3, 32, 20, 3, 1, 256), _layer(0, NONE, 20, 32, 16, 3, 1, 256)], False),
    ([_layer(-1, NONE, 3, 32, 16, 3, 1, 256, dil=2), _layer(0, NONE, 16, 30, 16, 3, 1, 256)], False),
    ([_layer(-1, NONE, 3, 64, 16, 3, 1, 256), _layer(0, NONE, 16, 64, 16, 3, 1, 256)], False),  # too large
    # one tensor read at both strides
    ([_layer(-1, NONE, 3, 16, 16, 3, 1, 8), _layer(0, NONE, 16, 16, 16, 3, 1, 8),
      _layer(0, NONE, 16, 16, 16, 3, 2, 8)], False),
])
def test_what_makes_a_chain(layers, ok):
    assert lib.conv_chain_info(layers)[0] is ok


def _net(n, hw, widths, blocks):
    """The network, its features under the pooling, and a result from the middle as well."""
    outs, params, vals = configs.resnet20(ng, n=n, hw=hw, widths=widths, blocks=blocks)
    return outs, params, vals


def _run(outs, params, vals, capture_after, peek=()):
    scales = (1.0, 1.7, 1.7, 1.0, 0.3)
    t = ng.transformers.allocate_transformer("b200", flex=True)
    comp = t.computation(outs, *params)
    got, chains = [], 0
    for i, sc in enumerate(scales):
        if i == capture_after:
            comp.capture()
            chains = [len(c.members) for c in comp.chains]
        got.append([np.array(r, copy=True) for r in comp(*[v * np.float32(sc) for v in vals])])
        # every exponent decision of the call: the maxima of all tensors it wrote
        got[-1].append(np.array([b.entry.dec for b in comp.written]))
        got[-1].append(t._stats_host.numpy()[:-2].copy())      # (the last ones are nobody's)
        got[-1].extend(t.device_tensor(op).get() for op in peek)
    t.close()
    return got, chains


@pytest.mark.gpu
@pytest.mark.parametrize("n,hw,widths,blocks,members", [
    (1, 32, (16, 32, 64), 3, [22]),           # one image to a block
    (148, 32, (16, 32, 64), 1, [10]),
    (149, 32, (16, 32, 64), 1, [10]),         # two, the last block with one
    (256, 32, (16, 32, 64), 3, [22]),
    (300, 32, (16, 32, 64), 2, [16]),         # more blocks than SMs
    (7, 12, (48, 16, 64), 1, [10]),           # three channel groups, ragged tiles
    (160, 20, (16, 48, 64), 2, [16]),
    (128, 8, (16, 32, 64), 1, [10]),
])
def test_recorded_chain_is_bit_identical(n, hw, widths, blocks, members):
    outs, params, vals = _net(n, hw, widths, blocks)
    ref, _ = _run(outs, params, vals, None)
    got, chains = _run(outs, params, vals, 2)
    assert chains == members
    for i, (a, b) in enumerate(zip(ref, got)):
        for k, (x, y) in enumerate(zip(a, b)):
            assert np.array_equal(x, y), "call %d, output %d" % (i, k)


@pytest.mark.gpu
def test_results_inside_a_chain_are_there_for_who_asks():
    """A result that only the chain reads is stored when it is read from outside, one that the
    computation returns always; filters that change between calls are used as they are then."""
    N, D = ng.make_axis(20, name="N"), ng.make_axis(1, name="D")
    H, W = ng.make_axis(16, name="H"), ng.make_axis(16, name="W")
    r = np.random.RandomState(2)
    x = ng.placeholder([ng.make_axis(5, name="C"), D, H, W, N])
    cur, mids, filters = x, [], []
    for i in range(7):
        K, T = ng.make_axis(16, name="C"), ng.make_axis(1, name="T")
        Kt = ng.make_axis(16, name="K%d" % i)
        f = ng.variable([cur.axes[0], T, ng.make_axis(3, name="R%d" % i), ng.make_axis(3, name="S%d" % i), Kt],
                        initial_value=r.standard_normal((cur.axes[0].length, 1, 3, 3, 16)) * 0.2)
        b = ng.variable([K], initial_value=r.standard_normal(16) * 0.1)
        o = ng.convolution(configs._conv_params(1, 1), cur, f, axes=[Kt, ng.make_axis(1, name="M"), H, W, N])
        o = ng.cast_axes(o, [K, D, H, W, N]) + b
        cur = ng.maximum(o + mids[1] if i == 3 else o, 0.0)
        mids.append(cur)
        filters.append(f)
    vals = [r.standard_normal((5, 1, 16, 16, 20)).astype(np.float32)]
    outs = [mids[2], mids[6]]                        # the third result is returned, and read inside
    ref, _ = _run(outs, [x], vals, None)
    got, chains = _run(outs, [x], vals, 1, peek=[mids[1]])
    assert chains == [7]
    for a, b in zip(ref, got):
        for u, v in zip(a[:3], b[:3]):
            assert np.array_equal(u, v)
    one, _ = _run([mids[1]], [x], vals, None)
    for i in range(5):                               # before the recording and after it
        assert np.array_equal(one[i][0], got[i][-1])

    # filters written between calls
    res = []
    for capture in (False, True):
        t = ng.transformers.allocate_transformer("b200", flex=True)
        comp = t.computation([cur], x)
        comp(*vals)
        if capture:
            comp.capture()
        comp(*vals)
        t.device_tensor(filters[1])[...] = np.full((16, 1, 3, 3, 16), 0.11, np.float32)
        res.append(np.array(comp(*vals)[0], copy=True))
        t.close()
    assert np.array_equal(res[0], res[1])
