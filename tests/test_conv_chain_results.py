"""Results inside a run of layers, read from outside after something else has happened: what the last call made,
or an error -- never what the layers would make of later arguments, filters or biases -- and reading one result
leaves the others as they are."""
import numpy as np
import pytest

import ngraph_python_b200 as ng
from ngraph_python_b200 import configs, kernels, lib


class _Net(object):
    """Six layers of 16 channels with bias, ReLU and two residual sums, which read results 1 and 3."""

    def __init__(self, flex=True, returned=(2, 5), behind=False, plan_only=False):
        ax = lambda length, name: ng.make_axis(length, name=name)   # noqa: E731
        N, D, H, W, M, T = ax(20, "N"), ax(1, "D"), ax(16, "H"), ax(16, "W"), ax(1, "M"), ax(1, "T")
        r = np.random.RandomState(2)
        self.x = ng.placeholder([ax(16, "C"), D, H, W, N])
        self.shape = [a.length for a in self.x.axes]
        cur, self.mids, self.filters, self.biases = self.x, [], [], []
        for i in range(6):
            K = ax(16, "C")
            Kt = ax(16, "K%d" % i)
            f = ng.variable([cur.axes[0], T, ax(3, "R%d" % i), ax(3, "S%d" % i), Kt],
                            initial_value=r.standard_normal((16, 1, 3, 3, 16)) * 0.12)
            b = ng.variable([K], initial_value=r.standard_normal(16) * 0.1)
            o = ng.convolution(configs._conv_params(1, 1), cur, f, axes=[Kt, M, H, W, N])
            o = ng.cast_axes(o, [K, D, H, W, N]) + b
            cur = ng.maximum(o + self.mids[i - 2] if i in (3, 5) else o, 0.0)
            self.mids.append(cur)
            self.filters.append(f)
            self.biases.append(b)
        self.t = ng.transformers.allocate_transformer("b200", flex=flex, plan_only=plan_only)
        outs = [self.mids[k] for k in returned]
        if behind:
            outs = [ng.sequential([outs[-1], ng.assign(self.biases[1], self.biases[1] * 0.5), outs[-1]])]
        self.infer = self.t.computation(outs, self.x)
        self.other = self.t.computation(ng.sum(self.x, reduction_axes=self.x.axes), self.x)
        self.inner = self.t.computation(self.mids[1], self.x)
        self.halve = self.t.computation(ng.assign(self.biases[0], self.biases[0] * 0.5))
        self.t.initialize()

    def values(self, seed, scale=1.0):
        return (np.random.RandomState(seed).uniform(-1, 1, self.shape) * scale).astype(np.float32)

    def get(self, k):
        return np.array(self.t.device_tensor(self.mids[k]).get(), copy=True)


def _pair(hold=None):
    """The network step by step and recorded, both after two calls; hold: a result asked for before the recording."""
    nets = _Net(), _Net()
    for net in nets:
        for c in (net.infer, net.other, net.inner):
            c(net.values(0))
        net.halve()
        if hold is not None:
            net.t.device_tensor(net.mids[hold])
    nets[1].infer.capture()
    assert [len(c.members) for c in nets[1].infer.chains] == [6]
    for net in nets:
        net.infer(net.values(1, 0.5))
        net.infer(net.values(2, 0.5))
    return nets


def _write_filter(net):
    net.t.device_tensor(net.filters[4])[...] = np.full((16, 1, 3, 3, 16), 0.03, np.float32)


def _write_window(net):
    net.t.device_tensor(net.filters[0])[2:4] = 0.05


def _write_bias(net):
    net.t.device_tensor(net.biases[3])[...] = np.full(16, 0.25, np.float32)


def _write_argument(net):
    net.t.device_tensor(net.x)[...] = net.values(7, 0.5)


CHANGES = [_write_filter, _write_window, _write_bias, _write_argument,
           lambda net: net.other(net.values(8, 0.5)), lambda net: net.halve()]


@pytest.mark.gpu
@pytest.mark.parametrize("change", range(len(CHANGES)))
def test_refused_once_something_has_changed(change):
    steps, net = _pair()
    for n in (steps, net):
        CHANGES[change](n)
    with pytest.raises(lib.B200Error, match="changed since"):
        net.get(1)
    for k in (2, 5):                                         # what the call stored is there all the same
        assert np.array_equal(net.get(k), steps.get(k))
    for n in (steps, net):
        n.infer(n.values(9, 0.5))
    for k in (0, 1, 2, 3, 4, 5):                             # and the next call has all its results
        assert np.array_equal(net.get(k), steps.get(k)), k


@pytest.mark.gpu
def test_one_result_leaves_the_others():
    steps, net = _pair()
    for n in (steps, net):                                   # (windows keep their tensor's exponent)
        n.t.device_tensor(n.mids[5])[:9] = 0.125
        n.t.device_tensor(n.mids[2])[3:5] = 0.25
    for k in (1, 3, 0, 2, 4, 5, 1):
        assert np.array_equal(net.get(k), steps.get(k)), k


@pytest.mark.gpu
def test_inner_results_then_returned_ones():
    steps, net = _pair()
    for k in (1, 0, 5, 2, 3, 4):
        assert np.array_equal(net.get(k), steps.get(k)), k
    _write_filter(net)                                       # (all were made before)
    assert np.array_equal(net.get(1), steps.get(1))


@pytest.mark.gpu
def test_a_window_written_into_an_inner_result():
    steps, net = _pair()
    for n in (steps, net):
        n.t.device_tensor(n.mids[1])[2:4] = 0.25
    assert np.array_equal(net.get(1), steps.get(1))


@pytest.mark.gpu
def test_the_last_computation_that_made_a_result_counts():
    steps, net = _pair()
    for n in (steps, net):
        n.inner(n.values(4, 0.5))
    assert np.array_equal(net.get(1), steps.get(1))
    with pytest.raises(lib.B200Error, match="changed since"):
        net.get(3)                                           # the argument is that of another call
    for n in (steps, net):
        n.infer(n.values(2, 0.5))
    assert np.array_equal(net.get(1), steps.get(1)) and np.array_equal(net.get(3), steps.get(3))


@pytest.mark.gpu
def test_results_asked_for_before_the_recording_are_stored():
    steps, net = _pair(hold=1)
    for n in (steps, net):
        _write_filter(n)
        n.other(n.values(8, 0.5))
    assert np.array_equal(net.get(1), steps.get(1))
    with pytest.raises(lib.B200Error, match="changed since"):
        net.get(3)
    net.infer.capture()                                      # now both are held; the old call's stays refused
    with pytest.raises(lib.B200Error, match="changed since"):
        net.get(3)
    for n in (steps, net):
        n.infer(n.values(3, 0.5))
        _write_bias(n)
    for k in (1, 3):
        assert np.array_equal(net.get(k), steps.get(k))


def test_no_layer_of_a_run_whose_bias_the_computation_changes_behind_it():
    for behind in (False, True):
        net = _Net(behind=behind, plan_only=True)
        steps = kernels.chain_convolutions(net.infer.steps, set(v.buffer for v in net.infer.return_views), net.t)
        read = [v.buffer for s in steps if s.kind == "conv_chain" for v in s.in_views]
        assert read and (net.t._view_of(net.biases[1]).buffer in read) != behind


@pytest.mark.gpu
def test_no_results_of_a_closed_transformer():
    _, net = _pair()
    tensor = net.t.device_tensor(net.mids[1])
    net.t.close()
    with pytest.raises(lib.B200Error, match="closed"):
        tensor.get()
