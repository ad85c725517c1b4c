"""Large fp32 arguments of recorded calls: read where the caller's tensor lies by the kernel that uses
them first, which stores them; later kernels, later calls with other kinds of arguments, unrecorded calls
and the placeholder itself see the values of the last call."""
import numpy as np
import pytest

import ngraph_python_b200 as ng
from ngraph_python_b200 import lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows, cols", [(512, 512), (300, 1001), (1, 262144), (64, 4096), (1200, 1024)])
def test_device_arguments_in_place(rows, cols):
    import torch
    A, B = ng.make_axis(rows, name="A"), ng.make_axis(cols, name="B")
    x = ng.placeholder([A, B])
    total = ng.sum(ng.exp(x) + x, reduction_axes=[B])
    again = ng.sum(x, reduction_axes=[A])                    # another kernel reads x after it
    t = ng.transformers.allocate_transformer("b200")
    comp = t.computation([total, again], x)
    other = t.computation(ng.sum(x * x, reduction_axes=[B]), x)
    third = t.computation(ng.max(x, reduction_axes=[B]), x)

    def check(value):
        v = value.cpu().numpy() if isinstance(value, torch.Tensor) else value
        v = v.astype(np.float64)
        got = comp(value)
        np.testing.assert_allclose(got[0], (np.exp(v) + v).sum(axis=1), rtol=2e-5, atol=1e-3)
        np.testing.assert_allclose(got[1], v.sum(axis=0), rtol=2e-5, atol=1e-3)
        np.testing.assert_array_equal(np.asarray(t.get_tensor_view_value(x)), v.astype(np.float32))
        np.testing.assert_allclose(other(value), (v * v).sum(axis=1), rtol=2e-5, atol=1e-3)

    def values(seed, extra=0):
        g = torch.Generator(device="cuda").manual_seed(seed)
        flat = torch.rand((rows * cols + extra,), device="cuda", generator=g)
        return flat[extra:].reshape(rows, cols)
    check(values(1))                                          # before recording
    comp.capture(), other.capture()
    check(values(2))
    check(values(3, extra=1))                                 # not 16-byte aligned
    check(np.random.RandomState(4).rand(rows, cols).astype(np.float32))
    check(values(5).double())                                 # converted on the way
    for pinned in (False, True):
        v = torch.rand((rows, cols), generator=torch.Generator().manual_seed(8))
        v = (v.pin_memory() if pinned else v).numpy()
        v.flags.writeable = False
        check(v)
    v = values(6)                                             # unrecorded, after recorded calls
    np.testing.assert_array_equal(third(v), v.cpu().numpy().max(axis=1))
    check(values(7))
    t.close()


def test_recorded_kernel_beside_an_unaligned_operand():
    """The kernel of a recorded call is compiled before the recording, also where another operand's
    address asks for the scalar variant."""
    import torch
    n = 1 << 18
    A, whole = ng.make_axis(n, name="A"), ng.make_axis(n + 1, name="A")
    w = np.random.RandomState(1).rand(n + 1).astype(np.float32)
    x = ng.placeholder([A])
    shifted = ng.cast_axes(ng.tensor_slice(ng.variable([whole], initial_value=w), (slice(1, None),)), [A])
    t = ng.transformers.allocate_transformer("b200")
    comp = t.computation(x * shifted, x)
    comp(np.zeros(n, np.float32))
    comp.capture()
    step = [s for s in comp.steps if s.kind == "ew"][-1]
    assert step.stores_argument and any(v.offset % 4 for v in step.in_views)
    for seed in (2, 3):
        v = torch.rand((n,), device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed))
        np.testing.assert_array_equal(comp(v), v.cpu().numpy() * w[1:])
        np.testing.assert_array_equal(np.asarray(t.get_tensor_view_value(x)), v.cpu().numpy())
    t.close()


def test_argument_that_the_computation_writes():
    """The caller's tensor is what a kernel before the argument's first reader writes: the argument is
    what the tensor held when the call was made, recorded or not."""
    A, B = ng.make_axis(512, name="A"), ng.make_axis(512, name="B")
    x = ng.placeholder([A, B])
    y = ng.variable([A, B], initial_value=np.ones((512, 512), np.float32))
    doubled = ng.assign(y, y * 2.0)
    total = ng.sum(y, reduction_axes=[A, B])
    t = ng.transformers.allocate_transformer("b200")
    comp = t.computation(ng.sequential([doubled, total, x + total]), x)
    comp(np.zeros((512, 512), np.float32))                    # y = 2
    held = t.device_tensor(y).view.buffer.tensor
    assert len([s for s in comp.steps if s.kind == "ew"]) > 1

    def check(value):
        np.testing.assert_array_equal(comp(held), np.full((512, 512), value + 2 * value * 512 * 512, np.float32))
    check(2.0)
    comp.capture()
    check(4.0)
    check(8.0)
    assert comp.steps[-1].stores_argument
    t.close()


def test_no_call_on_a_closed_transformer():
    """A recorded step list holds the addresses of memory that the transformer has given back."""
    A = ng.make_axis(64, name="A")
    x = ng.placeholder([A])
    t = ng.transformers.allocate_transformer("b200")
    comp = t.computation(ng.exp(x), x)
    comp(np.zeros(64, np.float32))
    comp.capture()
    launched = t.kernel_launches
    t.close()
    with pytest.raises(lib.B200Error, match="closed"):
        comp(np.zeros(64, np.float32))
    assert t.kernel_launches == launched
