"""Fused elementwise kernels on rows that do not start or end on a vector: every remainder, rows of a warp and of a
block, rows cut over blocks, gaps between rows (read by nobody, left as they are), and values at the ends of a row that
must not reach its neighbours."""
import numpy as np
import pytest

from tests.test_ew_kernels import test_c2_flex16 as c2_flex16, test_c2_fp32 as c2_fp32

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flex", [False, True])
@pytest.mark.parametrize("rows,cols", [(150, 1000 + i) for i in range(1, 8)] +
                         [(1025, 65), (1100, 515), (3, 40003), (999, 67), (1001, 4105)])
def test_remainders(rows, cols, flex):
    (c2_flex16 if flex else c2_fp32)(rows, cols)


@pytest.mark.parametrize("flex", [False, True])
@pytest.mark.parametrize("gap", [1, 3, 5])
def test_gaps_between_rows_and_values_at_their_ends(gap, flex):
    import torch
    from ngraph_python_b200 import lib
    A, B, C = 5, 61, 333
    dt = lib.FLEX16 if flex else lib.F32
    sb, sa = C + gap, B * (C + gap) + 2 * gap
    st = (sa, sb, 1)
    prog = lib.make_program((A, B, C), [dict(dtype=dt, slot=0 if flex else -1, strides=st)], [],
                            [("add", 0, 0)], [dict(dtype=dt, slot=1 if flex else -1, strides=st, reg=1)],
                            [dict(dtype=dt, slot=2 if flex else -1, strides=(B, 1, 0), reg=1, redop="max")], lib.REDUCE_C)
    r = np.random.RandomState(gap)
    if flex:
        host = r.randint(-9000, 9000, A * sa).astype(np.int16)
    else:
        host = r.standard_normal(A * sa).astype(np.float32)
    at = (np.arange(A)[:, None, None] * sa + np.arange(B)[None, :, None] * sb + np.arange(C)[None, None, :])
    inside = np.zeros(host.size, bool)
    inside[at] = True
    host[~inside] = 30000 if flex else np.nan
    ends = host[at]
    ends[:, ::2, 0], ends[:, ::3, -1] = (16000, -16000) if flex else (1e30, -1e30)
    host[at] = ends
    x = torch.from_numpy(host).cuda()
    y = torch.full_like(x, 77)
    m = torch.zeros((A * B,), dtype=x.dtype, device="cuda")
    table = torch.ones((3, 2), device="cuda")
    stats = torch.zeros((3,), dtype=torch.int32, device="cuda")
    k = lib.EwKernel(prog)
    scratch = torch.empty((max(k.scratch_bytes, 4),), dtype=torch.uint8, device="cuda")
    k.launch([x.data_ptr()], [y.data_ptr(), m.data_ptr()], flex_table=table.data_ptr(), flex_stats=stats.data_ptr(),
             scratch=scratch.data_ptr(), scratch_bytes=k.scratch_bytes)
    torch.cuda.synchronize()
    got, want = y.cpu().numpy(), 2 * ends.astype(np.float64 if not flex else np.int32)
    assert (got[~inside] == 77).all()
    assert np.array_equal(got[at], want.astype(host.dtype))
    assert np.array_equal(m.cpu().numpy().reshape(A, B), want.max(axis=2).astype(host.dtype))
    if flex:
        assert stats.cpu().tolist()[1:] == [32000, int(np.abs(want.max(axis=2)).max())]


@pytest.mark.parametrize("flex", [False, True])
def test_arguments_in_place(flex):
    """A recorded call: the kernel reads the caller's tensor where it lies and stores the placeholder on the way."""
    import torch
    import ngraph_python_b200 as ng
    rows, cols = 701, 1003
    R, Cc = ng.make_axis(rows, name="R"), ng.make_axis(cols, name="C")
    x, b = ng.placeholder([R, Cc]), ng.variable([R, Cc])
    y = ng.persistent_tensor([R, Cc])
    t = ng.transformers.make_transformer_factory("b200", flex=flex)()
    comp = t.computation([ng.sequential([ng.assign(y, x * b), ng.max(x * b, reduction_axes=[Cc])]), y], x)
    t.initialize()
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    xs = [torch.rand((rows, cols), device="cuda", generator=g) + 0.5 for _ in range(3)]
    t.device_tensor(b)[...] = xs[0]
    comp(xs[1])
    comp.capture()
    for v in (xs[1], xs[2]):
        top, whole = comp(v)
        want = (v * xs[0]).cpu().numpy()
        step = 2.0 ** -11 if flex else 1e-6           # (two quantised factors below 1.5, the product below 2.25)
        np.testing.assert_allclose(whole, want, atol=step)
        np.testing.assert_allclose(top, want.max(axis=1), atol=step)
    t.close()
