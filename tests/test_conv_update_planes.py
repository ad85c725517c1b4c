"""Filter and bias gradients from byte planes against exact integer sums: tiles of 1x1 to 2x2 pixels with
odd edges, ragged batches, several chunks of channels and tiles of filters, strides, the largest window;
twice on one workspace, which a call leaves as it found it."""
import ctypes as C

import numpy as np
import pytest

from ngraph_python_b200 import lib

pytestmark = pytest.mark.gpu

# C, H, W, N, K, R, S, pad, stride
CASES = [(16, 8, 8, 128, 16, 3, 3, 1, 1), (16, 7, 9, 100, 16, 3, 3, 1, 1), (3, 9, 9, 5, 17, 3, 3, 1, 1),
         (32, 8, 8, 130, 40, 3, 3, 1, 1), (70, 6, 6, 16, 70, 1, 1, 0, 2), (16, 9, 9, 33, 32, 3, 3, 1, 2),
         (2, 14, 14, 64, 5, 11, 11, 5, 1), (9, 5, 5, 48, 161, 2, 2, 0, 1), (1, 3, 3, 1, 1, 3, 3, 1, 1)]


def _rescale(v, shift):
    q = np.floor_divide(v, 1 << shift)
    rem = v - (q << shift)
    half = 1 << (shift - 1)
    q = q + ((rem > half) | ((rem == half) & (q & 1 == 1)))
    return np.clip(q, -32768, 32767)


@pytest.mark.parametrize("with_bias", [True, False])
@pytest.mark.parametrize("case", CASES)
def test_update_from_planes(case, with_bias):
    import torch
    Cc, H, W, N, K, R, S, pad, st = case
    P, Q = (H + 2 * pad - R) // st + 1, (W + 2 * pad - S) // st + 1
    d = lib.ConvDims()
    for k, v in dict(C=Cc, D=1, H=H, W=W, N=N, K=K, T=1, R=R, S=S, M=1, P=P, Q=Q, pad_h=pad, pad_w=pad,
                     str_d=1, str_h=st, str_w=st, dil_d=1, dil_h=1, dil_w=1).items():
        setattr(d, k, v)
    rng = np.random.RandomState(3)
    x = rng.randint(-32768, 32768, (Cc, H, W, N)).astype(np.int16)
    e = rng.randint(-32768, 32768, (K, P, Q, N)).astype(np.int16)
    xd = torch.from_numpy(x.astype(np.float64)).permute(3, 0, 1, 2)
    ed = torch.from_numpy(e.astype(np.float64)).permute(3, 0, 1, 2)
    # (whole numbers below 2^53: exact)
    u = torch.nn.grad.conv2d_weight(xd, (K, Cc, R, S), ed, stride=st, padding=pad)
    u = u.permute(1, 2, 3, 0).contiguous().numpy().astype(np.int64)
    b = e.astype(np.int64).sum(axis=(1, 2, 3))

    def planes(a):
        t = torch.from_numpy(a).cuda()
        mem = torch.full((2 * lib.plane_bytes(a.shape) + 1024,), 77, dtype=torch.uint8, device="cuda")
        ptr = mem.data_ptr() + (-mem.data_ptr()) % 1024
        lib.check(lib.raw().b2_conv_split_planes(t.data_ptr(), *a.shape, ptr, 0))
        torch.cuda.synchronize()
        return mem, ptr
    keep_x, px = planes(x)
    keep_e, pe = planes(e)
    ok, nbytes = lib.conv_update_planes_info(d)
    assert ok
    work = torch.zeros((nbytes + 1024,), dtype=torch.uint8, device="cuda")
    wp = work.data_ptr() + (-work.data_ptr()) % 1024
    shift_u = max(1, int(np.abs(u).max()).bit_length() - 15)
    shift_b = max(0, int(np.abs(b).max()).bit_length() - 15)
    table = torch.tensor([[1.0, 1.0], [1.0, 1.0], [2.0 ** shift_u, 2.0 ** -shift_u],
                          [2.0 ** shift_b, 2.0 ** -shift_b]], device="cuda")
    stats = torch.zeros((4,), dtype=torch.int32, device="cuda")
    probe = torch.zeros((2,), dtype=torch.int64, device="cuda")
    status = torch.zeros((1,), dtype=torch.int32, device="cuda")
    out = torch.zeros(u.shape, dtype=torch.int16, device="cuda")
    bias = torch.zeros((K,), dtype=torch.int16, device="cuda")
    for pr in (1, 0, 0):
        out.zero_(), bias.zero_()
        lib.check(lib.raw().b2_conv_update_flex16_planes(
            px, pe, out.data_ptr(), bias.data_ptr() if with_bias else None, C.byref(d), table.data_ptr(),
            0, 1, 2, 3 if with_bias else -1, stats.data_ptr(), wp, probe.data_ptr(), status.data_ptr(), pr, 0))
        torch.cuda.synchronize()
    assert int(status.item()) == 0 and int(work.max().item()) == 0
    want = _rescale(u, shift_u)
    assert np.array_equal(out.cpu().numpy(), want)
    assert int(probe[0].item()) == np.abs(u).max() and int(stats[2].item()) == np.abs(want).max()
    if with_bias:
        want = np.sign(b) * (np.abs(b) >> shift_b)
        assert np.array_equal(bias.cpu().numpy(), np.clip(want, -32768, 32767))
        assert int(probe[1].item()) == np.abs(b).max() and int(stats[3].item()) == np.abs(want).max()
