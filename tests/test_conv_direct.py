"""Convolutions that gather and convert their operands inside the product, with and without the layer's
tail, against torch in double precision: remainders of the 128-row tiles and of the 32-column blocks,
one and several tiles of channels, windows of 31 taps (the most a row's mask holds) and of 32 (the
unrolled path), strides and dilation."""
import ctypes as C

import pytest

from ngraph_python_b200 import lib

pytestmark = pytest.mark.gpu

# C, H, W, N, K, R, S, pad, stride, dilation, launches of the forward pass
CASES = [(3, 9, 7, 5, 17, 3, 3, 1, 1, 1, 1), (16, 8, 8, 100, 16, 3, 3, 1, 1, 1, 1),
         (5, 8, 9, 33, 40, 5, 5, 2, 2, 1, 1), (130, 5, 5, 20, 130, 3, 3, 2, 1, 2, 1),
         (2, 3, 40, 130, 9, 1, 31, 0, 1, 1, 1), (2, 3, 40, 130, 9, 1, 32, 0, 1, 1, 3),
         (64, 8, 8, 1, 64, 3, 3, 1, 1, 1, 1), (20, 33, 31, 40, 70, 3, 2, 1, 1, 1, 1), (33, 6, 6, 64, 32, 1, 1, 0, 2, 1, 1),
         # tiles of several pixels with ragged edges: forward, both passes, a strided gradient
         (3, 31, 33, 100, 16, 3, 3, 1, 1, 1, 1), (16, 31, 33, 250, 16, 3, 3, 1, 1, 1, 1),
         (16, 31, 33, 100, 32, 3, 3, 1, 2, 1, 1)]


@pytest.mark.parametrize("case", CASES)
def test_fp32_convolution_passes(case):
    import torch
    Cc, H, W, N, K, R, S, pad, st, dil, launches = case
    P, Q = (H + 2 * pad - dil * (R - 1) - 1) // st + 1, (W + 2 * pad - dil * (S - 1) - 1) // st + 1
    d = lib.ConvDims()
    for k, v in dict(C=Cc, D=1, H=H, W=W, N=N, K=K, T=1, R=R, S=S, M=1, P=P, Q=Q, pad_h=pad, pad_w=pad,
                     str_d=1, str_h=st, str_w=st, dil_d=1, dil_h=dil, dil_w=dil).items():
        setattr(d, k, v)
    g = torch.Generator().manual_seed(5)
    x, f = torch.randn((Cc, H, W, N), generator=g), torch.randn((Cc, R, S, K), generator=g)
    e, b = torch.randn((K, P, Q, N), generator=g), torch.randn((K,), generator=g)
    dx, df, de, db = (v.cuda() for v in (x, f, e, b))
    xn, fn, en = (v.double().permute(3, 0, 1, 2) for v in (x, f, e))
    raw = lib.raw()
    status = torch.zeros((1,), dtype=torch.int32, device="cuda")

    def run(fn_, size, args, shape):
        scratch = torch.empty((size + 1024,), dtype=torch.uint8, device="cuda")
        out = torch.full(shape, 7.0, device="cuda")
        sp = scratch.data_ptr() + (-scratch.data_ptr()) % 1024
        lib.check(fn_(args[0].data_ptr(), args[1].data_ptr(), out.data_ptr(), C.byref(d), sp, size,
                      status.data_ptr(), 0))
        torch.cuda.synchronize()
        return out.cpu().double()

    def close(got, want):
        assert (got - want).abs().max() <= 4e-6 * want.abs().max()

    assert lib.conv_launches(False, d, lib.CONV_FPROP) == launches
    y = torch.nn.functional.conv2d(xn, fn, stride=st, padding=pad, dilation=dil).permute(1, 2, 3, 0)
    close(run(raw.b2_conv_fprop_f32, lib.conv_fprop_scratch_bytes(False, d), (dx, df), (K, P, Q, N)), y)
    gx = torch.nn.grad.conv2d_input(xn.shape, fn, en, stride=st, padding=pad, dilation=dil)
    close(run(raw.b2_conv_bprop_f32, lib.conv_bprop_scratch_bytes(False, d), (de, df), (Cc, H, W, N)),
          gx.permute(1, 2, 3, 0))
    gf = torch.nn.grad.conv2d_weight(xn, fn.shape, en, stride=st, padding=pad, dilation=dil)
    close(run(raw.b2_conv_update_f32, lib.conv_update_scratch_bytes(False, d), (dx, de), (Cc, R, S, K)),
          gf.permute(1, 2, 3, 0))
    if launches != 1:
        return
    for bias, res, relu in ((db, de, 1), (db, None, 0), (None, de, 0)):
        out = torch.full((K, P, Q, N), 7.0, device="cuda")
        lib.check(raw.b2_conv_fprop_f32_fused(
            dx.data_ptr(), df.data_ptr(), out.data_ptr(), C.byref(d),
            bias.data_ptr() if bias is not None else None, res.data_ptr() if res is not None else None,
            relu, status.data_ptr(), 0))
        torch.cuda.synchronize()
        want = y.clone()
        want = want + b.double()[:, None, None, None] if bias is not None else want
        want = want + e.double() if res is not None else want
        close(out.cpu().double(), want.clamp(min=0) if relu else want)
    if lib.conv_launches(False, d, lib.CONV_BPROP) == 1:
        other, act = torch.randn(x.shape, generator=g), torch.randn(x.shape, generator=g)
        for res, mask in ((other, act), (None, act), (other, None)):
            out = torch.full(x.shape, 7.0, device="cuda")
            keep = [None if v is None else v.cuda() for v in (res, mask)]
            lib.check(raw.b2_conv_bprop_f32_fused(
                de.data_ptr(), df.data_ptr(), out.data_ptr(), C.byref(d),
                *(None if v is None else v.data_ptr() for v in keep), status.data_ptr(), 0))
            torch.cuda.synchronize()
            want = gx.permute(1, 2, 3, 0) + (0 if res is None else res.double())
            close(out.cpu().double(), want if mask is None else want * (mask > 0))
    assert int(status.item()) == 0


def test_filter_gradient_in_rounds():
    """More slices than the scratch holds at once: 28 copies of the filters fit, five rounds."""
    import torch
    Cc, side, N, K = 512, 32, 64, 512
    d = lib.ConvDims()
    for k, v in dict(C=Cc, D=1, H=side, W=side, N=N, K=K, T=1, R=3, S=3, M=1, P=side, Q=side, pad_h=1, pad_w=1,
                     str_d=1, str_h=1, str_w=1, dil_d=1, dil_h=1, dil_w=1).items():
        setattr(d, k, v)
    size = lib.conv_update_scratch_bytes(False, d)
    launches = lib.conv_launches(False, d, lib.CONV_UPDATE)
    assert size <= 256 << 20 and launches == 10
    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn((Cc, side, side, N), device="cuda", generator=g)
    e = torch.randn((K, side, side, N), device="cuda", generator=g)
    scratch = torch.empty((size + 2048,), dtype=torch.uint8, device="cuda").fill_(77)
    off = -scratch.data_ptr() % 1024
    out = torch.full((Cc, 3, 3, K), 7.0, device="cuda")
    status = torch.zeros((1,), dtype=torch.int32, device="cuda")
    for _ in range(2):                               # the second call on what the first left
        lib.check(lib.raw().b2_conv_update_f32(x.data_ptr(), e.data_ptr(), out.data_ptr(), C.byref(d),
                                               scratch.data_ptr() + off, size, status.data_ptr(), 0))
    torch.cuda.synchronize()
    assert int(status.item()) == 0 and bool((scratch[off + size:] == 77).all())
    padded = torch.nn.functional.pad(x.double(), (0, 0, 1, 1, 1, 1))
    ed = e.double().reshape(K, -1)
    for r in range(3):
        for s in range(3):
            want = padded[:, r:r + side, s:s + side].reshape(Cc, -1) @ ed.T
            assert (out[:, r, s].double() - want).abs().max() <= 4e-6 * want.abs().max()
