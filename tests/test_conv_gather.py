"""fp32 convolutions on filters laid out beforehand whose images come in fours: the kernel that copies sixteen bytes at
a time, its four-byte copies (a tensor that does not start on sixteen bytes), one k-block to many, slices, each tile
width, rows beyond the last tile; against torch in double precision, with and without tails."""
import ctypes as C

import pytest

from ngraph_python_b200 import lib
from tests.test_conv_filter_tiles import _dims

pytestmark = pytest.mark.gpu

# C, H, W, N, K, R, S, pad, stride, dilation
CASES = [(8, 5, 5, 4, 8, 1, 1, 0, 1, 1), (32, 4, 4, 32, 16, 1, 1, 0, 1, 1), (33, 5, 6, 12, 24, 3, 3, 1, 1, 1),
         (16, 16, 16, 100, 16, 3, 3, 1, 1, 1), (64, 8, 8, 16, 64, 3, 3, 1, 1, 1), (96, 7, 7, 36, 96, 3, 3, 1, 2, 1),
         (160, 6, 6, 8, 136, 3, 3, 1, 1, 1)]


@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("shift", [0, 1])
def test_both_passes(case, shift):
    import torch
    raw, g, d = lib.raw(), torch.Generator().manual_seed(sum(case)), _dims(case)
    status = torch.zeros((1,), dtype=torch.int32, device="cuda")
    f = torch.randn((d.C, d.R, d.S, d.K), generator=g)
    df, fn = f.cuda(), f.double().permute(3, 0, 1, 2)
    for conv_pass in (lib.CONV_FPROP, lib.CONV_BPROP):
        nbytes = lib.conv_filter_tiles_info(d, conv_pass)
        if not nbytes:
            continue
        tiles = torch.full((nbytes + 128,), 0x7f, dtype=torch.uint8, device="cuda")
        off, n = -tiles.data_ptr() % 128, C.c_int32()
        job = (lib.ConvFilterJob * 1)(lib.ConvFilterJob(filters=df.data_ptr(), planes=tiles.data_ptr() + off, dims=d,
                                                        conv_pass=conv_pass))
        lib.check(raw.b2_conv_filter_tiles(job, 1, C.byref(n), 0))
        fprop = conv_pass == lib.CONV_FPROP
        ins, outs = ((d.C, d.H, d.W, d.N), (d.K, d.P, d.Q, d.N))[::1 if fprop else -1]
        x, other, act, bias = (torch.randn(s, generator=g) for s in (ins, outs, outs, outs[:1]))
        xn = x.double().permute(3, 0, 1, 2)
        y = (torch.nn.functional.conv2d(xn, fn, stride=case[8], padding=case[7]) if fprop else
             torch.nn.grad.conv2d_input((d.N, d.C, d.H, d.W), fn, xn, stride=case[8], padding=case[7])).permute(1, 2, 3, 0)
        flat = torch.full((x.numel() + 8,), float("nan"), device="cuda")
        flat[shift:shift + x.numel()] = x.reshape(-1).cuda()
        keep = [v.cuda() for v in (bias, other, act)]
        for tail in (False, True):
            out = torch.full(outs, 7.0, device="cuda")
            at = [keep[0].data_ptr() if tail and fprop else None, keep[1].data_ptr() if tail else None,
                  keep[2].data_ptr() if tail and not fprop else None]
            lib.check(raw.b2_conv_f32_tiles(conv_pass, flat.data_ptr() + 4 * shift, tiles.data_ptr() + off, out.data_ptr(),
                                            C.byref(d), at[0], at[1], int(tail and fprop), at[2], status.data_ptr(), 0))
            torch.cuda.synchronize()
            want = y
            if tail:
                want = y + other.double()
                want = (want + bias.double()[:, None, None, None]).clamp(min=0) if fprop else want * (act > 0)
            # (the bar of the convolutions that take their filters as they lie)
            assert (out.cpu().double() - want).abs().max() <= 4e-6 * want.abs().max(), (case, conv_pass, tail)
    assert int(status.item()) == 0
