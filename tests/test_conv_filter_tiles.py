"""fp32 convolutions on filters laid out beforehand (b2_conv_filter_tiles, b2_conv_f32_tiles) against torch in
double precision, in both passes with and without tails: ragged rows, columns and tiles of pixels, one k-block
and slices, wide windows, strides; several filters to a launch, more than one launch takes."""
import ctypes as C

import pytest

from ngraph_python_b200 import lib

pytestmark = pytest.mark.gpu

# C, H, W, N, K, R, S, pad, stride, dilation
CASES = [(3, 9, 7, 5, 17, 3, 3, 1, 1, 1), (16, 8, 8, 100, 16, 3, 3, 1, 1, 1), (5, 8, 9, 33, 40, 5, 5, 2, 2, 1),
         (130, 5, 5, 20, 130, 3, 3, 2, 1, 2), (64, 8, 8, 1, 64, 3, 3, 1, 1, 1), (33, 6, 6, 64, 32, 1, 1, 0, 2, 1),
         (3, 31, 33, 100, 16, 3, 3, 1, 1, 1), (16, 31, 33, 130, 16, 3, 3, 1, 1, 1), (16, 31, 33, 100, 32, 3, 3, 1, 2, 1),
         (32, 16, 16, 100, 32, 3, 3, 1, 1, 1), (64, 8, 8, 100, 64, 3, 3, 1, 1, 1), (256, 7, 7, 8, 256, 3, 3, 1, 1, 1),
         (24, 15, 14, 3, 40, 3, 3, 1, 2, 1), (32, 16, 16, 250, 32, 3, 3, 1, 1, 1), (8, 9, 9, 1, 8, 1, 1, 0, 1, 1)]


def _dims(case):
    Cc, H, W, N, K, R, S, pad, st, dil = case
    P, Q = (H + 2 * pad - dil * (R - 1) - 1) // st + 1, (W + 2 * pad - dil * (S - 1) - 1) // st + 1
    d = lib.ConvDims()
    for k, v in dict(C=Cc, D=1, H=H, W=W, N=N, K=K, T=1, R=R, S=S, M=1, P=P, Q=Q, pad_h=pad, pad_w=pad,
                     str_d=1, str_h=st, str_w=st, dil_d=1, dil_h=dil, dil_w=dil).items():
        setattr(d, k, v)
    return d


def test_both_passes():
    import torch
    raw, g = lib.raw(), torch.Generator().manual_seed(5)
    status = torch.zeros((1,), dtype=torch.int32, device="cuda")
    todo, jobs = [], []
    for case in CASES:
        d = _dims(case)
        f = torch.randn((d.C, d.R, d.S, d.K), generator=g)
        df = f.cuda()
        for conv_pass in (lib.CONV_FPROP, lib.CONV_BPROP):
            nbytes = lib.conv_filter_tiles_info(d, conv_pass)
            if nbytes == 0:
                continue
            assert lib.conv_launches(False, d, conv_pass) == 1
            tiles = torch.full((nbytes + 256,), 0x7f, dtype=torch.uint8, device="cuda")
            off = -tiles.data_ptr() % 128
            todo.append((case, d, conv_pass, f, df, tiles, off, nbytes))
            jobs.append(lib.ConvFilterJob(filters=df.data_ptr(), planes=tiles.data_ptr() + off, dims=d,
                                          conv_pass=conv_pass))
    assert len(todo) > 20 and set(t[2] for t in todo) == {lib.CONV_FPROP, lib.CONV_BPROP}
    n = C.c_int32()
    lib.check(raw.b2_conv_filter_tiles((lib.ConvFilterJob * len(jobs))(*jobs), len(jobs), C.byref(n), 0))
    assert n.value == 2                                     # (16 to a launch)
    for case, d, conv_pass, f, df, tiles, off, nbytes in todo:
        st, pad, dil = case[8], case[7], case[9]
        fn = f.double().permute(3, 0, 1, 2)
        ins, outs = ((d.C, d.H, d.W, d.N), (d.K, d.P, d.Q, d.N))[::1 if conv_pass == lib.CONV_FPROP else -1]
        x, other, act = (torch.randn(s, generator=g) for s in (ins, outs, outs))
        bias = torch.randn((outs[0],), generator=g)
        xn = x.double().permute(3, 0, 1, 2)
        if conv_pass == lib.CONV_FPROP:
            y = torch.nn.functional.conv2d(xn, fn, stride=st, padding=pad, dilation=dil)
        else:
            y = torch.nn.grad.conv2d_input((d.N, d.C, d.H, d.W), fn, xn, stride=st, padding=pad, dilation=dil)
        y = y.permute(1, 2, 3, 0)
        dx, keep = x.cuda(), [v.cuda() for v in (bias, other, act)]
        tails = [(0, 0, 0, 0), (1, 1, 1, 0)] if conv_pass == lib.CONV_FPROP else [(0, 0, 0, 0), (0, 1, 0, 1)]
        for has_bias, has_res, relu, has_mask in tails:
            out = torch.full(outs, 7.0, device="cuda")
            at = [v.data_ptr() if has else None for v, has in zip(keep, (has_bias, has_res, has_mask))]
            lib.check(raw.b2_conv_f32_tiles(conv_pass, dx.data_ptr(), tiles.data_ptr() + off, out.data_ptr(), C.byref(d),
                                            at[0], at[1], relu, at[2], status.data_ptr(), 0))
            torch.cuda.synchronize()
            want = y.clone()
            want = want + bias.double()[:, None, None, None] if has_bias else want
            want = want + other.double() if has_res else want
            want = want.clamp(min=0) if relu else want
            want = want * (act > 0) if has_mask else want
            # (the bar of the convolutions that take their filters as they lie)
            assert (out.cpu().double() - want).abs().max() <= 4e-6 * want.abs().max(), (case, conv_pass)
        edge = torch.cat([tiles[:off], tiles[off + nbytes:]])
        assert bool((edge == 0x7f).all())
    assert int(status.item()) == 0
