"""How far an infinity or a NaN reaches in fp32 convolutions whose tiles hold several pixels: the results of its
image in the tiles whose window covers it, no others; with filters as they lie and laid out beforehand."""
import ctypes as C

import pytest

from ngraph_python_b200 import lib
from tests.test_conv_sums import _dims

pytestmark = pytest.mark.gpu

# C, H, W, K, R, stride, N: several pixels to a tile in one pass or both, ragged tiles, taps that skip pixels; one pixel
LAYERS = [(16, 32, 32, 16, 3, 1, 100), (16, 31, 33, 32, 3, 1, 100), (16, 31, 33, 32, 3, 2, 100), (16, 32, 32, 32, 1, 2, 100),
          (32, 16, 16, 32, 3, 1, 100), (64, 9, 9, 64, 3, 1, 130)]


def _covered(bprop, tiles, g, r, pad, stride, at):
    """Which of `tiles` tiles of g results have `at` in their window, along one axis."""
    def window(t):
        first, last = t * g, t * g + g - 1
        if not bprop:
            return first * stride - pad, last * stride - pad + r - 1
        return -(-(first + pad - r + 1) // stride), (last + pad) // stride
    return [window(t)[0] <= at <= window(t)[1] for t in range(tiles)]


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("layer", LAYERS)
def test_reach(layer, bad):
    import torch
    raw, d = lib.raw(), _dims(*layer)
    g = torch.Generator(device="cuda").manual_seed(3)
    f = torch.randn((d.C, d.R, d.S, d.K), device="cuda", generator=g)
    status = torch.zeros((1,), dtype=torch.int32, device="cuda")
    sizes = set()
    for bprop in (lib.CONV_FPROP, lib.CONV_BPROP):
        ins, outs = ((d.C, d.H, d.W, d.N), (d.K, d.P, d.Q, d.N))[::-1 if bprop else 1]
        for staged in (False, True):
            plan = lib.conv_f32_plan(d, bprop, staged)
            if plan is None:
                continue
            sizes.add(plan.tile_h * plan.tile_w)
            if staged:
                n, launches = lib.conv_filter_tiles_info(d, bprop), C.c_int32()
                tiles = torch.zeros((n + 128,), dtype=torch.uint8, device="cuda")
                at = tiles.data_ptr() + -tiles.data_ptr() % 128
                job = lib.ConvFilterJob(filters=f.data_ptr(), planes=at, dims=d, conv_pass=bprop)
                lib.check(raw.b2_conv_filter_tiles((lib.ConvFilterJob * 1)(job), 1, C.byref(launches), 0))

            def run(x):
                out = torch.zeros(outs, device="cuda")
                if staged:
                    lib.check(raw.b2_conv_f32_tiles(bprop, x.data_ptr(), at, out.data_ptr(), C.byref(d), None, None, 0,
                                                    None, status.data_ptr(), 0))
                elif bprop:
                    lib.check(raw.b2_conv_bprop_f32_fused(x.data_ptr(), f.data_ptr(), out.data_ptr(), C.byref(d), None,
                                                          None, status.data_ptr(), 0))
                else:
                    lib.check(raw.b2_conv_fprop_f32_fused(x.data_ptr(), f.data_ptr(), out.data_ptr(), C.byref(d), None,
                                                          None, 0, status.data_ptr(), 0))
                torch.cuda.synchronize()
                return out
            x = torch.randn(ins, device="cuda", generator=g)
            finite = run(x)
            for h, w in ((0, 0), (5, 3), (ins[1] - 1, ins[2] - 1)):
                y = x.clone()
                y[2, h, w, 1] = bad
                got = run(y)
                rows = _covered(bprop, -(-outs[1] // plan.tile_h), plan.tile_h, d.R, d.pad_h, d.str_h, h)
                columns = _covered(bprop, -(-outs[2] // plan.tile_w), plan.tile_w, d.S, d.pad_w, d.str_w, w)
                reach = torch.zeros(outs, dtype=torch.bool, device="cuda")
                for p in range(outs[1]):
                    for q in range(outs[2]):
                        if rows[p // plan.tile_h] and columns[q // plan.tile_w]:
                            reach[:, p, q, 1] = True
                assert torch.equal(got.isnan(), reach), (bprop, staged, h, w)
                assert torch.equal(got[~reach], finite[~reach]), (bprop, staged, h, w)
    assert (max(sizes) > 1) == (layer != LAYERS[-1]) and int(status.item()) == 0
