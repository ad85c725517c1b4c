"""fp32 convolutions on laid out filters: what the sums lose to the tensor core's rounding, restated here, is not more in
the kernel with A's planes in tensor memory than in the one it stands in for; and the device tests of that kernel do
reach it."""
import math

import pytest

from ngraph_python_b200 import lib
from tests.test_conv_filter_tiles import _dims as _case_dims
from tests.test_conv_gather import CASES, test_both_passes as _both_passes
from tests.test_conv_sums import _dims, _layers

# one and more k-blocks and slices of the widest tiles, which one thread issues
WIDE = [(56, 14, 11, 72, 72, 1, 1, 0, 1, 1), (64, 4, 10, 56, 72, 3, 3, 1, 1, 1), (8, 13, 13, 116, 80, 3, 3, 1, 1, 1),
        (104, 5, 8, 72, 64, 3, 3, 1, 1, 1)]


def _seen(bprop, tile, extent, pad, stride):
    """[pixel of the tile][tap of its window]: whether the pixel's own filter has that tap."""
    lo = -math.floor(-(pad - extent + 1) / stride) if bprop else -pad
    n = math.floor((tile - 1 + pad) / stride) - lo + 1 if bprop else (tile - 1) * stride + extent
    n = max(n, 1)
    return [[0 <= (pad - stride * lo - stride * t + g if bprop else t - stride * g) < extent for t in range(n)]
            for g in range(tile)]


def _loss(d, bprop, plan, sums):
    rows = _seen(bprop, plan.tile_h, d.R, d.pad_h, d.str_h)
    cols = _seen(bprop, plan.tile_w, d.S, d.pad_w, d.str_w)
    read, per, total = d.K if bprop else d.C, -(-plan.blocks // plan.slices), 0.0
    for row in rows:
        for col in cols:
            taps = [r and c for r in row for c in col]
            columns = [t for t in taps for _ in range(read)] if bprop else taps * read
            for first in range(0, plan.blocks, per):
                size, lost = [0] * sums, [0.0] * sums
                for b in range(first, min(first + per, plan.blocks)):
                    for k in range(32 * b, 32 * b + 32, 8):
                        n = sum(columns[k:k + 8])
                        if n:
                            size[b % sums] += n
                            lost[b % sums] += math.sqrt(size[b % sums])
                total += sum(x * x for x in lost)
    return total / (len(rows) * len(cols))


def test_sums_lose_no_more():
    kernels, blocks = {lib.CONV_DIRECT: 0, lib.CONV_GATHER: 0}, 0
    layers = list(_layers(300)) + [_dims(64, 8, 8, 64, 3, 1, 100), _dims(64, 8, 8, 64, 3, 1, 256),
                                   _dims(32, 24, 7, 8, 3, 1, 220), _dims(72, 21, 36, 16, 3, 1, 28)]
    for d in layers:
        for bprop in (0, 1):
            s, plan = lib.conv_f32_sums(d, bprop), lib.conv_f32_plan(d, bprop, 1)
            assert (s is None) == (plan is None) == (lib.conv_filter_tiles_info(d, bprop) == 0)
            if s is None:
                continue
            kernels[s.kernel] += 1
            what = [getattr(d, n) for n in ("C", "H", "W", "K", "R", "str_h", "N")], bprop
            assert s.large == plan.in_one_sum and s.large <= s.small <= 2 * s.large, what
            assert s.loss <= s.other_loss * (1 + 1e-8), what
            if s.kernel == lib.CONV_GATHER:
                assert d.N % 4 == 0
                per, sums = -(-plan.blocks // plan.slices), 2 if plan.tile_n >= 96 else 4
                assert s.large == -(-per // sums) and s.small == -(-per // (sums // 2)), what
                assert abs(_loss(d, bprop, plan, sums) / s.loss - 1) < 1e-9, what
                blocks = max(blocks, plan.blocks)
            else:
                assert s.loss == s.other_loss and s.small == s.large, what
    assert kernels[lib.CONV_GATHER] > 100 and kernels[lib.CONV_DIRECT] > 100 and blocks > 30, (kernels, blocks)


def test_device_cases_reach_the_kernel():
    taken = []
    for case in CASES + WIDE:
        d = _case_dims(case)
        for bprop in (0, 1):
            s = lib.conv_f32_sums(d, bprop)
            if s is not None and s.kernel == lib.CONV_GATHER:
                plan = lib.conv_f32_plan(d, bprop, 1)
                taken.append((plan.tile_n, plan.slices > 1, plan.blocks, plan.tile_h * plan.tile_w))
    assert {t[:2] for t in taken} >= {(n, cut) for n in (16, 64, 96, 128) for cut in (False, True)}, taken
    assert 32 in [t[0] for t in taken] and max(t[3] for t in taken) > 1, taken
    assert min(t[2] for t in taken) == 1 and max(t[2] for t in taken) > 40, taken


@pytest.mark.gpu
@pytest.mark.parametrize("case", WIDE)
@pytest.mark.parametrize("shift", [0, 1])
def test_widest_tiles(case, shift):
    _both_passes(case, shift)


@pytest.mark.parametrize("layer, bprop, kernel", [
    ((3, 32, 32, 16, 3, 1, 128), 1, lib.CONV_DIRECT), ((16, 32, 32, 32, 3, 2, 200), 1, lib.CONV_DIRECT),
    ((8, 14, 35, 24, 5, 1, 480), 0, lib.CONV_DIRECT), ((16, 32, 32, 16, 3, 1, 100), 0, lib.CONV_GATHER),
    ((64, 8, 8, 64, 3, 1, 256), 1, lib.CONV_GATHER), ((24, 16, 35, 56, 3, 2, 144), 1, lib.CONV_GATHER)])
def test_kernel_of_a_layer(layer, bprop, kernel):
    """Several waves in the shape that the other kernel has, two CTAs of it to an SM: that one (measured)."""
    assert lib.conv_f32_sums(_dims(*layer), bprop).kernel == kernel
