"""fp32 convolutions that gather their operands: the tensor core's sum loses bits with every k-block that goes
into it, so no shape adds more of them in one go than a kernel with one group of producers, one pair of sums to a
tile and filters as they lie.  That kernel's shape is restated here from its cost rule."""
import math
import random

from ngraph_python_b200 import lib

CLUSTERS = (0, 148, 148, 135, 132, 130, 132, 105, 120)        # CTAs at once in clusters of 1 to 8


def _window(bprop, g, r, pad, stride):
    if not bprop:
        return (g - 1) * stride + r
    return max((g - 1 + pad) // stride + (r - 1 - pad) // stride + 1, 1)


def _plain_shape(rows, columns, depth, tiled, channel_last):
    """(cost, k-blocks in one sum, k-blocks) of the cheapest shape."""
    blocks, best = -(-depth // 32), None
    for bn in (16, 32, 64, 128):
        if bn > 16 and bn // 2 >= columns:
            break
        tiles = -(-rows // 128) * -(-columns // bn)
        for want in range(1, min(8, blocks) + 1):
            per = -(-blocks // want)
            slices = -(-blocks // per)
            ring, table = (3 if bn == 128 else 2) * 2 * (128 + bn) * 128, per * 32 * (16 if tiled else 8)
            if slices != want or per > 16 or 1152 + ring + table > 232448:
                continue
            row_b = 1.0 if not tiled else 3.5 if channel_last else 1.5
            pace = int((128 * 1.5 + bn * row_b) * 7)
            wait = 3500 if bn >= 64 else 1600 + 25 * bn
            ctas, per_sm = tiles * slices, 1 if bn == 128 or 1152 + ring + table > 115000 else 2
            together = 1 if ctas <= 148 else per_sm
            one = 7000 + per * max(together * pace, wait) + together * bn * (24 if slices > 1 else 12)
            one += 0 if slices == 1 else 18000 if tiled else 3000
            cost = -(-ctas // (CLUSTERS[slices] * per_sm)) * one
            if best is None or cost < best[0]:
                best = cost, per, blocks
    return best


def _in_one_sum(d, bprop):
    result, read = (d.C, d.K) if bprop else (d.K, d.C)
    p, q = (d.H, d.W) if bprop else (d.P, d.Q)
    best = None
    for a in (1, 2):
        for b in (1, 2):
            gh, gw = (a * d.str_h, b * d.str_w) if bprop else (a, b)
            tiled = gh * gw > 1
            if tiled and result % 8:
                continue
            th, tw = (_window(bprop, gh, d.R, d.pad_h, d.str_h), _window(bprop, gw, d.S, d.pad_w, d.str_w)) \
                if tiled else (d.R, d.S)
            if th * tw > 31 or read * th * tw > 4608:
                continue
            shape = _plain_shape(-(-p // gh) * -(-q // gw) * d.N, gh * gw * result, read * th * tw, tiled, bprop)
            if shape is not None and (best is None or shape[0] < best[0]):
                best = shape
    return best[1:]


def _dims(C, H, W, K, R, stride, N):
    d = lib.ConvDims()
    d.C, d.H, d.W, d.K, d.R, d.S, d.str_h, d.str_w, d.N = C, H, W, K, R, R, stride, stride, N
    d.D = d.T = d.M = d.str_d = d.dil_d = d.dil_h = d.dil_w = 1
    d.pad_h = d.pad_w = R // 2
    d.P, d.Q = [(n + 2 * (R // 2) - R) // stride + 1 for n in (H, W)]
    return d


def _layers(count):
    """Layers of up to 128 channels (with more of them an unrolled product may be cheaper), and those of the
    22-layer networks."""
    rng = random.Random(7)

    def pick(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    for N in (1, 2, 10, 32, 50, 64, 100, 128, 200, 256, 384, 512, 1000, 1024):
        for C, H, K, R, stride in ((3, 32, 16, 3, 1), (16, 32, 16, 3, 1), (16, 32, 32, 3, 2), (16, 32, 32, 1, 2),
                                   (32, 16, 32, 3, 1), (32, 16, 64, 3, 2), (32, 16, 64, 1, 2), (64, 8, 64, 3, 1)):
            yield _dims(C, H, H, K, R, stride, N)
    for _ in range(count):
        C, K = pick(3, 128), pick(8, 128)
        if rng.random() < 0.7:
            C, K = max(8, C // 8 * 8), K // 8 * 8
        yield _dims(C, pick(4, 40), pick(4, 40), K, rng.choice([1, 1, 3, 3, 3, 5]), rng.choice([1, 1, 2]), pick(1, 512))


def test_no_longer_sums():
    plans = {0: 0, 1: 0}
    for d in _layers(2000):
        for bprop in (0, 1):
            for tiles in (0, 1):
                plan = lib.conv_f32_plan(d, bprop, tiles)
                if plan is None:
                    continue
                plans[tiles] += 1
                most, blocks = _in_one_sum(d, bprop)
                assert 1 <= plan.in_one_sum <= most and (blocks > 1 or plan.blocks == 1), \
                    ([getattr(d, n) for n in ("C", "H", "W", "K", "R", "str_h", "N")], bprop, tiles, most)
    assert plans[0] > 3500 and plans[1] > 2500, plans
