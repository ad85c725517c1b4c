"""Every form of the one-launch product with A's planes in tensor memory that a product can take: tile widths, slices of K,
several chains to a CTA, lines on and off sixteen bytes, waves, either operand first.  That these sizes take them is
checked without a device; what they compute as the tests of the dispatch do."""
import pytest

from ngraph_python_b200 import lib
from tests.test_gemm_dispatch import _run
from tests.test_gemm_routes import _route

# flex, layout, M, N, K: columns of a tile, slices
SHAPES = [
    (False, "nt", 1, 1, 652, 16, 1), (False, "nn", 8, 8, 520, 16, 1), (False, "nn", 3368, 8, 2128, 16, 3),
    (False, "tn", 65, 3830, 143, 32, 1), (False, "tn", 3770, 23, 2127, 32, 3), (False, "nt", 400, 304, 528, 32, 2),
    (False, "tn", 956, 584, 200, 64, 1), (False, "tn", 144, 3832, 136, 64, 1), (False, "tn", 2372, 112, 601, 64, 2),
    (False, "tn", 729, 1571, 134, 128, 1), (False, "tn", 1591, 2736, 131, 128, 1), (False, "tn", 136, 3400, 696, 128, 2),
    (True, "tn", 8, 8, 16, 16, 1), (True, "tn", 1, 1, 265, 16, 3), (True, "tn", 89, 2436, 16, 32, 1), (True, "nn", 270, 3771, 160, 32, 1),
    (True, "nt", 897, 18, 825, 32, 7), (True, "tn", 2541, 154, 18, 64, 1), (True, "nn", 3202, 37, 970, 64, 4),
    (True, "nt", 40, 3112, 1592, 64, 5), (True, "tn", 3330, 258, 37, 128, 1), (True, "tn", 296, 3808, 136, 128, 1),
    (True, "nn", 3256, 87, 1549, 128, 5), (True, "tn", 804, 2980, 130, 128, 1),
]


def test_shapes_are_taken():
    forms = set()
    for flex, layout, M, N, K, tile, slices in SHAPES:
        kernel, tile_n, cut, waves, launches = _route(flex, layout, M, N, K)
        assert (kernel, tile_n, cut, launches) == (lib.GEMM_STREAM, tile, slices, 1), (flex, layout, M, N, K)
        forms.add((flex, tile_n, cut > 1))
        forms.add((flex, "waves", waves > 1))
        blocks = -(-(-(-K // 32)) // cut)
        if not flex:
            forms.add(("chains", blocks > 16, cut > 1))
    for flex in (False, True):
        assert forms >= {(flex, n, cut) for n in (16, 32, 64, 128) for cut in (False, True)}
        assert forms >= {(flex, "waves", False), (flex, "waves", True)}
    assert forms >= {("chains", several, cut) for several in (False, True) for cut in (False, True)}


@pytest.mark.gpu
@pytest.mark.parametrize("flex,layout,M,N,K,tile,slices", SHAPES)
def test_results(flex, layout, M, N, K, tile, slices):
    import torch
    for offset in (0, 1):
        _run(torch, flex, layout, M, N, K, offset=offset)
