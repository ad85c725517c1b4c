"""Which kernel a matrix product takes, at the sizes where the choice was measured to matter (one B200): products that a
line in K and in the number of results sent to a slower kernel, and edges of the rule.  What each computes is checked
beside the others' by the tests of the dispatch."""
import random

import pytest

import ngraph_python_b200 as ng
from ngraph_python_b200 import lib
from tests.test_gemm_dispatch import _run

#         flex, layout, M, N, K, kernel
ROUTES = [
    (True, "nn", 512, 128, 784, "stream"), (True, "nn", 7053, 271, 336, "stream"), (True, "nn", 4735, 178, 206, "stream"),
    (True, "nn", 2984, 135, 2684, "stream"), (True, "nt", 448, 84, 3072, "stream"), (True, "nt", 64, 65, 27, "stream"),
    # many k-blocks to a CTA, both operands along K
    (True, "nt", 78, 3096, 3360, "direct"), (True, "nt", 4396, 44, 5248, "direct"), (True, "nt", 78, 3096, 3361, "stream"),
    # one k-block: few results along K off sixteen bytes, or many
    (True, "nt", 7, 128, 31, "direct"), (True, "nt", 7, 128, 32, "stream"), (True, "nn", 7, 128, 31, "stream"),
    (True, "nn", 2929, 567, 122, "direct"), (True, "nn", 1500, 250, 122, "stream"),
    (True, "nt", 1759, 1045, 6261, "planes"), (True, "nt", 546, 2841, 3841, "planes"),
    (False, "nn", 512, 128, 512, "stream"), (False, "tn", 1489, 605, 176, "direct"), (False, "tn", 1784, 508, 952, "planes"),
    (False, "nt", 3291, 704, 144, "direct"), (False, "nn", 512, 128, 128, "direct"), (False, "nt", 99, 1347, 2389, "direct"),
]


def _strides(layout, M, N, K):
    return ((1, M) if layout == "tn" else (K, 1)), ((1, K) if layout == "nt" else (N, 1))


def _route(flex, layout, M, N, K):
    return lib.gemm_route(flex, *_strides(layout, M, N, K), M, N, K)


@pytest.mark.parametrize("flex,layout,M,N,K,kernel", ROUTES)
def test_kernel(flex, layout, M, N, K, kernel):
    taken, _, _, _, launches = _route(flex, layout, M, N, K)
    want = {"stream": (lib.GEMM_STREAM,), "direct": (lib.GEMM_DIRECT,), "planes": (lib.GEMM_PAIRS, lib.GEMM_TILES)}[kernel]
    assert taken in want and (launches == 1) == (kernel != "planes")


def test_queries_without_row_strides_mean_dense_operands():
    rng = random.Random(2)
    for _ in range(2000):
        flex, layout = rng.random() < 0.5, rng.choice(["nn", "nt", "tn"])
        M, N, K = (int(2 ** rng.uniform(1, 13)) for _ in range(3))
        (_, a_k), (b_k, _) = _strides(layout, M, N, K)
        kernel, *rest, launches = _route(flex, layout, M, N, K)
        assert lib.gemm_launches(flex, a_k, b_k, M, N, K) == launches
        assert lib.gemm_plan(flex, a_k, b_k, M, N, K) == (lib.GEMM_DIRECT if kernel == lib.GEMM_STREAM else kernel, *rest)
    with pytest.raises(lib.B200Error):
        lib.gemm_route(True, (7, 2), (1, 7), 4, 4, 7)
    # rows further apart, off sixteen bytes
    assert lib.gemm_route(False, (512, 1), (128, 1), 512, 128, 512)[0] == lib.GEMM_STREAM
    assert lib.gemm_route(False, (513, 1), (128, 1), 512, 128, 512)[0] == lib.GEMM_DIRECT


@pytest.mark.gpu
@pytest.mark.parametrize("flex,layout,M,N,K,kernel", [r for r in ROUTES if r[2] * r[3] * r[4] < 2e9])
def test_results(flex, layout, M, N, K, kernel):
    import torch
    _run(torch, flex, layout, M, N, K)


@pytest.mark.parametrize("extra", [0, 1])
def test_a_steps_launches_are_those_of_its_strides(extra):
    """Rows further apart than they are long, off sixteen bytes: on planes, where dense ones take one launch."""
    M, N, K = 1000, 480, 1360
    A, B, W = ng.make_axis(M, name="A"), ng.make_axis(N, name="B"), ng.make_axis(K + extra, name="W")
    x = ng.placeholder([A, W])
    rows = ng.tensor_slice(x, [slice(None), slice(0, K)], axes=ng.make_axes([A, ng.make_axis(K, name="K")])) if extra else x
    y = ng.placeholder([rows.axes[1], B])
    t = ng.transformers.allocate_transformer("b200", plan_only=True)
    comp = t.computation(ng.dot(rows, y), x, y)
    t.initialize()
    step, = [s for s in comp.steps if s.kind == "gemm"]
    assert step.a_str == (K + extra, 1)
    assert step.launches == 1 + extra == lib.gemm_route(False, step.a_str, step.b_str, M, N, K)[-1]
