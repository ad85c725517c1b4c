"""One-launch products at the edges of the kernel that keeps A's planes in tensor memory: one k-block and one column
more, rings that come round, ragged tiles, lines on every place within sixteen bytes, slices, several chains to a CTA.
flex16 equals the int64 product, rescaled; fp32 against float64 (the tolerance of the dispatch tests)."""
import pytest

from tests.test_gemm_dispatch import _run

pytestmark = pytest.mark.gpu

#        one k-block more     ring comes round     unaligned by 1, 2, 3 elements      one narrow tile, many chains
SIZES = [(128, 16, 128), (129, 17, 129), (64, 48, 257), (200, 70, 640), (77, 33, 1023), (260, 96, 301), (66, 130, 514),
         (513, 24, 2500), (24, 513, 2560), (700, 32, 1024), (1, 5, 4096), (304, 528, 768)]


@pytest.mark.parametrize("flex", [False, True])
@pytest.mark.parametrize("layout", ["nn", "nt", "tn"])
@pytest.mark.parametrize("M,N,K", SIZES)
def test_edges(M, N, K, layout, flex):
    import torch
    for offset in (0, 1):
        _run(torch, flex, layout, M, N, K, offset=offset)


def test_many_results_of_one_k_block():
    import torch
    _run(torch, True, "nn", 1501, 701, 100)
    _run(torch, True, "tn", 1500, 600, 128)


def test_products_without_scratch():
    """What one launch did without scratch it still does; what needed it is refused."""
    import torch
    from ngraph_python_b200 import lib
    status = torch.zeros((1,), dtype=torch.int32, device="cuda")
    for M, N, K, taken in ((64, 130, 129, True), (512, 128, 784, True), (300, 40, 2048, True), (4097, 4098, 32, False)):
        a, b = torch.randn((M, K), device="cuda"), torch.randn((K, N), device="cuda")
        c = torch.zeros((M, N), device="cuda")
        rc = lib.raw().b2_gemm_f32(a.data_ptr(), K, 1, b.data_ptr(), N, 1, c.data_ptr(), N, M, N, K, None, 0,
                                   status.data_ptr(), 0)
        torch.cuda.synchronize()
        assert (rc == 0) == taken
        if taken:
            torch.testing.assert_close(c.double(), a.double() @ b.double(), rtol=1e-4, atol=1e-5 * K ** 0.5 * 4)
    assert int(status.item()) == 0
