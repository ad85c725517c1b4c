"""The direct product kernel with two groups of producer warps: k-blocks go to the groups by turns, so
the counts that can go wrong are one more and one less than a round of the ring (2 to 5 k-blocks), odd
ones, a last one that is not whole, and slices of different lengths.  A k-block is 32 fp32 or 128 int16
values; the tolerances are those of the plane kernels' tests (flex16: the exact sum)."""
import pytest

from tests.test_gemm_kernels import test_gemm_f32 as gemm_f32, test_gemm_flex16 as gemm_flex16

pytestmark = pytest.mark.gpu

# M, N, k-blocks, columns missing from the last one
SIZES = [(129, 16, 2, 0), (128, 17, 3, 1), (257, 40, 4, 0), (100, 33, 5, 7), (300, 130, 6, 0),
         (64, 64, 9, 2), (1000, 129, 7, 3), (1, 1, 16, 0), (500, 200, 17, 1), (40, 24, 31, 0)]


@pytest.mark.parametrize("layout", ["nn", "nt", "tn"])
@pytest.mark.parametrize("M,N,blocks,less", SIZES)
def test_fp32(M, N, blocks, less, layout):
    gemm_f32(M, N, blocks * 32 - less, layout)


@pytest.mark.parametrize("layout", ["nn", "nt", "tn"])
@pytest.mark.parametrize("M,N,blocks,less", SIZES)
def test_flex16(M, N, blocks, less, layout):
    gemm_flex16(M, N, blocks * 128 - less, layout)
