"""The pre-pass of the plane products takes both operands in one launch, each its own way: contiguous along K
or along its rows, on 16-byte boundaries or not, in every pairing; flex16 row sums with whole and partial units
and few rows.  Checked through products that take planes, against the plane kernels' tests' bars (flex16: the
exact sum, which the row sums enter)."""
import pytest

from ngraph_python_b200 import lib
from tests.test_gemm_kernels import test_gemm_f32 as gemm_f32, test_gemm_flex16 as gemm_flex16

pytestmark = pytest.mark.gpu

# aligned, K not, M not, N not, none
SIZES = [(1024, 1024, 1040), (1000, 1032, 1547), (1001, 1032, 1552), (1000, 1029, 1552), (1027, 1031, 1553)]


@pytest.mark.parametrize("layout", ["nn", "nt", "tn"])
@pytest.mark.parametrize("M,N,K", SIZES)
@pytest.mark.parametrize("flex", [False, True])
def test_both_operands(flex, M, N, K, layout):
    assert lib.gemm_launches(flex, M if layout == "tn" else 1, 1 if layout == "nt" else N, M, N, K) in (1, 2)
    (gemm_flex16 if flex else gemm_f32)(M, N, K, layout)
