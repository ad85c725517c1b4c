"""What a row of a fused kernel with row reductions goes to -- a warp, a block, several blocks -- and whether in vectors,
where that was measured to matter, and the results on both sides of the lines."""
import re

import pytest

from ngraph_python_b200 import lib
from tests.test_ew_kernels import c2_program, test_c2_flex16 as _c2_flex16, test_c2_fp32 as _c2_fp32

#       flex, rows, columns: values to a load, threads to a row, several blocks
ROWS = [
    (True, 1000, 4096, 8, 256, False), (True, 1024, 2048, 8, 256, False), (False, 1200, 2048, 4, 256, False),
    (True, 1000, 512, 8, 32, False), (True, 1000, 1024, 8, 32, False), (True, 999, 1024, 8, 256, False), (True, 2900, 728, 8, 32, False), (False, 6167, 384, 4, 32, False),
    (True, 2000, 1536, 8, 32, False), (True, 2000, 1544, 8, 256, False), (True, 1999, 1536, 8, 256, False), (True, 1000, 513, 8, 32, False),
    (False, 6000, 1152, 4, 32, False), (False, 5999, 1152, 4, 256, False), (False, 6000, 1156, 4, 256, False),
    # rows that do not start or end on a vector
    (True, 3000, 3001, 8, 256, False), (False, 3370, 937, 4, 256, False), (True, 7972, 861, 8, 32, False),
    (True, 2094, 1446, 8, 32, False), (False, 63, 1041, 1, 256, False), (False, 105, 1066, 4, 256, False), (True, 187, 439, 1, 256, False),
    (True, 20, 15001, 1, 256, True), (True, 31, 8193, 1, 256, True), (True, 32, 9001, 8, 256, True),
    (False, 64, 6115, 4, 256, True), (False, 65, 6115, 4, 256, False), (True, 40, 8177, 8, 256, False),
    (True, 200, 16383, 8, 256, True), (True, 900, 73, 8, 32, False),
]


@pytest.mark.parametrize("flex,rows,cols,vector,threads,cut", ROWS)
def test_plan(flex, rows, cols, vector, threads, cut):
    source = lib.ew_check(c2_program(lib, rows, cols, flex), vec=True, want_source=True)
    assert [int(re.search(r"#define %s (\d+)" % n, source).group(1)) for n in ("V", "GROUP")] == [vector, threads]
    assert ("b2_ew_finalize" in source) == cut


@pytest.mark.gpu
@pytest.mark.parametrize("flex,rows,cols,vector,threads,cut", [r for r in ROWS if r[1] * r[2] < 4e6])
def test_results(flex, rows, cols, vector, threads, cut):
    (_c2_flex16 if flex else _c2_fp32)(rows, cols)

# two tensors read, one sum: the same
LIGHT = [
    (True, 1000, 1760, 8, 32, False), (True, 1000, 1768, 8, 256, False), (True, 2340, 2784, 8, 32, False),
    (True, 1079, 2464, 8, 256, False), (True, 2100, 1897, 8, 32, False), (True, 3000, 3001, 8, 256, False),
    (False, 1024, 2048, 4, 32, False), (False, 1000, 4096, 4, 256, False), (False, 999, 2048, 4, 256, False),
    (False, 1786, 1093, 4, 32, False), (False, 1024, 1999, 1, 256, False), (False, 4520, 1502, 4, 32, False),
    (False, 1010, 4001, 1, 256, False), (False, 766, 11787, 1, 256, False), (False, 293, 2767, 4, 256, False),
    (False, 16, 7001, 4, 256, False), (True, 15, 7001, 8, 256, False), (True, 4100, 4096, 8, 32, False),
]


def _light_program(rows, cols, flex):
    dt = lib.FLEX16 if flex else lib.F32
    ins = [dict(dtype=dt, slot=k if flex else -1, strides=(rows * cols, cols, 1)) for k in range(2)]
    return lib.make_program((1, rows, cols), ins, [], [("mul", 0, 1)], [],
                            [dict(dtype=dt, slot=2 if flex else -1, strides=(rows, 1, 0), reg=2, redop="sum")], lib.REDUCE_C)


@pytest.mark.parametrize("flex,rows,cols,vector,threads,cut", LIGHT)
def test_plan_of_a_sum(flex, rows, cols, vector, threads, cut):
    source = lib.ew_check(_light_program(rows, cols, flex), vec=True, want_source=True)
    assert [int(re.search(r"#define %s (\d+)" % n, source).group(1)) for n in ("V", "GROUP")] == [vector, threads]
    assert ("b2_ew_finalize" in source) == cut


def test_sums_of_single_values_are_not_a_warps():
    """Tensors that do not start on a vector: a lane would add more values one after another than a thread of a block."""
    for flex in (False, True):
        for rows, cols in ((4000, 65), (4000, 300), (1000, 512)):
            source = lib.ew_check(_light_program(rows, cols, flex), vec=False, want_source=True)
            assert [int(re.search(r"#define %s (\d+)" % n, source).group(1)) for n in ("V", "GROUP")] == [1, 256]


@pytest.mark.gpu
@pytest.mark.parametrize("rows,cols", [(r[1], r[2]) for r in LIGHT if not r[0]])
def test_sums(rows, cols):
    """fp32 sums of a row against float64: each of at most cols roundings of 2^-24 of the sum of magnitudes, of which those
    along one path of the tree count, at most a hundred here."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(rows)
    a, b = (torch.randn((rows, cols), device="cuda", generator=g) for _ in range(2))
    k = lib.EwKernel(_light_program(rows, cols, False))
    out = torch.full((rows,), float("nan"), device="cuda")
    scratch = torch.empty((max(k.scratch_bytes, 4),), dtype=torch.uint8, device="cuda")
    k.launch([a.data_ptr(), b.data_ptr()], [out.data_ptr()], scratch=scratch.data_ptr(), scratch_bytes=k.scratch_bytes)
    torch.cuda.synchronize()
    p = a.double() * b.double()
    assert ((out.double() - p.sum(1)).abs() <= 100 * 2.0 ** -24 * p.abs().sum(1)).all()
