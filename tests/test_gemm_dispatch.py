"""The GEMM entry points at the edges of their dispatch: products small enough for the kernel that
converts its operands on the way in (one launch; narrow, odd and unaligned operands, slices of K over
a cluster), and products for pairs of SMs (ragged row and column tiles, one k-block, slices, fp32
accumulation chains of 512 and one column more).  flex16 equals the int64 product, rescaled; fp32
against float64."""
import numpy as np
import pytest

from oracle import flex_oracle as fx

pytestmark = pytest.mark.gpu

DIRECT = [(1, 1, 1), (3, 16, 31), (127, 17, 33), (129, 33, 127), (10, 256, 64), (64, 130, 129), (300, 40, 515),
          (65, 63, 1025), (257, 7, 2049)]
PAIRS = [(4097, 4098, 32), (2049, 1200, 513), (1500, 1601, 1024), (700, 650, 6000), (500, 500, 6000), (1001, 900, 3001)]


def _operands(torch, flex, layout, M, N, K, seed, offset=0):
    rng = np.random.RandomState(seed)
    if flex:
        A = rng.randint(-32768, 32768, (M, K)).astype(np.int16)
        B = rng.randint(-32768, 32768, (K, N)).astype(np.int16)
    else:
        A = rng.standard_normal((M, K)).astype(np.float32)
        B = rng.standard_normal((K, N)).astype(np.float32)

    def put(x):
        flat = torch.zeros((x.size + offset,), dtype=torch.from_numpy(x).dtype, device="cuda")
        flat[offset:] = torch.from_numpy(np.ascontiguousarray(x).reshape(-1)).cuda()
        return flat
    dA = put(A.T if layout == "tn" else A)
    dB = put(B.T if layout == "nt" else B)
    strides = ((1, M) if layout == "tn" else (K, 1)) + ((1, K) if layout == "nt" else (N, 1))
    return A, B, dA, dB, strides


def _run(torch, flex, layout, M, N, K, offset=0):
    from ngraph_python_b200 import lib
    A, B, dA, dB, s = _operands(torch, flex, layout, M, N, K, M + 3 * N + 7 * K, offset)
    size = 2 if flex else 4
    dC = torch.zeros((M, N), dtype=torch.int16 if flex else torch.float32, device="cuda")
    nbytes = lib.gemm_scratch_bytes(flex, M, N, K)
    scratch = torch.empty((nbytes + 1024,), dtype=torch.uint8, device="cuda")
    sp = scratch.data_ptr() + (-scratch.data_ptr()) % 1024
    status = torch.zeros((1,), dtype=torch.int32, device="cuda")
    a, b = dA.data_ptr() + offset * size, dB.data_ptr() + offset * size
    if not flex:
        lib.check(lib.raw().b2_gemm_f32(a, s[0], s[1], b, s[2], s[3], dC.data_ptr(), N, M, N, K, sp,
                                        nbytes, status.data_ptr(), 0))
        torch.cuda.synchronize()
        assert int(status.item()) == 0
        expect = A.astype(np.float64) @ B.astype(np.float64)
        np.testing.assert_allclose(dC.cpu().numpy(), expect, rtol=1e-4, atol=1e-5 * np.sqrt(K) * 4)
        return
    exact = A.astype(np.int64) @ B.astype(np.int64)
    dec_c = fx.fit_dec(float(np.abs(exact).max()) * 2.0 ** -27)
    table = torch.tensor([[2.0 ** -15, 2.0 ** 15], [2.0 ** -12, 2.0 ** 12], [2.0 ** -dec_c, 2.0 ** dec_c]],
                         dtype=torch.float32, device="cuda")
    stats = torch.zeros((3,), dtype=torch.int32, device="cuda")
    probe = torch.zeros((1,), dtype=torch.int64, device="cuda")
    for flag in (1, 0):
        lib.check(lib.raw().b2_gemm_flex16(
            a, s[0], s[1], b, s[2], s[3], dC.data_ptr(), N, M, N, K, table.data_ptr(), 0, 1, 2,
            stats.data_ptr(), sp, nbytes, probe.data_ptr(), status.data_ptr(), flag, 0))
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    assert int(probe.item()) == int(np.abs(exact).max())
    sh = 27 - dec_c
    if sh > 0:
        expect = (exact + (1 << (sh - 1)) - 1 + ((exact >> sh) & 1)) >> sh
    else:
        expect = exact << -sh
    expect = np.clip(expect, -32768, 32767)
    got = dC.cpu().numpy().astype(np.int64)
    assert np.array_equal(got, expect)
    assert int(stats[2].item()) == int(np.abs(got).max())


@pytest.mark.parametrize("flex", [False, True])
@pytest.mark.parametrize("layout", ["nn", "nt", "tn"])
@pytest.mark.parametrize("M,N,K", DIRECT)
def test_small_products(M, N, K, layout, flex):
    import torch
    from ngraph_python_b200 import lib
    assert lib.gemm_launches(flex, M if layout == "tn" else 1, 1 if layout == "nt" else N, M, N, K) == 1
    _run(torch, flex, layout, M, N, K)


@pytest.mark.parametrize("flex", [False, True])
def test_operands_that_start_at_an_odd_element(flex):
    import torch
    for layout in ("nn", "nt", "tn"):
        _run(torch, flex, layout, 70, 48, 96, offset=1)


@pytest.mark.parametrize("flex", [False, True])
@pytest.mark.parametrize("M,N,K", PAIRS)
def test_products_for_pairs_of_sms(M, N, K, flex):
    import torch
    from ngraph_python_b200 import lib
    assert lib.gemm_launches(flex, 1, N, M, N, K) > 1
    _run(torch, flex, "nn", M, N, K)


SAME_BITS = {512: {(0, 1)}, 520: {(0, 2), (1, 2)}, 1024: {(0, 2)}, 1500: {(0, 3), (1, 2)},
             2048: {(0, 4), (1, 2)}, 3000: {(0, 6), (1, 2), (1, 3)}, 4096: {(0, 8), (1, 2), (1, 3), (1, 4)}}


@pytest.mark.parametrize("K", sorted(SAME_BITS))
def test_fp32_rounding_does_not_depend_on_the_kernel(K):
    """Rows and columns of a product that no slice cuts, computed again as smaller products: 1 to 8
    chains, slices of one to four of them, either operand first, narrow and wide tiles."""
    import torch
    from ngraph_python_b200 import lib
    M, N = 2304, 1152
    g = torch.Generator(device="cuda").manual_seed(K)
    A = torch.randn((M, K), device="cuda", generator=g)
    B = torch.randn((K, N), device="cuda", generator=g)
    A[3] = 0.0
    A[7, 0::2], A[7, 1::2] = B[0::2, 5], -B[1::2, 5]            # a sum that nearly vanishes
    status = torch.zeros((1,), dtype=torch.int32, device="cuda")

    def product(m, n):
        c = torch.full((m, n), 7.0, device="cuda")
        nbytes = lib.gemm_scratch_bytes(False, m, n, K)
        scratch = torch.empty((nbytes + 1024,), dtype=torch.uint8, device="cuda")
        lib.check(lib.raw().b2_gemm_f32(A.data_ptr(), K, 1, B.data_ptr(), N, 1, c.data_ptr(), n, m, n, K,
                                        scratch.data_ptr() + (-scratch.data_ptr()) % 1024, nbytes,
                                        status.data_ptr(), 0))
        torch.cuda.synchronize()
        return c
    assert lib.gemm_plan(False, 1, N, M, N, K)[:3] == (lib.GEMM_PAIRS, 128, 1)
    whole, taken = product(M, N), set()
    for m, n in ((40, 24), (24, 40), (128, 512), (512, 128), (1000, 777), (768, 512), (1024, 512), (1536, 512),
                 (2304, 64), (65, 1152)):
        kernel, _, slices, _ = lib.gemm_plan(False, 1, N, m, n, K)
        taken.add((kernel, slices))
        assert torch.equal(product(m, n).view(torch.int32), whole[:m, :n].contiguous().view(torch.int32)), (m, n)
    assert SAME_BITS[K] <= taken
    assert int(status.item()) == 0
