"""GEMMs of few rows and few weight tiles: the CTA that arrives last at a tile adds all its partial sums.  Around the row counts
where that begins and ends (8 rows, for general FP8 scales 16), with CTAs that hold parts of one and of two tiles: exact bits, the
order of the additions, and call after call on one scratch."""
import pytest
import torch

from test_gemm_sum_order_gpu import test_partial_sums_are_added_in_order as check_order
from test_gemm_tc_gpu import KINDS, call, operands

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(256, 7168), (2112, 4096), (4096, 2048)])
@pytest.mark.parametrize("m", [1, 3, 5, 8, 9, 13, 16])
@pytest.mark.parametrize("kind", KINDS)
def test_exact_bits(wuda, kind, m, n, k):
    args, ref = operands(kind, m, n, k, seed=m + n)
    args = [x.cuda() if torch.is_tensor(x) else x for x in args]
    want = ref.float().bfloat16()
    for _ in range(20):
        got = call(wuda, kind, args)
    assert torch.equal(got.cpu(), want)


@pytest.mark.parametrize("m,n,k", [(1, 256, 7168), (4, 2112, 7168), (8, 2624, 7168), (16, 2112, 7168), (13, 4096, 7168), (5, 520, 4096)])
@pytest.mark.parametrize("kind", ["bf16", "fp8", "fp8_pow2"])
def test_order(wuda, kind, m, n, k):
    check_order(wuda, kind, m, n, k)


@pytest.mark.parametrize("m,n,k", [(8, 1152, 7168), (8, 1280, 7168), (16, 1152, 7168), (16, 1280, 7168), (16, 1408, 7168), (16, 1536, 7168),
                                   (16, 2048, 4864), (16, 2048, 4608)])
@pytest.mark.parametrize("kind", KINDS)
def test_two_quads_per_thread(wuda, kind, m, n, k):
    """Either side of whole ranges (9 and 10 weight tiles on 148 SMs); general FP8 scales also of 13 ranges per tile and of four units per range."""
    test_exact_bits(wuda, kind, m, n, k)
    if kind == "fp8":
        args, ref = operands(kind, m, n, k, seed=m + n)
        args = [x.cuda() for x in args]
        for _ in range(20):
            got = wuda.fp8_gemm(*args)
        assert torch.equal(got.cpu(), ref.float().bfloat16())
