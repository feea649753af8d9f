"""The FP8 GEMM with general scales at the edges of its row counts and work splits, on operands whose products and sums are
exact in fp32 (small integers, scales 3 x 2^e): the bits must equal a float64 product rounded once."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# few tiles, K blocks no multiple of four, ragged last tile; more tiles than SMs, row stride no multiple of four elements
@pytest.mark.parametrize("n,k", [(520, 1152), (19074, 640)])
@pytest.mark.parametrize("m", [1, 16, 17, 48, 64, 80, 128, 129, 176])
def test_rows_and_splits_bit_exact(wuda, m, n, k):
    g = torch.Generator().manual_seed(m + n)
    a, w = (torch.randint(-2, 3, (rows, k), generator=g) for rows in (m, n))
    ea, ew = (torch.randint(-2, 3, shape, generator=g).double() for shape in ((m, k // 128), ((n + 127) // 128, k // 128)))
    a_s, w_s = 3 * torch.exp2(ea), 3 * torch.exp2(ew)
    ref = (a.double() * a_s.repeat_interleave(128, 1)) @ (w.double() * w_s.repeat_interleave(128, 0)[:n].repeat_interleave(128, 1)).T
    args = [x.cuda() for x in (a.float().to(torch.float8_e4m3fn), a_s.float(), w.float().to(torch.float8_e4m3fn), w_s.float())]
    for _ in range(2):      # the second call finds the scratch as the first left it
        assert torch.equal(wuda.fp8_gemm(*args).cpu(), ref.float().bfloat16())
