"""The GEMM that accumulates in tensor memory, at the edges of its row counts and of its two work splits, on operands whose
products and sums are exact in fp32: every kind's bits must equal a float64 product rounded once."""
import numpy as np
import pytest
import torch

from wuda_b200 import workloads
from wuda_b200._lib import lib

pytestmark = pytest.mark.gpu

CODES = torch.tensor([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0])
KINDS = ("bf16", "fp8", "fp8_fp4", "nvfp4")


def fp4(codes):
    mag = CODES[(codes & 7).long()].double()
    return torch.where(codes & 8 > 0, -mag, mag)


def pack(codes):
    return (codes[:, 0::2] | codes[:, 1::2] << 4).contiguous()


def operands(kind, m, n, k, seed):
    """(arguments on the GPU, float64 product): small integers times powers of two between 2^-2 and 2^2."""
    g = torch.Generator().manual_seed(seed)
    ints = lambda rows: torch.randint(-2, 3, (rows, k), generator=g)
    exps = lambda rows, cols: torch.randint(-2, 3, (rows, cols), generator=g)
    nibbles = lambda rows: (torch.randint(0, 5, (rows, k), generator=g) | torch.randint(0, 2, (rows, k), generator=g) << 3).to(torch.uint8)
    if kind == "bf16":
        a, w = ints(m), ints(n)
        return (a.bfloat16(), w.bfloat16()), a.double() @ w.double().T
    if kind in ("fp8", "fp8_fp4"):
        a, ea = ints(m), exps(m, k // 128)
        av = a.double() * torch.exp2(ea.double()).repeat_interleave(128, 1)
        a8, a_s = a.float().to(torch.float8_e4m3fn), torch.exp2(ea.float())
        if kind == "fp8":
            w, ew = ints(n), exps((n + 127) // 128, k // 128)
            wv = w.double() * torch.exp2(ew.double()).repeat_interleave(128, 0)[:n].repeat_interleave(128, 1)
            return (a8, a_s, w.float().to(torch.float8_e4m3fn), torch.exp2(ew.float())), av @ wv.T
        c, ew = nibbles(n), exps(n, k // 32)
        wv = fp4(c) * torch.exp2(ew.double()).repeat_interleave(32, 1)
        return (a8, a_s, pack(c).view(torch.float4_e2m1fn_x2), (ew + 127).to(torch.uint8)), av @ wv.T
    ca, cw, ea, ew = nibbles(m), nibbles(n), exps(m, k // 16), exps(n, k // 16)
    value = lambda c, e: fp4(c) * torch.exp2(e.double()).repeat_interleave(16, 1)
    sf = lambda e: torch.from_numpy(np.ascontiguousarray(workloads.pack_nvfp4_scales((0x38 + 8 * e).to(torch.uint8).numpy())))
    return (pack(ca), sf(ea), 1.0, pack(cw), sf(ew), 1.0), value(ca, ea) @ value(cw, ew).T


def call(wuda, kind, args):
    args = [x.cuda() if torch.is_tensor(x) else x for x in args]
    if kind == "bf16":
        return wuda.bf16_gemm(*args)
    if kind == "fp8":
        return wuda.fp8_gemm(*args, pow2_scales=True)
    return wuda.fp4_gemm(*args) if kind == "fp8_fp4" else wuda.nvfp4_gemm(*args)


# few tiles: split evenly, ragged last tile; more tiles than SMs: stream-K, row stride no multiple of four elements
@pytest.mark.parametrize("n,k", [(520, 1280), (19074, 512)])
@pytest.mark.parametrize("m", [1, 16, 17, 48, 80, 112, 128, 129, 176, 256])
@pytest.mark.parametrize("kind", KINDS)
def test_rows_and_splits_bit_exact(wuda, kind, m, n, k):
    if kind == "bf16" and m > 128:
        pytest.skip("BF16 takes at most 128 rows")
    args, ref = operands(kind, m, n, k, seed=m + n)
    for _ in range(2):      # the second call finds the scratch as the first left it
        got = call(wuda, kind, args)
        assert torch.equal(got.cpu(), ref.float().bfloat16())


@pytest.mark.parametrize("kind", ("fp8", "fp8_fp4", "nvfp4"))
def test_a_scratch_for_128_rows_takes_more_rows_in_passes(wuda, kind):
    m, n, k = 200, 1000, 1024
    args, ref = operands(kind, m, n, k, seed=5)
    args = [x.cuda() if torch.is_tensor(x) else x for x in args]
    size = (lib.wuda_gemm_nvfp4_scratch_bytes if kind == "nvfp4" else lib.wuda_gemm_fp8_scratch_bytes)(128, n)
    scratch = torch.zeros(size, dtype=torch.uint8, device="cuda")
    out = torch.empty(m, n, dtype=torch.bfloat16, device="cuda")
    entry = dict(fp8=lib.wuda_gemm_fp8_blockscaled_pow2, fp8_fp4=lib.wuda_gemm_fp8_fp4_pow2, nvfp4=lib.wuda_gemm_nvfp4)[kind]
    raw = [x.data_ptr() if torch.is_tensor(x) else x for x in args]
    assert entry(*raw, out.data_ptr(), m, n, k, scratch.data_ptr(), size, None, torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    assert torch.equal(out.cpu(), ref.float().bfloat16())
    assert int(scratch[:1024].max()) == 0
