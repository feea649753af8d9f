"""A GEMM whose waits run out (the two-rank form with a peer that never answers, so every tile's exchange reaches its limit) must
leave its flags at zero: the scratch then serves the next call like a fresh one."""
import pytest
import torch

from wuda_b200._lib import lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [16, 64, 100])
def test_a_timed_out_call_leaves_the_scratch_clean(wuda, m):
    n, k = 25600, 256       # more tiles than SMs, two K blocks each: ranges hold whole tiles and share their last one
    g = torch.Generator(device="cuda").manual_seed(m)
    a, w = (torch.randint(-2, 3, (rows, k), generator=g, device="cuda").float().to(torch.float8_e4m3fn) for rows in (m, n))
    a_s, w_s = torch.ones(m, k // 128, device="cuda"), torch.ones(n // 128, k // 128, device="cuda")
    size = lib.wuda_gemm_fp8_scratch_bytes(m, n)
    scratch = torch.zeros(size, dtype=torch.uint8, device="cuda")
    inbox, nowhere = (torch.zeros(lib.wuda_tp2_inbox_bytes(m, n), dtype=torch.uint8, device="cuda") for _ in range(2))
    status = wuda.device_status_word()
    out = torch.empty(m, n, dtype=torch.bfloat16, device="cuda")
    operands = [x.data_ptr() for x in (a, a_s, w, w_s, out)]
    stream = torch.cuda.current_stream().cuda_stream
    assert lib.wuda_gemm_fp8_blockscaled_tp2(*operands, m, n, k, scratch.data_ptr(), size, inbox.data_ptr(), nowhere.data_ptr(), 1, 20,
                                             status.data_ptr(), stream) == 0
    torch.cuda.synchronize()
    assert int(status) == 131
    assert int(scratch[:1024].max()) == 0
    assert lib.wuda_gemm_fp8_blockscaled(*operands, m, n, k, scratch.data_ptr(), size, None, stream) == 0
    assert torch.equal(out, (a.float() @ w.float().T).bfloat16())
