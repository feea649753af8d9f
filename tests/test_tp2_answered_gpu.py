"""The exchange of the two-rank GEMM against a peer that has already answered: its tiles and flags are in this rank's inbox before
the launch, so one GPU is enough and nothing waits.  What this rank sends must be its own fp32 sums, flagged; what it returns,
the sum of both."""
import pytest
import torch

from wuda_b200._lib import lib

pytestmark = pytest.mark.gpu
FLAG_BYTES, CTRL_BYTES = 4096, 64


# ranges that share tiles, few tiles (each still finished by one CTA), more tiles than SMs with a ragged last one
@pytest.mark.parametrize("n,k", [(7168, 2048), (520, 1152), (19080, 640)])
@pytest.mark.parametrize("m", [1, 16, 30, 64, 100])
@pytest.mark.parametrize("device_sequence", [False, True])
def test_sums_with_an_answer_that_is_there(wuda, m, n, k, device_sequence):
    g = torch.Generator(device="cuda").manual_seed(m + n)
    a, w = (torch.randint(-2, 3, (rows, k), generator=g, device="cuda").float().to(torch.float8_e4m3fn) for rows in (m, n))
    n_tiles, m_pad = (n + 127) // 128, max(16, 1 << (m - 1).bit_length())
    a_s = torch.exp2(torch.randint(-2, 3, (m, k // 128), generator=g, device="cuda").float())
    w_s = 3 * torch.exp2(torch.randint(-2, 3, (n_tiles, k // 128), generator=g, device="cuda").float())
    own = (a.double() * a_s.double().repeat_interleave(128, 1)) @ (
        w.double() * w_s.double().repeat_interleave(128, 0)[:n].repeat_interleave(128, 1)).T
    peer = torch.randn(m_pad, n_tiles * 128, generator=g, device="cuda") * 100
    size = lib.wuda_tp2_inbox_bytes(m, n)
    inbox, sent = (torch.zeros(size, dtype=torch.uint8, device="cuda") for _ in range(2))
    flags = lambda box: box[:FLAG_BYTES].view(torch.int32)[:2 * n_tiles].view(2, n_tiles)
    tiles = lambda box: box[FLAG_BYTES:].view(torch.float32).view(2, n_tiles, m_pad, 128)
    scratch_bytes = lib.wuda_gemm_fp8_scratch_bytes(m, n)
    scratch = torch.zeros(scratch_bytes, dtype=torch.uint8, device="cuda")
    status = wuda.device_status_word()
    for call in (1, 2, 3):
        flags(inbox)[call & 1] = call
        tiles(inbox)[call & 1] = peer.view(m_pad, n_tiles, 128).transpose(0, 1) * call
        out = torch.full((m, n), float("nan"), dtype=torch.bfloat16, device="cuda")
        assert lib.wuda_gemm_fp8_blockscaled_tp2(a.data_ptr(), a_s.data_ptr(), w.data_ptr(), w_s.data_ptr(), out.data_ptr(), m, n, k,
                                                 scratch.data_ptr(), scratch_bytes, inbox.data_ptr(), sent.data_ptr(),
                                                 0 if device_sequence else call, 1000, status.data_ptr(),
                                                 torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        assert int(status) == 0
        assert torch.equal(flags(sent)[call & 1], torch.full((n_tiles,), call, dtype=torch.int32, device="cuda"))
        mine = tiles(sent)[call & 1].transpose(0, 1).reshape(m_pad, n_tiles * 128)[:m, :n]
        assert torch.equal(mine.double(), own)
        assert torch.equal(out, (own.float() + peer[:m, :n] * call).bfloat16())
        assert int(scratch[:1024].max()) == 0
    if device_sequence:
        assert inbox[FLAG_BYTES - CTRL_BYTES:FLAG_BYTES].view(torch.int32)[:2].tolist() == [3, 0]
