"""The kernels between the routed experts' GEMMs at the sizes where their work split changes: dispatch around its rounds of 1024
pairs, gather + NVFP4 quantisation around one walk over the batch.  Whole numbers and bytes, so equality with the oracle."""
import numpy as np
import pytest
import torch

import oracle
from wuda_b200._lib import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,k,experts,first,total", [(1, 1, 1, 0, 1), (31, 33, 40, 0, 40), (128, 8, 256, 0, 256),
                                                          (1025, 1, 3, 0, 3), (341, 6, 512, 0, 512), (700, 7, 100, 30, 160)])
def test_dispatch_ranks_over_warps_and_rounds(wuda, tokens, k, experts, first, total):
    rng = np.random.default_rng(tokens + k)
    idx = rng.integers(0, total, (tokens, k)).astype(np.int32)
    idx[rng.random((tokens, k)) < 0.4] = first            # one expert in many warps and rounds
    w = rng.random((tokens, k)).astype(np.float32)
    most = wuda.lib.wuda_moe_max_groups(tokens, k, experts)
    d_idx, d_w = torch.from_numpy(idx).cuda(), torch.from_numpy(w).cuda()
    i32 = lambda *s: torch.full(s, 77, dtype=torch.int32, device="cuda")
    group_expert, groups, row_token, pair_row = i32(most), i32(1), i32(most * 16), i32(tokens, k)
    row_weight, status = torch.full((most * 16,), 7.0, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    check(wuda.lib.wuda_moe_dispatch_range(d_idx.data_ptr(), d_w.data_ptr(), group_expert.data_ptr(), groups.data_ptr(),
                                           row_token.data_ptr(), row_weight.data_ptr(), pair_row.data_ptr(), tokens, k, experts,
                                           first, total, most, status.data_ptr(), None))
    torch.cuda.synchronize()
    ge, rt, pr = oracle.moe_dispatch(np.where((idx >= first) & (idx < first + experts), idx - first, -1), experts)
    n = len(ge)
    assert int(status.item()) == 0 and int(groups.item()) == n
    assert np.array_equal(group_expert.cpu().numpy(), np.concatenate([ge, np.full(most - n, -1)]))
    assert np.array_equal(pair_row.cpu().numpy(), pr)
    assert np.array_equal(row_token.cpu().numpy(), np.concatenate([rt, np.full((most - n) * 16, -1)]))
    want = np.zeros(most * 16, np.float32)
    want[pr[pr >= 0]] = w[pr >= 0]
    assert np.array_equal(row_weight.cpu().numpy(), want)


@pytest.mark.parametrize("tokens,topk,k,gs,values", [(1, 1, 256, 1.0 / 448, "normal"), (3, 5, 768, 0.25, "ties"),
                                                     (64, 8, 7168, 1.0 / 448, "normal"), (43, 8, 7168, 1e-3, "exponents"),
                                                     (7, 3, 512, 1e-25, "exponents"), (5, 2, 512, 3e20, "exponents")])
def test_gather_and_nvfp4_codes(wuda, tokens, topk, k, gs, values):
    rng = np.random.default_rng(tokens * topk)
    if values == "normal":
        x = rng.standard_normal((tokens, k)).astype(np.float32)
    elif values == "ties":      # multiples of 1/16 of the tensor scale under an amax of 6: quotients on every midpoint
        x = (rng.integers(-96, 97, (tokens, k)) / 16.0 * gs).astype(np.float32)
        x[:, ::16] = 6 * gs
    else:                       # any finite bf16 that does not overflow the oracle's own products
        bits = rng.integers(0, 1 << 16, (tokens, k)).astype(np.uint16)
        x = oracle.bf16_to_f32(bits)
        x = np.where(np.isfinite(x), x, np.float32(0))
    x16 = oracle.f32_to_bf16(x)
    x = oracle.bf16_to_f32(x16)
    pairs = tokens * topk
    rows = rng.permutation((pairs + 15) // 16 * 16 + 16)[:pairs].astype(np.int32)
    rows[rng.random(pairs) < 0.1] = -1
    n = (pairs + 15) // 16 * 16 + 16
    a4 = torch.full((n, k // 2), 0x5a, dtype=torch.uint8, device="cuda")
    sf = torch.zeros(n // 16 * (k // 256) * 2048, dtype=torch.uint8, device="cuda")
    d_x, d_rows = torch.from_numpy(x16.view(np.int16).copy()).cuda(), torch.from_numpy(rows).cuda()
    check(wuda.lib.wuda_moe_gather_quant_nvfp4(d_x.data_ptr(), d_rows.data_ptr(), a4.data_ptr(), sf.data_ptr(), gs, tokens, topk, k,
                                               None))
    torch.cuda.synchronize()
    live = rows >= 0
    q, s = oracle.quantize_nvfp4_rows(x[np.arange(pairs) // topk][live], gs)
    got = a4.cpu().numpy()
    assert np.array_equal(got[rows[live]], q)
    untouched = np.ones(n, bool)
    untouched[rows[live]] = False
    assert np.all(got[untouched] == 0x5a)
    image = sf.cpu().numpy().reshape(n // 16, k // 256, 4, 32, 16)[:, :, :, :16, :4]     # [group, kb, step, row, byte]
    image = image.reshape(n // 16, k // 256, 4, 16, 4).transpose(0, 3, 1, 2, 4).reshape(n, k // 16)
    assert np.array_equal(image[rows[live]], s)


# CTAs of 128 threads and of 768, either side of the line between them, more tokens than one walk takes, more rows than one look-up
@pytest.mark.parametrize("tokens,topk,k", [(26, 4, 7168), (27, 9, 7168), (160, 2, 7168), (46, 1, 4096), (170, 13, 7168)])
def test_gather_stores_a_token_to_all_its_rows(wuda, tokens, topk, k):
    test_gather_and_nvfp4_codes(wuda, tokens, topk, k, 1.0 / 448, "normal")


# the lines between the grids of a call by itself (at 148 SMs): CTAs of 128 threads and of 768, of 768 and of 256, one walk and more
@pytest.mark.parametrize("tokens,topk,k", [(84, 2, 7168), (85, 2, 7168), (253, 1, 7168), (254, 2, 7168), (680, 1, 7168)])
def test_gather_grids(wuda, tokens, topk, k):
    test_gather_and_nvfp4_codes(wuda, tokens, topk, k, 1.0 / 448, "normal")


def test_gather_of_as_many_blocks_as_it_takes(wuda):
    """2^31 - 32768 blocks of 16 values, 69 GB: the walk's last steps lie beyond 2^31.  The last token's row is that of a call by itself."""
    tokens, k = 65535, 1 << 19
    if torch.cuda.mem_get_info()[0] < 80 << 30:
        pytest.skip("needs 80 GB")
    x = torch.empty(tokens, k, dtype=torch.bfloat16, device="cuda")
    x[-1] = torch.randn(k, device="cuda")
    rows = torch.full((tokens, 1), -1, dtype=torch.int32, device="cuda")
    rows[-1] = 0
    got = []
    for t in (tokens, 1):
        a4, sf = (torch.full((n,), 0x5a, dtype=torch.uint8, device="cuda") for n in (16 * k // 2, k // 256 * 2048))
        check(wuda.lib.wuda_moe_gather_quant_nvfp4(x[-t:].data_ptr(), rows[-t:].data_ptr(), a4.data_ptr(), sf.data_ptr(), 1.0 / 448, t, 1, k,
                                                   torch.cuda.current_stream().cuda_stream))
        got.append((a4, sf))
    torch.cuda.synchronize()
    del x
    torch.cuda.empty_cache()
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    assert bool((got[0][0][:k // 2] != 0x5a).any()) and bool((got[0][0][k // 2:] == 0x5a).all())
