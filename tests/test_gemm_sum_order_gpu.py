"""The order in which the GEMMs add a tile's partial sums is part of their results: contiguous ranges of K blocks, one per CTA,
at most max_split of them to a tile, added from the tile's start on.  The operands make every sum inside a range exact and
let the sums across ranges round: a large value in the first range, its opposite in the last one, small ones between."""
import pytest
import torch

pytestmark = pytest.mark.gpu

UNIT = {"bf16": 64, "fp8": 128, "fp8_pow2": 128}
MAX_SPLIT = {16: 16, 32: 12, 64: 8, 128: 6}


def ranges_of_tiles(n_tiles, kb, m_pad, sms):
    """For every weight tile the K-block ranges of its CTAs, in order."""
    units = n_tiles * kb
    grid = min(units, sms, n_tiles * MAX_SPLIT[m_pad])
    cuts = sorted({units * c // grid for c in range(grid + 1)} | {t * kb for t in range(n_tiles + 1)})
    tiles = [[] for _ in range(n_tiles)]
    for a, b in zip(cuts, cuts[1:]):
        tiles[a // kb].append((a % kb, a % kb + b - a))
    return tiles


# few tiles: ranges of whole tiles' thirds to sixteenths and ranges across two tiles; more tiles: the CTA with a tile's start adds
@pytest.mark.parametrize("m,n,k", [(64, 256, 7168), (64, 2624, 7168), (9, 2112, 7168), (100, 4096, 7168), (128, 520, 4096),
                                   (30, 1000, 2048), (64, 4096, 7168), (48, 7168, 2048)])
@pytest.mark.parametrize("kind", ["bf16", "fp8", "fp8_pow2"])
def test_partial_sums_are_added_in_order(wuda, kind, m, n, k):
    unit = UNIT[kind]
    n_tiles, kb = (n + 127) // 128, k // unit
    m_pad = max(16, 1 << (m - 1).bit_length())
    g = torch.Generator(device="cuda").manual_seed(m + n)
    a = torch.randint(-2, 3, (m, k), generator=g, device="cuda").double()
    w = torch.randint(-2, 3, (n_tiles * 128, k), generator=g, device="cuda").double()
    tiles = ranges_of_tiles(n_tiles, kb, m_pad, wuda.num_sms())
    # the unit of the large value: in the first range with the first K block, in the last one with the last; their ranges hold
    # nothing else, and both have the same activations and opposite weights
    a[:, -unit:] = a[:, :unit]
    exps = torch.zeros(n_tiles, kb, dtype=torch.float64, device="cuda")
    want = torch.zeros(m, n_tiles * 128, device="cuda")
    for t, parts in enumerate(tiles):
        rows = slice(t * 128, t * 128 + 128)
        if len(parts) > 1:
            w[rows, unit:parts[0][1] * unit] = 0
            w[rows, parts[-1][0] * unit:] = 0
            w[rows, -unit:] = -w[rows, :unit]
            exps[t, 0] = exps[t, -1] = 24
        scaled = w[rows] * torch.exp2(exps[t]).repeat_interleave(unit)
        total = None
        for k0, k1 in parts:
            part = a[:, k0 * unit:k1 * unit] @ scaled[:, k0 * unit:k1 * unit].T
            assert torch.equal(part.float().double(), part)
            total = part.float() if total is None else total + part.float()
        want[:, rows] = total
    want = want[:, :n]
    scale = torch.exp2(exps)
    if kind == "bf16":
        w16 = (w * scale.repeat_interleave(unit, 1).repeat_interleave(128, 0))[:n].bfloat16()
        got = wuda.bf16_gemm(a.bfloat16(), w16, out_dtype=torch.float32)
    else:
        a_s = torch.ones(m, kb, device="cuda")
        got = wuda.fp8_gemm(a.float().to(torch.float8_e4m3fn), a_s, w[:n].float().to(torch.float8_e4m3fn), scale.float().contiguous(),
                            pow2_scales=kind == "fp8_pow2").float()
        want = want.bfloat16().float()
    assert torch.equal(got, want)
