"""The 1x128 FP8 quantisation divides by multiplying with a reciprocal and one correction: its codes must be those of a true
division, bit for bit, over the whole exponent range, at ties, for signed zeros and in groups with an infinity."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale_fmt", [None, "ue8m0"])
@pytest.mark.parametrize("kind", ["normal", "exponents", "ties", "tiny"])
def test_codes_are_those_of_a_true_division(wuda, kind, scale_fmt):
    g = torch.Generator(device="cuda").manual_seed(5)
    n = (512, 7168)
    x = torch.randn(n, generator=g, device="cuda")
    if kind == "exponents":     # any bf16 but infinities and NaN
        bits = torch.randint(-32768, 32768, n, generator=g, device="cuda", dtype=torch.int32).to(torch.int16)
        x = bits.view(torch.bfloat16).float()
        x = torch.where(torch.isfinite(x), x, -0.0)
    elif kind == "ties":        # k / 16 of powers of two: quotients by power-of-two scales fall between codes
        x = torch.randint(-480, 481, n, generator=g, device="cuda") / 16.0
    elif kind == "tiny":
        x = x * 1e-30
    x = x.bfloat16()
    x[0, :128] = -0.0
    _, q, s = wuda.rmsnorm_quant(x, None, scale_fmt=scale_fmt)
    want = (x.float().view(512, 56, 128) / s[..., None]).clamp(-448, 448).view(n).to(torch.float8_e4m3fn)
    assert torch.equal(q.view(torch.uint8), want.view(torch.uint8))


def test_a_group_with_an_infinity(wuda):
    x = torch.randn(1, 256, device="cuda").bfloat16()
    x[0, 5] = float("inf")
    _, q, s = wuda.rmsnorm_quant(x, None)
    q = q.view(torch.uint8)[0]
    assert torch.isinf(s[0, 0]) and int(q[5]) == 0xFE       # inf / inf is no number; the clamp makes -448 of it
    rest = torch.arange(128, device="cuda") != 5
    assert torch.equal(q[:128][rest], ((x[0, :128] < 0).to(torch.uint8) << 7)[rest])   # zeros of the value's sign
    assert torch.isfinite(s[0, 1])
