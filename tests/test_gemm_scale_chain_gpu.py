"""Weights quantised and multiplied in one chain of programmatic launches: the GEMM is resident while the quantiser still writes
the scales, so every replay must see this replay's scales and none of the last one's."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def quantise(wuda, kind, w, scales_from):
    """(weights, their scales), both written by kernels of the library."""
    if kind == "fp8_fp4":
        return wuda.fp4_act_quant(w, 32)
    fmt = "ue8m0" if kind == "fp8_pow2" else None
    w8, _ = wuda.act_quant(w, 128, fmt)
    return w8, wuda.act_quant(scales_from, 128, fmt)[1]      # one scale per 128 columns of ceil(N / 128) rows


def multiply(wuda, kind, a, a_s, w, w_s):
    if kind == "fp8_fp4":
        return wuda.fp4_gemm(a, a_s, w, w_s)
    return wuda.fp8_gemm(a, a_s, w, w_s, pow2_scales=kind == "fp8_pow2")


@pytest.mark.parametrize("k", [1024, 1152])       # scales in 16-byte loads, and one by one
@pytest.mark.parametrize("kind", ["fp8", "fp8_pow2", "fp8_fp4"])
def test_replays_see_the_scales_of_their_own_quantisation(wuda, kind, k):
    n, m = 2048, 32
    g = torch.Generator(device="cuda").manual_seed(k)
    x = torch.randn(m, k, generator=g, device="cuda").bfloat16()
    a, a_s = wuda.act_quant(x, 128, "ue8m0")
    w = torch.randn(n, k, generator=g, device="cuda").bfloat16()
    src = torch.randn(n // 128, k, generator=g, device="cuda").bfloat16()
    multiply(wuda, kind, a, a_s, *quantise(wuda, kind, w, src))
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = multiply(wuda, kind, a, a_s, *quantise(wuda, kind, w, src))
    for i in range(12):
        w.copy_(torch.randn(n, k, generator=g, device="cuda") * 2.0 ** (i % 7 - 3))
        src.copy_(torch.randn(n // 128, k, generator=g, device="cuda") * 2.0 ** (3 - i % 7))
        graph.replay()
        torch.cuda.synchronize()
        operands = quantise(wuda, kind, w, src)
        torch.cuda.synchronize()                  # nothing overlaps here
        assert torch.equal(out, multiply(wuda, kind, a, a_s, *operands))
