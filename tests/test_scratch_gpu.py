"""The operators' scratch on the GPU: graphs of small GEMMs survive larger calls, captures start clean, streams and graphs may
overlap, graphs may share a memory pool."""
import pytest
import torch

from wuda_b200 import ops, scratch

pytestmark = pytest.mark.gpu


def operands(m, n=512, k=2048, seed=0):
    """Few weight tiles, so that every tile is shared by several CTAs."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    a, w = (torch.randint(-2, 3, (rows, k), generator=g, device="cuda").bfloat16() for rows in (m, n))
    return a, w, (a.double() @ w.double().T).float()


def captured(call, pool=None):
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, pool=pool):
        out = call()
    return graph, out


def test_a_graph_survives_larger_calls_and_whatever_takes_freed_memory(wuda):
    a, w, want = operands(16)
    wuda.bf16_gemm(a, w)
    graph, out = captured(lambda: wuda.bf16_gemm(a, w, out_dtype=torch.float32))
    x8, xs = wuda.act_quant(torch.randn(256, 2048, device="cuda").bfloat16(), 128)
    w8, ws = w.float().to(torch.float8_e4m3fn), torch.ones(4, 16, device="cuda")
    for _ in range(3):
        wuda.fp8_gemm(x8, xs, w8, ws)
    junk = [torch.full((1 << 20,), 0x5A, dtype=torch.uint8, device="cuda") for _ in range(64)]
    for _ in range(3):
        out.zero_()
        graph.replay()
        assert torch.equal(out, want)
    assert all(int(j.min()) == 0x5A and int(j.max()) == 0x5A for j in junk)


def test_graphs_and_eager_calls_overlap_on_their_streams(wuda):
    """Four streams of small grids (two weight tiles, 16 to 32 CTAs each, so that all fit the GPU at once, early launches
    included): two eager ones, two graphs captured on the same stream and replayed on different ones."""
    jobs, status = [], wuda.device_status_word()
    for i, m in enumerate((16, 64, 30, 64)):
        a, w, want = operands(m, n=256, seed=i)
        out = torch.empty(m, 256, device="cuda")
        step = lambda a=a, w=w, out=out: wuda.bf16_gemm(a, w, out=out, status_word=status)
        jobs.append((torch.cuda.Stream(), step if i < 2 else captured(step)[0].replay, out, want, (a, w)))
    torch.cuda.synchronize()
    for _ in range(200):
        for stream, step, _, _, _ in jobs:
            with torch.cuda.stream(stream):
                step()
    torch.cuda.synchronize()
    assert int(status) == 0
    for _, _, out, want, _ in jobs:
        assert torch.equal(out, want)


@pytest.mark.parametrize("eager_first", [False, True])      # flags cleared in the graph, flags of the capture's own
def test_graphs_of_one_pool_take_turns(wuda, monkeypatch, eager_first):
    kept = scratch.Scratch(zeroed=True)
    monkeypatch.setattr(ops, "_gemm_scratch", kept)
    jobs, pool = [], torch.cuda.graph_pool_handle()
    for i, m in enumerate((64, 16, 120)):
        a, w, want = operands(m, seed=10 + i)
        if eager_first:
            wuda.bf16_gemm(a, w)

        def twice(a=a, w=w):
            fill = torch.full((4 << 20,), 0x77, dtype=torch.uint8, device="cuda")     # what the next graph's scratch lies on
            del fill
            return wuda.bf16_gemm(a, w, out_dtype=torch.float32), wuda.bf16_gemm(a, w, out_dtype=torch.float32)

        jobs.append((*captured(twice, pool), want, (a, w)))
    assert (kept._flags[0][1] if eager_first else len(kept._flags)) == (3 if eager_first else 0)
    for i in (0, 1, 2, 2, 0, 1, 0):
        graph, outs, want, _ = jobs[i]
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(outs[0], want) and torch.equal(outs[1], want)
    for block in kept._flags.get(0, ([], 0))[0]:
        assert int(block.max()) == 0
