"""The native call path of the operators (csrc/fast_ops.cpp): it performs a call exactly as the Python function does or leaves it
alone.  Host logic on the CPU; on the GPU every operator's outputs with and without it, and what is refused either way."""
import pytest
import torch

import wuda_b200 as wuda
from wuda_b200 import _fast, ops

ARGUMENTS = dict(mqa_logits_fp8=10, mqa_logits_fp4=11, topk=7, rmsnorm_quant=6, act_quant=2, rope_quant=9, fp8_gemm=8, fp4_gemm=7,
                 bf16_gemm=6, nvfp4_gemm=9, sparse_mla_decode=13)


class Off:
    def __getattr__(self, name):
        return lambda *a: None


@pytest.mark.parametrize("name", sorted(ARGUMENTS))
def test_leaves_what_it_does_not_know_to_python(name):
    f, n = getattr(_fast, name), ARGUMENTS[name]
    with pytest.raises(TypeError):
        f(*[None] * (n + 1))
    host = torch.zeros(2, 256)
    for value in (None, 3, "x", host, host.bfloat16(), torch.zeros(2, 3, 512).bfloat16()):
        assert f(*[value] * n) is None
    with pytest.raises((RuntimeError, TypeError, AttributeError)):      # and the Python function says why
        wuda.rmsnorm_quant(host, None)


PYTHON = {"act_quant of a column slice", "fp8 exponent bytes", "fp4 exponent bytes"}      # cases of _cases() that the native path leaves to Python


class Recorder:
    """The native path, and what it did with each call: (operator, whether it took the call)."""

    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        f = getattr(_fast, name)

        def call(*args):
            done = f(*args)
            self.calls.append((name, done is not None))
            return done
        return call


def _cases():
    g = torch.Generator(device="cuda").manual_seed(7)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    e4 = lambda *s: rnd(*s).to(torch.float8_e4m3fn)
    i32 = lambda *s, hi=8: torch.randint(0, hi, s, generator=g, device="cuda", dtype=torch.int32)
    x = rnd(5, 1024).bfloat16()
    heads, pos, cos, sin = rnd(5, 16, 192).bfloat16(), torch.arange(5, device="cuda"), rnd(9, 32), rnd(9, 32)
    a, a_s = wuda.act_quant(x, 128, "ue8m0")
    w, w_s = e4(384, 1024), torch.exp2(torch.randint(-4, 1, (3, 8), generator=g, device="cuda").float())
    w4, w4_s = wuda.fp4_act_quant(rnd(256, 1024).bfloat16())
    status = wuda.device_status_word()
    yield "rmsnorm", lambda: wuda.rmsnorm_quant(x, rnd(1024).fill_(1.5))
    yield "rmsnorm bf16 weights", lambda: wuda.rmsnorm_quant(x, rnd(1024).fill_(1.5).bfloat16())
    yield "rmsnorm rows of a wider matrix", lambda: wuda.rmsnorm_quant(x[:, :512], None, scale_fmt="ue8m0")
    yield "rmsnorm without quantisation", lambda: wuda.rmsnorm_quant(x, None, quant=False)
    yield "rmsnorm quantisation alone", lambda: wuda.rmsnorm_quant(x, None, 1e-5, return_bf16=False)
    yield "no rows", lambda: wuda.rmsnorm_quant(x[:0], None)
    yield "act_quant", lambda: wuda.act_quant(x.view(5, 1, 1024))
    yield "act_quant of a column slice", lambda: wuda.act_quant(x[:, 512:], 128, "ue8m0")
    yield "rope", lambda: wuda.rope_quant(heads, pos, cos, sin, 64, inverse=True, return_bf16=True)
    yield "rope rows of one", lambda: wuda.rope_quant(heads[:1], pos[:1], cos, sin, 64, quant=False, return_bf16=True, scale_fmt="ue8m0")
    for pow2 in (False, True):
        yield f"fp8 {pow2}", lambda pow2=pow2: wuda.fp8_gemm(a.view(1, 5, 1024), a_s.view(1, 5, 8), w, w_s, pow2_scales=pow2)
    yield "fp8 given output", lambda: wuda.fp8_gemm(a, a_s, w, w_s, out=torch.empty(5, 384, device="cuda", dtype=torch.bfloat16), status_word=status)
    yield "fp4 given output", lambda: wuda.fp4_gemm(a, a_s, w4, w4_s, out=torch.empty(5, 256, device="cuda", dtype=torch.bfloat16))
    yield "bf16 given output", lambda: wuda.bf16_gemm(x, rnd(64, 1024).fill_(0.5).bfloat16(), out=torch.empty(5, 64, device="cuda"), status_word=status)
    yield "fp8 exponent bytes", lambda: wuda.fp8_gemm(a, a_s.to(torch.float8_e8m0fnu), w, w_s.to(torch.float8_e8m0fnu))
    yield "fp4 exponent bytes", lambda: wuda.fp4_gemm(a, a_s.to(torch.float8_e8m0fnu), w4, w4_s)
    yield "fp8 parameter", lambda: wuda.fp8_gemm(a, a_s, torch.nn.Parameter(w, requires_grad=False), w_s)
    yield "fp4", lambda: wuda.fp4_gemm(a, a_s, w4, w4_s)
    yield "bf16", lambda: wuda.bf16_gemm(x, rnd(64, 1024).fill_(0.5).bfloat16())
    yield "bf16 fp32", lambda: wuda.bf16_gemm(x, rnd(64, 1024).fill_(0.5).bfloat16(), out_dtype=torch.float32)
    codes, sf = i32(5, 512, hi=256).byte(), i32(128 * 64, hi=0x38).byte()
    wcodes, wsf = i32(256, 512, hi=256).byte(), i32(256 * 64, hi=0x38).byte()
    yield "nvfp4", lambda: wuda.nvfp4_gemm(codes, sf, 0.5, wcodes, wsf, 2)
    yield "nvfp4 given output", lambda: wuda.nvfp4_gemm(codes, sf, 0.5, wcodes, wsf, 2, out=torch.empty(5, 256, device="cuda", dtype=torch.bfloat16),
                                                        status_word=status)
    pages, table, lens = i32(8, 64 * 132, hi=100).byte(), i32(3, 4), torch.tensor([200, 0, 77], dtype=torch.int32, device="cuda")
    wts, q = rnd(3, 64), e4(3, 64, 128)
    yield "logits fp8", lambda: wuda.mqa_logits_fp8_decode_out(q, pages, wts, lens, table, None, torch.zeros(3, 256, device="cuda"), 64)
    q2, lens2 = e4(6, 64, 128), torch.tensor([199, 200, 0, 0, 76, 77], dtype=torch.int32, device="cuda")
    yield "logits fp8 two rows a request", lambda: wuda.mqa_logits_fp8_decode_out(q2, pages, rnd(6, 64).fill_(0.25), lens2, table, None,
                                                                                  torch.zeros(6, 256, device="cuda"), 64, 64 * 132, next_n=2)
    q4, q4_sf, pages4 = i32(3, 64, 64, hi=256).byte(), i32(3, 64, hi=0x70), i32(8, 64 * 68, hi=0x70).byte()
    yield "logits fp4", lambda: wuda.mqa_logits_fp4_decode_out(q4, q4_sf, pages4, wts, lens, table, torch.zeros(3, 256, device="cuda"))
    yield "logits fp4 longest context given", lambda: wuda.mqa_logits_fp4_decode_out(q4, q4_sf, pages4, wts, lens, table, torch.zeros(3, 300, device="cuda"),
                                                                                     200, 64, 64 * 68, status_word=status)
    scores = rnd(3, 256)
    raw = torch.empty(3, 64, dtype=torch.int32, device="cuda")
    yield "topk", lambda: (wuda.topk_v2(scores, lens, table, 64, raw_indices=raw), raw.clone())
    scores2 = rnd(6, 256)
    yield "topk two rows a table row", lambda: wuda.topk_v2(scores2, lens2, table, 64, rows_per_table_row=2)
    from test_sparse_mla_gpu import model1_pool, view4
    import numpy as np
    pool = view4(model1_pool(np.random.default_rng(3), 6, 64), 64)
    qa, idx, n = rnd(2, 64, 512).bfloat16(), i32(2, 512, hi=6 * 64), torch.tensor([300, 512], dtype=torch.int32, device="cuda")
    for split in (False, True):
        yield f"attention {split}", lambda split=split: wuda.sparse_mla_decode(qa, pool, idx[:, :128].contiguous(), n.clamp_max(128), pool, idx, n,
                                                                               rnd(64).fill_(0.1), 0.04, split=split)
    yield "attention given output", lambda: wuda.sparse_mla_decode(qa, pool, idx, n, out=torch.empty_like(qa))
    yield "attention one pool", lambda: wuda.sparse_mla_decode(qa, None, None, None, pool, idx, n, status_word=status)


def _refused():
    x = torch.zeros(4, 256, device="cuda").bfloat16()
    a, a_s = wuda.act_quant(x)
    w, w_s = torch.zeros(128, 256, device="cuda").to(torch.float8_e4m3fn), torch.ones(1, 2, device="cuda")
    yield lambda: wuda.rmsnorm_quant(x.float(), None)
    yield lambda: wuda.rmsnorm_quant(x[:, ::2], None)
    yield lambda: wuda.rmsnorm_quant(x, torch.ones(255, device="cuda"))
    yield lambda: wuda.rmsnorm_quant(x[:, 4:132], None)                                   # rows not 16-byte aligned
    yield lambda: wuda.rmsnorm_quant(x, None, quant=False, return_bf16=False)
    yield lambda: wuda.act_quant(x, 64)
    yield lambda: wuda.rope_quant(x.view(4, 2, 128), torch.zeros(3, dtype=torch.long, device="cuda"), a_s, a_s, 64)
    yield lambda: wuda.fp8_gemm(a, a_s, w[:, :128], w_s)
    yield lambda: wuda.fp8_gemm(a, a_s[:2], w, w_s)
    yield lambda: wuda.fp8_gemm(a.repeat(65, 1), a_s.repeat(65, 1), w, w_s)               # 260 rows
    yield lambda: wuda.bf16_gemm(x, x[:, :128])
    yield lambda: wuda.topk_v2(torch.zeros(2, 8, device="cuda"), torch.zeros(3, dtype=torch.int32, device="cuda"), torch.zeros(2, 1, dtype=torch.int32, device="cuda"), 4)


@pytest.mark.gpu
def test_every_operator_with_and_without(wuda, monkeypatch):
    def run(recorder=None):
        out = []
        for name, f in _cases():
            if recorder:
                recorder.calls.clear()
            r = f()
            out += [(name, t) for t in (r if isinstance(r, tuple) else (r,))]
            if recorder:                    # (a case that falls through to another operator's Python function makes two calls)
                assert recorder.calls and recorder.calls[0][1] == (name not in PYTHON), (name, recorder.calls)
                taken.update(op for op, done in recorder.calls if done)
        torch.cuda.synchronize()
        return out
    run()                                   # every scratch has its size
    taken, recorder = set(), Recorder()
    monkeypatch.setattr(ops, "_fast", recorder)
    fast = run(recorder)
    assert taken == set(ARGUMENTS)
    monkeypatch.setattr(ops, "_fast", Off())
    for (name, a), (_, b) in zip(fast, run(), strict=True):
        assert (a is None) == (b is None), name
        if a is not None:
            assert (a.shape, a.stride(), a.dtype, a.device, a.requires_grad) == (b.shape, b.stride(), b.dtype, b.device, b.requires_grad), name
            assert torch.equal(a.contiguous().view(torch.uint8), b.contiguous().view(torch.uint8)), name


@pytest.mark.gpu
def test_refusals_are_the_same(wuda, monkeypatch):
    said = []
    for off in (False, True):
        if off:
            monkeypatch.setattr(ops, "_fast", Off())
        said.append([])
        for f in _refused():
            with pytest.raises(Exception) as e:
                f()
            said[-1].append((type(e.value), str(e.value)))
    assert said[0] == said[1]


@pytest.mark.gpu
def test_modes_and_capture_go_through_python(wuda):
    from torch.utils._python_dispatch import TorchDispatchMode
    seen = []

    class Watch(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))
    x = torch.ones(2, 256, device="cuda").bfloat16()
    with Watch():
        wuda.rmsnorm_quant(x, None)
    assert sum("new_empty" in s for s in seen) == 3
    with torch.inference_mode():
        assert wuda.rmsnorm_quant(x, None)[0].is_inference()
    a, a_s = wuda.act_quant(x)
    w, w_s = torch.ones(128, 256, device="cuda").to(torch.float8_e4m3fn), torch.ones(1, 2, device="cuda")
    eager = wuda.fp8_gemm(a, a_s, w, w_s)
    graph = torch.cuda.CUDAGraph()
    before = set(ops._gemm_scratch._captures)
    with torch.cuda.graph(graph):
        out = wuda.fp8_gemm(a, a_s, w, w_s)
    assert set(ops._gemm_scratch._captures) - before            # a scratch and flags of the capture's own
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, eager)


@pytest.mark.gpu
def test_threads_and_streams_on_the_native_path(wuda, monkeypatch):
    """Threads that share a stream or have their own look scratches up at once, with a scratch that grows and one that is dropped meanwhile."""
    import threading
    from test_gemm_tc_gpu import operands
    work = []
    for m, n, k in ((3, 2112, 2048), (9, 384, 1024), (40, 4096, 2048), (120, 640, 1024)):
        args, ref = operands("fp8", m, n, k, seed=m)
        work.append(([x.cuda() for x in args], ref.float().bfloat16().cuda()))
    recorder = Recorder()
    monkeypatch.setattr(ops, "_fast", recorder)
    streams = [torch.cuda.Stream() for _ in range(3)]
    torch.cuda.synchronize()
    wrong, failed = [], []

    def run(i):
        try:
            with torch.cuda.stream(streams[i // 2]):
                for step in range(150):
                    args, want = work[(step + i) % 4]
                    for pow2 in (False, True):
                        if not torch.equal(wuda.fp8_gemm(*args, pow2_scales=pow2), want):
                            wrong.append((i, step, pow2))
                    if i == 0 and step % 50 == 25:      # the next call of this stream goes through Python and makes one anew
                        ops._gemm_scratch._streams.pop((0, streams[0].cuda_stream), None)
        except Exception as e:
            failed.append(e)
    threads = [threading.Thread(target=run, args=(i,)) for i in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not failed and not wrong
    assert sum(done for _, done in recorder.calls) > 1700        # of 1800
