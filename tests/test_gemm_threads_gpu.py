"""Two host threads call GEMMs that share a kernel but not its shared-memory size, each on its own stream and scratch: no call may
be refused because the other thread set the kernel up for fewer rows in between."""
import threading

import pytest
import torch

from wuda_b200._lib import lib

pytestmark = pytest.mark.gpu


def caller(kind, m, n=512, k=1024):
    """(a function that launches once and returns the status, its output, what it keeps alive)"""
    g = torch.Generator(device="cuda").manual_seed(m)
    stream = torch.cuda.Stream()
    byte = lambda *shape: torch.randint(0, 120, shape, generator=g, device="cuda", dtype=torch.uint8)
    out = torch.empty(m, n, dtype=torch.bfloat16, device="cuda")
    if kind == "nvfp4":
        pad = (m + 127) // 128 * 128
        keep = (byte(m, k // 2), byte(pad, k // 16), byte(n, k // 2), byte(n, k // 16))
        scratch = torch.zeros(lib.wuda_gemm_nvfp4_scratch_bytes(m, n), dtype=torch.uint8, device="cuda")
        args = (keep[0].data_ptr(), keep[1].data_ptr(), 1e-4, keep[2].data_ptr(), keep[3].data_ptr(), 1e-4)
        entry = lib.wuda_gemm_nvfp4
    else:
        ones = lambda *shape: torch.ones(shape, device="cuda")
        keep = (byte(m, k), ones(m, k // 128), byte(n, k), ones(n // 128, k // 128))
        scratch = torch.zeros(lib.wuda_gemm_fp8_scratch_bytes(m, n), dtype=torch.uint8, device="cuda")
        args = tuple(x.data_ptr() for x in keep)
        entry = lib.wuda_gemm_fp8_blockscaled_pow2
    tail = (out.data_ptr(), m, n, k, scratch.data_ptr(), scratch.numel(), None, stream.cuda_stream)
    return lambda: entry(*args, *tail), out, (keep, scratch, stream)


@pytest.mark.parametrize("kind", ["nvfp4", "fp8_pow2"])
def test_two_threads_with_different_row_counts(wuda, kind):
    few, many = caller(kind, 48), caller(kind, 64)
    torch.cuda.synchronize()
    assert few[0]() == 0 and many[0]() == 0
    torch.cuda.synchronize()
    want = few[1].clone(), many[1].clone()
    refused = [0, 0]

    def loop(i, call):
        torch.cuda.set_device(0)
        torch.cuda.synchronize()        # (the thread's context)
        for _ in range(20000):
            refused[i] += call() != 0

    threads = [threading.Thread(target=loop, args=(i, c[0])) for i, c in enumerate((few, many))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert refused == [0, 0]
    assert torch.equal(few[1], want[0]) and torch.equal(many[1], want[1])
