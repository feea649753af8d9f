"""The memory that the operators use beside their operands: who shares a buffer and how long it lives (host logic, no GPU)."""
import gc
import weakref

import pytest
import torch

from wuda_b200 import scratch

CPU = torch.device("cpu")


class Captures:
    """Stands in for CUDA's stream capture: which streams take part in which capture, and which stream is current."""

    def __init__(self, monkeypatch):
        self.of_stream, self.current = {}, None
        monkeypatch.setattr(scratch, "_capturing", lambda: self.current in self.of_stream)
        monkeypatch.setattr(scratch, "_capture_id", lambda stream: self.of_stream[stream])


@pytest.fixture
def captures(monkeypatch):
    return Captures(monkeypatch)


def call(kept, captures, stream, nbytes):
    captures.current = stream
    at, size, flags, buf = kept.get(CPU, stream, nbytes)
    assert at == buf.data_ptr() and size == buf.numel() >= nbytes
    return buf, flags


def test_streams_have_buffers_of_their_own(captures):
    kept = scratch.Scratch(zeroed=True)
    (a, fa), (b, fb) = call(kept, captures, 1, 5 << 20), call(kept, captures, 2, 5 << 20)
    assert a.data_ptr() != b.data_ptr() and a.numel() >= 5 << 20 and int(a.max()) == 0 and fa is fb is None
    assert call(kept, captures, 1, 1 << 20)[0] is a
    assert call(kept, captures, 1, 9 << 20)[0].numel() >= 9 << 20


def test_a_captured_call_shares_nothing_with_eager_calls_or_other_graphs(captures):
    kept = scratch.Scratch(zeroed=True)
    eager, _ = call(kept, captures, 1, 1 << 20)
    flags = []
    for capture in (7, 8):
        captures.of_stream = {1: capture, 2: capture}
        buf, first = call(kept, captures, 1, 1 << 20)
        assert buf is not eager and weakref.ref(buf)() is not None
        where = weakref.ref(buf)
        del buf
        gc.collect()
        assert where() is None                              # a temporary: the capture's pool has it back
        assert call(kept, captures, 1, 4 << 20)[1] == first     # calls of one stream of a capture follow one another
        flags += [first, call(kept, captures, 2, 1 << 20)[1]]   # its branches do not
    captures.of_stream = {}
    again, none = call(kept, captures, 1, 1 << 20)
    assert again is eager and none is None
    blocks, used = kept._flags[None]
    assert used == 4 and len(set(flags)) == 4
    for at in flags:
        assert 0 <= at - blocks[0].data_ptr() <= blocks[0].numel() - scratch.FLAG_BYTES and at % 64 == 0
    assert min(abs(a - b) for a in flags for b in flags if a != b) >= scratch.FLAG_BYTES


@pytest.mark.parametrize("eager_first", [False, True])
def test_without_flags_of_its_own_a_captured_call_clears_those_in_its_buffer(captures, monkeypatch, eager_first):
    monkeypatch.setattr(scratch, "_FLAGS_PER_BLOCK", 2)
    monkeypatch.setattr(scratch, "_MOST_BLOCKS", 1)
    kept = scratch.Scratch(zeroed=True)
    if eager_first:
        call(kept, captures, 1, 1 << 20)
    for capture in range(7, 11):
        captures.of_stream = {1: capture}
        buf, flags = call(kept, captures, 1, 1 << 20)
        assert (flags is not None) == (eager_first and capture < 9)
        assert flags is not None or int(buf[:scratch.FLAG_BYTES].max()) == 0


def test_eager_calls_lay_in_flags_and_both_are_bounded(captures, monkeypatch):
    monkeypatch.setattr(scratch, "_FLAGS_PER_BLOCK", 2)
    kept = scratch.Scratch(zeroed=True)
    buffers = []
    for i in range(100):
        captures.of_stream = {}
        buffers.append(weakref.ref(call(kept, captures, i, 1 << 10)[0]))
        captures.of_stream = {1: 1000 + i}
        call(kept, captures, 1, 1 << 10)
    gc.collect()
    assert sum(b() is not None for b in buffers) <= 16
    assert len(kept._flags[None][0]) == 4 and kept._flags[None][1] == 8 and len(kept._captures) <= 64


def test_a_scratch_that_needs_no_zeros_keeps_no_flags(captures):
    kept = scratch.Scratch(zeroed=False)
    call(kept, captures, 1, 1 << 10)
    captures.of_stream = {1: 7}
    assert call(kept, captures, 1, 1 << 10)[1] is None and not kept._flags


@pytest.mark.parametrize("kind", ["fp8", "nvfp4", "bf16"])
def test_operators_ask_the_library_for_the_size(kind):
    from wuda_b200 import ops
    name = "wuda_gemm_%s_scratch_bytes" % kind
    for m in (1, 16, 17, 128, 128, 129, 257):
        assert ops._scratch_bytes(name, m, 300) == getattr(ops.lib, name)(m, 300)
