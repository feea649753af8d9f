"""Device memory that the operators called directly use beside their operands: the GEMMs' scratch, the attention's partial sums.

Eager calls: one buffer per stream.  Calls that may overlap on the GPU never share one (the kernels that work in it forbid
that), and calls on one stream are ordered, so a buffer that became too small can be dropped: it was allocated on the stream
that used it.

Calls under stream capture: a temporary of the capture, so that the graph's own memory pool keeps it and nothing of it is shared
with another graph or with eager calls.  What the GEMMs want as zeros and leave as zeros (FLAG_BYTES at the front) must outlive a
replay, though, and a temporary does not; a captured memset in front of every GEMM would do (and is the last resort), but costs
2 us and the early launch.  So the flags of a capture are FLAG_BYTES of their own, per captured stream, from a block that was
zeroed before; they are never used for anything else again.
"""
import ctypes
import threading

import torch

from ._lib import check, lib

FLAG_BYTES = 1024
_SMALLEST = 1 << 20
_MOST_STREAMS = 16          # streams beyond that take turns (25 MB each at most)
_FLAGS_PER_BLOCK = 1024     # captures that one block of flags serves
_MOST_BLOCKS = 4            # captures beyond that take the memset
_CAPTURES_AT_ONCE = 64      # a capture that is forgotten while it is under way takes new flags

_lock = threading.Lock()


_capturing = torch._C._cuda_isCurrentStreamCapturing


def _capture_id(stream):
    got = ctypes.c_ulonglong()
    check(lib.wuda_capture_id(stream, ctypes.byref(got)))
    return got.value


class Scratch:
    """zeroed: the first FLAG_BYTES of a buffer start as zeros (and the kernels leave them so)."""

    def __init__(self, zeroed):
        self.zeroed = zeroed
        self._streams = {}      # (device index, stream) -> what get() returns; csrc/fast_ops.cpp reads it, too
        self._flags = {}        # device index -> (blocks, flags handed out)
        self._captures = {}     # (device index, stream, capture) -> address of its flags

    def get(self, device, stream, nbytes):
        """(address, bytes, address of the flags or None where they lead the buffer, the buffer: hold it until the launch)"""
        if _capturing():
            return self._captured(device, stream, nbytes)
        held = self._streams.get((device.index, stream))
        if held is None or held[1] < nbytes:
            held = self._grown(device, stream, nbytes)
        return held

    def _grown(self, device, stream, nbytes):
        with _lock:
            if self.zeroed:
                self._more_flags(device)
            buf = (torch.zeros if self.zeroed else torch.empty)(max(nbytes, _SMALLEST), dtype=torch.uint8, device=device)
            self._streams.pop((device.index, stream), None)
            while len(self._streams) >= _MOST_STREAMS:
                self._streams.pop(next(iter(self._streams)))
            held = self._streams[device.index, stream] = buf.data_ptr(), buf.numel(), None, buf
            return held

    def _more_flags(self, device):
        blocks, used = self._flags.get(device.index, ([], 0))
        if used == len(blocks) * _FLAGS_PER_BLOCK and len(blocks) < _MOST_BLOCKS:
            block = torch.zeros(_FLAGS_PER_BLOCK * FLAG_BYTES, dtype=torch.uint8, device=device)
            if block.is_cuda:
                torch.cuda.current_stream(device).synchronize()      # a replay need not come after this stream
            self._flags[device.index] = blocks + [block], used

    def _captured(self, device, stream, nbytes):
        buf = torch.empty(nbytes, dtype=torch.uint8, device=device)
        if not self.zeroed:
            return buf.data_ptr(), nbytes, None, buf
        with _lock:
            key = (device.index, stream, _capture_id(stream))
            flags = self._captures.get(key)
            if flags is None:
                blocks, used = self._flags.get(device.index, ([], 0))
                if used == len(blocks) * _FLAGS_PER_BLOCK:
                    buf[:FLAG_BYTES].zero_()
                    return buf.data_ptr(), nbytes, None, buf
                flags = blocks[-1].data_ptr() + used % _FLAGS_PER_BLOCK * FLAG_BYTES
                self._flags[device.index] = blocks, used + 1
                while len(self._captures) >= _CAPTURES_AT_ONCE:
                    self._captures.pop(next(iter(self._captures)))
                self._captures[key] = flags
            return buf.data_ptr(), nbytes, flags, buf
