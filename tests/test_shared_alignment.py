"""A shared array that is read or written through a wider vector type must say that type's alignment itself: where the compiler
places the array among a kernel's others is no promise."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "wuda_b200", "csrc")
FILES = sorted(glob.glob(os.path.join(CSRC, "*.cu*")))
VECTORS = {"uint4": 16, "int4": 16, "float4": 16, "ulonglong2": 16, "uint2": 8, "int2": 8, "float2": 8, "uint64_t": 8}
SCALARS = {"float": 4, "int": 4, "int32_t": 4, "uint32_t": 4, "uint16_t": 2, "__nv_bfloat16": 2, "uint8_t": 1, **VECTORS}
SHARED = re.compile(r"(?:(?<!extern )__shared__)\s+(?:(?:__align__|alignas)\((\d+)\)\s+)?(\w+)\s+(\w+)\s*\[")


def too_narrow(source):
    found = []
    for m in SHARED.finditer(source):
        stated, kind, name = m.groups()
        aligned = max(int(stated or 0), SCALARS.get(kind, 0))
        for vector, bytes_ in VECTORS.items():
            if re.search(r"reinterpret_cast<(?:const\s+)?%s\s*[*&]>\(\s*&?%s\b" % (vector, name), source) and aligned < bytes_:
                found.append((name, vector))
    return found


@pytest.mark.parametrize("path", FILES, ids=os.path.basename)
def test_shared_arrays_have_the_alignment_of_their_accesses(path):
    with open(path) as f:
        assert too_narrow(f.read()) == []
