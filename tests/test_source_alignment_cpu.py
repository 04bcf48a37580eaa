"""Arrays that CUDA code declares itself and reads through a wider vector type
must be declared with that type's alignment: in local memory the compiler may
place them at their element's, and a misaligned vector access faults."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nostrum_pray_gb300", "csrc")
WIDE = {"uint2": 8, "float2": 8, "ulonglong2": 16, "uint4": 16, "float4": 16}


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu*"))), ids=os.path.basename)
def test_arrays_read_as_vectors_are_aligned(path):
    src = open(path).read()
    for m in re.finditer(r"reinterpret_cast<(?:const )?(\w+) \*>\((\w+)(?: \+ \w+)?\)", src):
        wide, name = m.groups()
        if wide not in WIDE:
            continue
        # the array declaration that is nearest above the cast
        decl = list(re.finditer(r"^ *(alignas\((\d+)\) )?(?:__nv_bfloat16|__half|float|uint32_t) %s\[\d+\];" % name,
                                src[:m.start()], re.M))
        if decl:
            assert int(decl[-1].group(2) or 0) >= WIDE[wide], f"{name} read as {wide}"
