"""A shared array read or written in 8- or 16-byte vectors has to say so: without an alignment of its own it is only as aligned as
its element, and where the compiler happens to place it decides whether the access faults."""
import glob
import os
import re

import pytest

import lightron_b200

_CSRC = os.path.join(os.path.dirname(lightron_b200.__file__), "csrc")
_BYTES = {"float": 4, "int": 4, "unsigned": 4, "bf16": 2, "uint8_t": 1, "uint64_t": 8, "float2": 8, "float4": 16, "uint4": 16}
_VECTOR = {"float2": 8, "uint2": 8, "int2": 8, "float4": 16, "uint4": 16, "int4": 16}


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(_CSRC, "*.cu*"))), ids=os.path.basename)
def test_vector_accesses_to_shared_arrays_are_aligned(path):
    src = re.sub(r"//[^\n]*", "", open(path).read())
    for align, typ, names in re.findall(r"__shared__\s+(?:__align__\((\d+)\)\s+)?(\w+)\s+([^;]+);", src):
        for name in re.findall(r"(\w+)\s*\[", re.sub(r"\[[^\]]*\]", "[", names)):
            for vec in re.findall(r"reinterpret_cast<(?:const )?(\w+)\*>\(&?%s\b" % name, src):
                if vec in _VECTOR:
                    assert max(int(align or 0), _BYTES.get(typ, 1)) >= _VECTOR[vec], f"{typ} {name} accessed as {vec}"
