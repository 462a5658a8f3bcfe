"""Shared arrays of the kernels that are read or written in vectors declare an alignment: where the compiler places a plain array is its
own affair, and a misaligned vector access ends the context."""
import re
from pathlib import Path

import pytest

KERNELS = Path(__file__).resolve().parent.parent / "phaseshift_b200" / "csrc" / "kernels"
VECTOR = r"reinterpret_cast<(?:const )?(?:float2|float4|double2|uint2|uint4|int2|int4|uint32_t|uint64_t)\s*\*>\(\s*&?\(?"


@pytest.mark.parametrize("path", sorted(p for p in KERNELS.iterdir() if p.suffix in (".cu", ".cuh")), ids=lambda p: p.name)
def test_vector_accesses_to_shared_arrays_are_aligned(path):
    text = re.sub(r"//[^\n]*", "", path.read_text())
    for kernel in re.split(r"__global__", text)[1:]:
        for kind, names in re.findall(r"^\s*__shared__ (float|__half|__nv_bfloat16|uint8_t|uint16_t) ([^;]*);", kernel, re.M):
            for name in re.findall(r"(\w+)(?:\[[^\]]*\])+", names):
                alias = re.findall(r"\b(?:%s|auto)\s*\*\s*(\w+)\s*=\s*&?%s\b" % (kind, name), kernel)
                for n in [name, *alias]:
                    assert not re.search(VECTOR + re.escape(n) + r"\b", kernel), (path.name, name)
