"""Source rules of the prompt kernels that may start while the kernel before them still runs (launch_pdl): what that kernel writes is not read
through the non-coherent path, which wants memory that nobody writes during the reader's whole life."""
import re
from pathlib import Path

import pytest

KERNELS = Path(__file__).resolve().parents[1] / "phaseshift_b200" / "csrc" / "kernels"
CONSTANT = re.compile(r"\b(conv_w|norm_w|bias|wa|wb)\b")          # weights of the model


def bodies(text):
    """(name, text up to the next kernel) of the kernels of a file."""
    parts = re.split(r"\n__global__ ", text)
    return [(re.search(r"(\w+_kernel)\s*\(", p).group(1), p) for p in parts[1:]]


@pytest.mark.parametrize("file", ["gdn_chunked.cu", "gla.cu", "gemm_tc.cu", "attn_tc.cuh"])
def test_results_of_the_predecessor_are_not_read_as_constants(file):
    seen = 0
    for name, body in bodies((KERNELS / file).read_text()):
        if "cudaGridDependencySynchronize();" not in body:
            continue
        seen += 1
        for m in re.finditer(r"__ldg\(([^;]*)", body):
            assert CONSTANT.search(m.group(1)), (name, m.group(0)[:90])
    assert seen
