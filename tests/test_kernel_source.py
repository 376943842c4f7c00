"""Rules that the kernel sources keep and that no run on a healthy GPU can show."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "channel_passive_b200" / "csrc"


def _kernels(name):
    """(kernel, body) of the __global__ functions of a source file, comments removed."""
    text = re.sub(r"//[^\n]*", "", (CSRC / name).read_text())
    for part in text.split("__global__")[1:]:
        head, body = part.split("{", 1)
        end = body.find("\n}\n")
        yield re.findall(r"(\w+)\s*\(", head)[-1], body[:end]


@pytest.mark.parametrize("source", ["line_solver.cu", "mean.cu"])
def test_blocks_leave_a_failed_step_together(source):
    """k_lines raises the error flag while other blocks of it, and k_mean beside it, start: a kernel with
    barriers may not let each thread decide on its own reading of the flag."""
    seen = 0
    for kernel, body in _kernels(source):
        if "__syncthreads" not in body:
            continue
        seen += 1
        assert "block_failed(a.dsc)" in body, kernel
        assert not re.search(r"if\s*\([^)]*dsc->err", body), kernel
        assert body.index("block_failed") < body.index("__syncthreads"), kernel
    assert seen >= 1
