"""Every kernel that launch_dependent starts may run while its predecessor in the stream still does, so it has to wait for it
before it touches the predecessor's outputs: its body must hold the dependency wait.  Kernels started in the plain way
(triple chevrons, cooperative launches) begin when their predecessor has finished."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "llmoop_b200" / "csrc"
KERNEL = re.compile(r"__global__\s+void(?:\s+__launch_bounds__\((?:[^()]|\([^()]*\))*\))?\s+(\w+)\s*\(")


def _body(text, begin):
    depth, start = 0, text.index("{", begin)
    for at in range(start, len(text)):
        depth += {"{": 1, "}": -1}.get(text[at], 0)
        if depth == 0:
            return text[start:at]
    raise AssertionError("unbalanced braces")


@pytest.mark.parametrize("source", sorted(path.name for path in CSRC.glob("kernels_*.cu")))
def test_dependent_kernels_wait(source):
    text = (CSRC / source).read_text()
    kernels = {match.group(1): _body(text, match.end()) for match in KERNEL.finditer(text)}
    assert kernels
    cooperative = "cudaLaunchCooperativeKernel" in text or "cudaLaunchAttributeCooperative" in text
    for name, body in kernels.items():
        plain = re.search(name + r"(<[^;()]*>)?\s*<<<", text) or (cooperative and "launch_dependent" not in text)
        assert plain or "grid_dependency_wait()" in body, f"{source}: {name} does not wait for its predecessor"
