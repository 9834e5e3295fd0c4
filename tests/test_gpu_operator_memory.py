"""The operator-level linears of more than eight lanes take their activations' memory from the library's pool: the very first
call of a process may be captured, its graph replays on new inputs, and calls from several threads on streams of their own
do not disturb one another."""

import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = """
import ctypes, threading
import torch
import llmoop_b200 as nb

lib, n, k = nb.library(), 1024, 2048
p = lambda tensor: ctypes.c_void_p(tensor.data_ptr())
generator = torch.Generator(device="cuda")
generator.manual_seed(1)
weight = torch.randint(-(2**31), 2**31, (n, k // 8), generator=generator, device="cuda").to(torch.int32)
scales = torch.full((n, k // 128), 0.01, dtype=torch.bfloat16, device="cuda")
inputs = [torch.randn((lanes, k), generator=generator, device="cuda").to(torch.bfloat16) for lanes in (9, 24, 160, 512)]

def linear(x, y):
    status = lib.nerve_b200_op_linear_int4(p(x), p(weight), p(scales), p(y), None, x.shape[0], n, k, 128, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert status == 0, lib.nerve_b200_last_error()

new = lambda x: torch.zeros((x.shape[0], n), dtype=torch.bfloat16, device="cuda")
graphs = []
for x in inputs:  # the first one is the process's first call
    buffer, y, graph = torch.zeros_like(x), new(x), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        linear(buffer, y)
    graphs.append((buffer, y, graph))
want = [new(x) for x in inputs]
for x, y in zip(inputs, want):
    linear(x, y)
torch.cuda.synchronize()
for x, y, (buffer, out, graph) in zip(inputs, want, graphs):
    for _ in range(2):
        buffer.copy_(x)
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, y) and bool(y.abs().max() > 0)

failures = []
def worker(x, y):
    try:
        with torch.cuda.stream(torch.cuda.Stream()):
            outs = [new(x) for _ in range(20)]
            for out in outs:
                linear(x, out)
            torch.cuda.current_stream().synchronize()
            assert all(torch.equal(out, y) for out in outs)
    except BaseException as error:
        failures.append(error)

threads = [threading.Thread(target=worker, args=pair) for pair in zip(inputs, want)]
for thread in threads: thread.start()
for thread in threads: thread.join()
assert not failures, failures
print("operators ok")
"""


def test_first_call_under_capture_then_threads():
    result = subprocess.run([sys.executable, "-c", PROGRAM], cwd=Path(__file__).resolve().parent.parent, capture_output=True, text=True, timeout=300)
    assert result.returncode == 0 and "operators ok" in result.stdout, result.stderr[-2000:]
