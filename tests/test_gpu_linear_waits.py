"""The tcgen05 linears start while the kernel in front of them still runs; their bounded waits must not count its time.  In
front stands one CTA that normalises a row of 2^30 columns (about half a second; 2^17 tries of
a wait, the bound that once was too short, take 0.2); the linear's outputs are those it has with nothing in front."""

import ctypes

import pytest

pytestmark = pytest.mark.gpu

WIDTH = 1 << 30


@pytest.fixture(scope="module")
def long_row():
    import torch

    return torch.zeros(WIDTH, dtype=torch.bfloat16, device="cuda"), torch.empty(WIDTH, dtype=torch.bfloat16, device="cuda")


@pytest.mark.parametrize("form,lanes,n,k", [("int4", 16, 4096, 4096), ("int4", 160, 28672, 4096), ("int4", 512, 1024, 8192), ("bf16", 16, 4096, 4096)])
def test_long_kernel_in_front(long_row, form, lanes, n, k):
    import torch

    import llmoop_b200 as nb

    lib = nb.library()
    p = lambda tensor: ctypes.c_void_p(tensor.data_ptr())  # noqa: E731
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    generator = torch.Generator(device="cuda")
    generator.manual_seed(lanes)
    x = torch.randn((lanes, k), generator=generator, device="cuda").to(torch.bfloat16)
    if form == "int4":
        weight = torch.randint(-(2**31), 2**31, (n, k // 8), generator=generator, device="cuda").to(torch.int32)
        scales = torch.full((n, k // 128), 0.01, dtype=torch.bfloat16, device="cuda")
        run = lambda y: lib.nerve_b200_op_linear_int4(p(x), p(weight), p(scales), p(y), None, lanes, n, k, 128, stream)  # noqa: E731
    else:
        weight = torch.randn((n, k), generator=generator, device="cuda").to(torch.bfloat16)
        run = lambda y: lib.nerve_b200_op_linear_bf16(p(x), p(weight), p(y), None, lanes, n, k, 0, ctypes.c_float(1.0), stream)  # noqa: E731
    alone, behind = (torch.zeros((lanes, n), dtype=torch.bfloat16, device="cuda") for _ in range(2))
    assert run(alone) == 0
    row, out = long_row
    begin, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    begin.record()
    assert lib.nerve_b200_op_rms_norm(p(row), p(row), p(out), 1, WIDTH, ctypes.c_float(1e-5), ctypes.c_float(0.0), stream) == 0
    assert run(behind) == 0
    end.record()
    torch.cuda.synchronize()
    assert begin.elapsed_time(end) > 200.0
    assert torch.equal(alone, behind) and bool(alone.abs().max() > 0)
