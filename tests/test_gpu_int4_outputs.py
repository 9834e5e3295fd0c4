"""Outputs and residuals of the INT4 linears need no more alignment than their elements: one bf16 element off, the rows of a
pair no longer share an aligned word.  Equal to the aligned call bit for bit, nothing written around the output."""

import ctypes

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lanes,n,k", [(9, 256, 256), (33, 255, 512), (160, 1024, 256)])
@pytest.mark.parametrize("form", ["plain", "residual", "silu"])
def test_outputs_one_element_off(lanes, n, k, form):
    import torch

    import llmoop_b200 as nb

    lib, generator = nb.library(), torch.Generator(device="cuda")
    generator.manual_seed(n)
    p = lambda tensor: ctypes.c_void_p(tensor.data_ptr())  # noqa: E731
    weights = [torch.randint(-(2**31), 2**31, (n, k // 8), generator=generator, device="cuda").to(torch.int32) for _ in range(2)]
    scales = torch.full((n, k // 128), 0.01, dtype=torch.bfloat16, device="cuda")
    x = torch.randn((lanes, k), generator=generator, device="cuda").to(torch.bfloat16)
    addend = torch.randn(lanes * n, generator=generator, device="cuda").to(torch.bfloat16)

    def run(shift_y, shift_residual):
        memory = torch.full((lanes * n + 8,), 7.0, dtype=torch.bfloat16, device="cuda")
        y, residual = memory[shift_y : shift_y + lanes * n], torch.zeros(lanes * n + 8, dtype=torch.bfloat16, device="cuda")[shift_residual : shift_residual + lanes * n]
        residual.copy_(addend)
        if form == "silu":
            status = lib.nerve_b200_op_linear_int4_silu_pair(p(x), p(weights[0]), p(scales), p(weights[1]), p(scales), p(y), lanes, n, k, None)
        else:
            status = lib.nerve_b200_op_linear_int4(p(x), p(weights[0]), p(scales), p(y), p(residual) if form == "residual" else None, lanes, n, k, 128, None)
        assert status == 0, lib.nerve_b200_last_error()
        torch.cuda.synchronize()
        assert bool((memory[:shift_y] == 7).all()) and bool((memory[shift_y + lanes * n :] == 7).all())
        return y.clone()

    want = run(0, 0)
    for shifts in ((1, 0), (0, 1), (3, 5)):
        assert torch.equal(run(*shifts), want), shifts
