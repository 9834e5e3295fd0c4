"""The INT4 tensor-core linear of more than eight lanes at the edges of its tiles and ranges, through the operator-level
entry point against the CPU oracle: lane tiles of 16 with remainders, one and two row tiles per CTA, ragged last row
tiles, a single group of K, K split over a cluster, more than one lane tile; activations and group scales far from 1
(both enter the tensor core as fp16 behind a power of two per lane and per row), and scales of a row far from and close
to one another (two forms of the operands)."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lanes,n,k", [
    (9, 128, 128), (16, 130, 256), (17, 64, 4096), (64, 1000, 384), (65, 257, 1152), (128, 96, 2048), (129, 384, 640), (256, 128, 128), (257, 300, 256),
    (150, 19000, 384), (310, 18945, 128),  # two row tiles of 160 lanes: half groups
])
@pytest.mark.parametrize("x_scale,w_scale,spread", [(1.0, 0.02, 8), (2.0 ** 90, 2.0 ** -60, 3), (2.0 ** -100, 2.0 ** 40, 5)])
def test_int4_gemm_edges_match_oracle(lanes, n, k, x_scale, w_scale, spread):
    import torch

    import llmoop_b200 as nb
    from llmoop_b200.safetensors_io import bf16_bits_to_f32, f32_to_bf16_bits
    from llmoop_b200.synth import quantize_int4_group
    from oracle import nerve_oracle as orc

    rng = np.random.default_rng(lanes * 7 + n + k)
    packed, scales = quantize_int4_group(rng.standard_normal((n, k), dtype=np.float32))
    scales = f32_to_bf16_bits(bf16_bits_to_f32(scales) * np.float32(w_scale) * (2.0 ** rng.integers(-spread, 1, size=scales.shape)).astype(np.float32))
    x = rng.standard_normal((lanes, k), dtype=np.float32) * np.float32(x_scale)
    x[:, ::7] *= np.float32(2.0 ** -12)  # far smaller values beside them
    x = f32_to_bf16_bits(x)
    want = np.empty((lanes, n), dtype=np.uint16)
    orc.lib().orc_linear_int4_ct(orc._p(x, orc._u16p), orc._p(packed.view(np.uint32), orc._u32p), orc._p(scales, orc._u16p),
                                 orc._p(want, orc._u16p), lanes, n, k, 128)

    def dev(array):
        return torch.from_numpy(np.ascontiguousarray(array).view(np.uint8).reshape(-1)).cuda()

    dx, dq, ds = dev(x), dev(packed), dev(scales)
    dy = torch.zeros(lanes * n * 2, dtype=torch.uint8, device="cuda")
    pointers = [ctypes.c_void_p(t.data_ptr()) for t in (dx, dq, ds, dy)]
    status = nb.library().nerve_b200_op_linear_int4(*pointers, None, lanes, n, k, 128, None)
    assert status == 0, nb.library().nerve_b200_last_error()
    torch.cuda.synchronize()
    got_bits = dy.cpu().numpy().view(np.uint16).reshape(lanes, n)
    got, reference = bf16_bits_to_f32(got_bits).astype(np.float64), bf16_bits_to_f32(want).astype(np.float64)
    # one bf16 ulp of the value, or - for sums that cancel to almost nothing - of the typical output magnitude of the lane
    ulp = np.maximum(np.abs(reference), 0.05 * np.sqrt((reference ** 2).mean(axis=1, keepdims=True))) * 2.0 ** -7
    assert (np.abs(got - reference) / ulp).max() <= 1.01
    assert (got_bits == want).mean() > 0.97
