"""FP8 and bf16 linears at the edges of their forms, through the operator-level entry points against the CPU oracle: two,
four and eight lanes to a tile with remainders, rows that fill no tile, one block of K and more blocks than are staged at
a time (FP8); one row per warp with one, two or four lanes, K that is no multiple of 8 or 128, more lanes than a tile of
the tensor-core form holds (bf16)."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _setup(values):
    import torch

    from llmoop_b200.safetensors_io import f32_to_bf16_bits

    def dev(array):
        return torch.from_numpy(np.ascontiguousarray(array).view(np.uint8).reshape(-1)).cuda()

    return f32_to_bf16_bits(values), dev


def _check(got, want):
    from llmoop_b200.safetensors_io import bf16_bits_to_f32

    got, reference = bf16_bits_to_f32(got).astype(np.float64), bf16_bits_to_f32(want).astype(np.float64)
    ulp = np.maximum(np.abs(reference), 0.05 * np.sqrt((reference ** 2).mean(axis=1, keepdims=True))) * 2.0 ** -7
    assert (np.abs(got - reference) / ulp).max() <= 1.01
    assert (got == reference).mean() > 0.95


@pytest.mark.parametrize("lanes,n,k", [(1, 31, 128), (2, 100, 128), (3, 33, 256), (4, 64, 384), (5, 129, 768), (8, 130, 2048), (9, 257, 33 * 128), (17, 64, 65 * 128)])
def test_fp8_linear_edges_match_oracle(lanes, n, k):
    import torch

    import llmoop_b200 as nb
    from llmoop_b200.synth import quantize_fp8_block
    from oracle import nerve_oracle as orc

    rng = np.random.default_rng(lanes + n + k)
    wq, wscale = quantize_fp8_block(rng.standard_normal((n, k), dtype=np.float32) * 0.05)
    x, dev = _setup(rng.standard_normal((lanes, k), dtype=np.float32))
    xq, xs = orc.quantize_fp8(x)
    want = np.empty((lanes, n), dtype=np.uint16)
    orc.lib().orc_linear_fp8(orc._p(xq, orc._u8p), orc._p(xs, orc._f32p), orc._p(wq, orc._u8p), orc._p(wscale, orc._u16p), None,
                             orc._p(want, orc._u16p), lanes, n, k, 128, 128)
    buffers = [dev(x), dev(wq), dev(wscale), torch.zeros(lanes * n * 2, dtype=torch.uint8, device="cuda")]
    scratch = [torch.zeros(lanes * k, dtype=torch.uint8, device="cuda"), torch.zeros(lanes * (k // 128), dtype=torch.float32, device="cuda")]
    pointers = [ctypes.c_void_p(t.data_ptr()) for t in buffers + scratch]
    assert nb.library().nerve_b200_op_linear_fp8(*pointers[:4], None, *pointers[4:], lanes, n, k, None) == 0
    torch.cuda.synchronize()
    _check(buffers[3].cpu().numpy().view(np.uint16).reshape(lanes, n), want)


@pytest.mark.parametrize("lanes,n,k", [(1, 7, 64), (2, 33, 64), (3, 130, 200), (5, 64, 100), (8, 129, 2048), (9, 65, 200), (11, 257, 256), (257, 300, 128), (300, 129, 384)])
def test_bf16_linear_edges_match_oracle(lanes, n, k):
    import torch

    import llmoop_b200 as nb
    from oracle import nerve_oracle as orc

    rng = np.random.default_rng(lanes + n + k)
    x, dev = _setup(rng.standard_normal((lanes, k), dtype=np.float32))
    w, _ = _setup(rng.standard_normal((n, k), dtype=np.float32) * 0.05)
    want = np.empty((lanes, n), dtype=np.uint16)
    orc.lib().orc_linear_bf16(orc._p(x, orc._u16p), orc._p(w, orc._u16p), orc._p(want, orc._u16p), lanes, n, k)
    buffers = [dev(x), dev(w), torch.zeros(lanes * n * 2, dtype=torch.uint8, device="cuda")]
    pointers = [ctypes.c_void_p(t.data_ptr()) for t in buffers]
    assert nb.library().nerve_b200_op_linear_bf16(*pointers, None, lanes, n, k, 0, ctypes.c_float(1.0), None) == 0
    torch.cuda.synchronize()
    _check(buffers[2].cpu().numpy().view(np.uint16).reshape(lanes, n), want)
