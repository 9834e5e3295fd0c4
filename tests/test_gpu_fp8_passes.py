"""FP8 linears and experts whose CTAs take more rows than their warps hold at a time.

The rows of a CTA go with the size of the launch (32 to 256 for a linear, one to four passes for experts); the sums and their
order do not depend on it, so a large batch has the bits of the same lanes in batches of eight, and a prompt prefilled at
once the logits of one prefilled in shorter pieces, which take fewer passes.  Rows that end inside a pass, and a last lane
tile that is not full."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lanes,n,k", [(50, 2040, 384), (765, 2040, 128), (1485, 2040, 256), (1483, 2050, 4224)])
def test_linear_has_the_bits_of_batches_of_eight(lanes, n, k):
    import torch

    import llmoop_b200 as nb
    from llmoop_b200.synth import quantize_fp8_block

    library, pointer = nb.library(), lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    rng = np.random.default_rng(lanes)
    packed, scales = quantize_fp8_block(rng.standard_normal((n, k), dtype=np.float32) * 0.05)
    w, s = torch.from_numpy(packed).cuda(), torch.from_numpy(scales.view(np.int16)).cuda()
    torch.manual_seed(lanes)
    x = torch.randn(lanes, k, device="cuda").to(torch.bfloat16)

    def linear(rows):
        y = torch.zeros(len(rows), n, dtype=torch.int16, device="cuda")
        xq = torch.zeros(len(rows) * k, dtype=torch.uint8, device="cuda")
        xs = torch.zeros(len(rows) * (k // 128), dtype=torch.float32, device="cuda")
        assert library.nerve_b200_op_linear_fp8(pointer(rows), pointer(w), pointer(s), pointer(y), None, pointer(xq), pointer(xs), len(rows), n, k, None) == 0
        torch.cuda.synchronize()
        return y

    together = linear(x)
    for first in range(0, lanes, 8):
        assert torch.equal(together[first : first + 8], linear(x[first : first + 8])), first


def test_prompt_through_experts_at_once_and_in_pieces(tmp_path):
    import llmoop_b200 as nb
    from llmoop_b200.package_writer import write_package
    from llmoop_b200.synth import ModelSpec

    spec = ModelSpec(name="experts_passes", hidden=256, layers=1, q_heads=2, kv_heads=1, head_dim=128, ffn=256, vocab=512, max_positions=2048, quant="fp8", std=0.05,
                     experts=16, experts_per_token=8, moe_ffn=384, qk_norm=True, seed=5)
    package = nb.Package(write_package(spec, tmp_path / spec.name), capacity_tokens=2048, page_tokens=16, max_streams=2, max_lanes=1024, verify_level=0)
    prompt = [int(t) for t in np.random.default_rng(2).integers(0, spec.vocab, size=1024)]
    logits = []
    for chunk in (1024, 400, 24):  # four passes, two, one
        engine = nb.Engine(package)
        engine.set_prefill_chunk(chunk)
        engine.add_stream(1)
        engine.submit_input_event_until_idle(1, prompt, 0)
        logits.append(engine.debug_target_logits(1, prompt[:3])[0].copy())
        engine.close()
    package.unmount()
    assert np.array_equal(logits[0], logits[1]), np.abs(logits[0] - logits[1]).max()
    assert np.array_equal(logits[0], logits[2]), np.abs(logits[0] - logits[2]).max()
