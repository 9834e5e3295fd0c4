"""The persistent decode stack kernel at every batch width.

Its products are exact integers (weights as signed bytes, activations as four signed bytes behind a power of two per
group), with one, two or four MMA column tiles by the number of lanes: 1-2, 3-4 and 5-8.  A lane's result must not depend on
the width, so lane 0 of a batch of n lanes has the logits of the same lane alone, bit for bit, and all of them lie within
the bars of the other tests of this kernel against the oracle: 2e-2 and 2e-3 (mean) for logits of the scale that 1024
columns of N(0, 0.01) give them.  Two faithful orders of summation differ by roundings of the hidden state, which the
lm_head carries on as it carries the hidden state itself, so the bars grow as the logits do, with the root of the columns
(8192: by 2.83).  The shapes: a group count that is not a multiple of the
warps' (ragged last step), each built head shape, and rows too wide to be staged whole for eight lanes (8192 columns:
staged in windows, accumulators carried from one to the next)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = {
    # name: hidden, layers, q heads, kv heads, head width, ffn, vocab
    "ragged": (1152, 2, 8, 2, 128, 2176, 512),
    "hd64": (512, 2, 8, 2, 64, 1408, 512),
    "hd32": (384, 2, 8, 4, 32, 640, 512),
    "wide": (8192, 1, 16, 2, 128, 1024, 256),
}


@pytest.fixture(scope="module", params=sorted(SHAPES))
def package(request, tmp_path_factory):
    import llmoop_b200 as nb
    from llmoop_b200.package_writer import write_package
    from llmoop_b200.synth import ModelSpec

    hidden, layers, q_heads, kv_heads, head, ffn, vocab = SHAPES[request.param]
    spec = ModelSpec(name=f"stack_lanes_{request.param}", hidden=hidden, layers=layers, q_heads=q_heads, kv_heads=kv_heads, head_dim=head, ffn=ffn,
                     vocab=vocab, max_positions=512, quant="int4", std=0.01, seed=11)
    directory = tmp_path_factory.mktemp("packages") / spec.name
    write_package(spec, directory)
    mounted = nb.Package(directory, capacity_tokens=256, page_tokens=16, max_streams=2, max_lanes=96, verify_level=0)
    assert mounted.info["target_decode_stack"] == 1
    yield mounted, directory, spec
    mounted.unmount()


def test_every_width_agrees_with_one_lane_and_with_the_oracle(package):
    import llmoop_b200 as nb
    from oracle.nerve_oracle import Oracle, OraclePackage, OracleStream

    mounted, directory, spec = package
    rng = np.random.default_rng(5)
    context = [int(t) for t in rng.integers(0, spec.vocab, size=67)]
    probe = [int(t) for t in rng.integers(0, spec.vocab, size=8)]
    oracle_package = OraclePackage(directory)
    oracle = Oracle(oracle_package)
    stream = OracleStream(oracle_package, 256)
    oracle.target_forward(stream, context, 0, want_logits=False)
    _, expected = oracle.target_forward(stream, probe, len(context), want_logits=True)

    engine = nb.Engine(mounted)
    engine.set_decode_stack(True)
    engine.add_stream(1)
    engine.submit_input_event_until_idle(1, context, 0)
    alone, wider = None, max(1.0, spec.hidden / 1024) ** 0.5
    for lanes in range(1, 9):
        logits, _ = engine.debug_target_logits(1, probe[:lanes])
        if alone is None:
            alone = logits[0].copy()
        assert np.array_equal(logits[0], alone), (lanes, np.abs(logits[0] - alone).max())
        difference = np.abs(logits - expected[:lanes])
        assert difference.max() <= 2e-2 * wider and difference.mean() <= 2e-3 * wider, (lanes, difference.max(), difference.mean())
    engine.close()
