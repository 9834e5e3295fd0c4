"""Prompts of several streams prefilled in one pass: chunks of equal and of different lengths, more than one query-row
block per stream, single-token chunks, prompts that end in the batch beside ones that go on.  The tokens of each stream must
be those of a run of its own, up to near-ties of the oracle (the 1e-3 rule of the other engine tests)."""

import numpy as np
import pytest

from conftest import GOLDEN

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["tiny_int4_mtp", "tiny_moe_fp8_mtp", "cfg1_bf16_mtp"])
@pytest.mark.parametrize("lengths", [(5, 5, 5, 5), (1, 1, 1), (3, 17, 40, 1, 9), (2, 3, 1), (33, 20)])
def test_batched_prompts_follow_the_oracle(name, lengths):
    import llmoop_b200 as nb
    from oracle.nerve_oracle import Oracle, OraclePackage, OracleStream
    from oracle.parity import follow_generation, summary

    opkg = OraclePackage(GOLDEN / name)
    oracle = Oracle(opkg)
    rng = np.random.default_rng(sum(lengths))
    prompts = [[int(t) for t in rng.integers(0, opkg.vocab, size=n)] for n in lengths]
    package = nb.Package(GOLDEN / name, capacity_tokens=128, page_tokens=16, max_streams=len(prompts), max_lanes=48)
    engine = nb.Engine(package)
    engine.set_prefill_chunk(32)
    engine.set_cycle_logging(True)
    for i, prompt in enumerate(prompts):
        engine.add_stream(i, speculative_draft_tokens=2)
        engine.enqueue_input_event(i, prompt, 8)
    outputs, _ = engine.run_until_idle()
    cycles = engine.cycle_log()
    for i, prompt in enumerate(prompts):
        tokens = [t for sid, t, _, _ in outputs if sid == i]
        report = follow_generation(oracle, OracleStream(opkg, 128), prompt, tokens, [c for c in cycles if c["stream_id"] == i], 2, prefill_chunk=32)
        assert report["tokens_compared"] == len(tokens) == 8 and not report["violations"], (i, summary(report), report["violations"])
        assert engine.stream_tick(i) == len(prompt) + 8
    engine.close()
    package.unmount()
