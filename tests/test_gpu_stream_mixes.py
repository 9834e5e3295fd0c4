"""Streams that differ, in one batch: speculation windows of different lengths in one cycle, prompts of equal and of
different lengths over layers of the tiled attention (INT4) and of the scalar f32 one (FP8), heads of 64 and 128, 1 to 8 query
heads per KV head, and a fork of more streams than one launch copies pages for.  A stream must follow the CPU oracle as if it
were alone, up to near-ties of the oracle (the 1e-3 rule of the other engine tests)."""

import numpy as np
import pytest

from conftest import GOLDEN

pytestmark = pytest.mark.gpu


def _follow(directory, prompts, drafts, lengths, capacity=128, max_lanes=64, chunk=32):
    import llmoop_b200 as nb
    from oracle.nerve_oracle import Oracle, OraclePackage, OracleStream
    from oracle.parity import follow_generation, summary

    opkg = OraclePackage(directory)
    oracle = Oracle(opkg)
    package = nb.Package(directory, capacity_tokens=capacity, page_tokens=16, max_streams=len(prompts), max_lanes=max_lanes, verify_level=0)
    engine = nb.Engine(package)
    engine.set_prefill_chunk(chunk)
    engine.set_cycle_logging(True)
    for i, prompt in enumerate(prompts):
        engine.add_stream(i, speculative_draft_tokens=drafts[i])
        engine.enqueue_input_event(i, prompt, lengths[i])
    outputs, _ = engine.run_until_idle()
    cycles = engine.cycle_log()
    for i, prompt in enumerate(prompts):
        tokens = [t for sid, t, _, _ in outputs if sid == i]
        report = follow_generation(oracle, OracleStream(opkg, capacity), prompt, tokens, [c for c in cycles if c["stream_id"] == i], drafts[i], prefill_chunk=chunk)
        assert report["tokens_compared"] == len(tokens) == lengths[i] and not report["violations"], (i, summary(report), report["violations"])
        assert report["accepted_equal"], i
        assert engine.stream_tick(i) == len(prompt) + lengths[i]
    engine.close()
    package.unmount()


def _prompts(vocab, lengths, seed):
    rng = np.random.default_rng(seed)
    return [[int(t) for t in rng.integers(0, vocab, size=n)] for n in lengths]


@pytest.mark.parametrize("name,vocab", [("tiny_int4_mtp", 16), ("cfg1_bf16_mtp", 256), ("tiny_moe_fp8_mtp", 16)])
@pytest.mark.parametrize("drafts,lengths", [((3, 3, 3, 3), (2, 5, 9, 12)), ((1, 4, 0, 2, 3), (11, 6, 7, 1, 10))])
def test_windows_of_different_lengths(name, vocab, drafts, lengths):
    _follow(GOLDEN / name, _prompts(vocab, [4 + i for i in range(len(drafts))], sum(lengths)), drafts, lengths)


HEADS = [(2, 2, 64), (8, 1, 64), (2, 2, 128), (8, 1, 128), (4, 2, 128)]


@pytest.mark.parametrize("q_heads,kv_heads,head", HEADS)
def test_wide_int4_heads_uniform_and_ragged(tmp_path, q_heads, kv_heads, head):
    from llmoop_b200.package_writer import write_package
    from llmoop_b200.synth import ModelSpec

    spec = ModelSpec(name="mix_int4", hidden=256, layers=2, q_heads=q_heads, kv_heads=kv_heads, head_dim=head, ffn=256, vocab=256, max_positions=256,
                     quant="int4", std=0.01, seed=31)
    directory = write_package(spec, tmp_path / spec.name)
    for lengths in ((7, 7, 7), (3, 26, 1, 40)):
        _follow(directory, _prompts(spec.vocab, lengths, head + q_heads), [2] * len(lengths), [6] * len(lengths), max_lanes=96, chunk=48)


@pytest.mark.parametrize("q_heads,kv_heads,head", HEADS)
def test_wide_fp8_heads_in_company_and_alone(tmp_path, q_heads, kv_heads, head):
    """FP8 layers add in an order of their own, whatever the batch: a stream in a uniform or ragged batch emits, bit for bit,
    what it emits alone.  (The last bit of an attention output moves quantised values behind it by a sixteenth, which on
    these random layers is up to 0.25 of a logit, so the oracle's tokens say little here; the attention itself is held
    against 64-bit arithmetic by test_gpu_attention_precision.py.)"""
    import llmoop_b200 as nb
    from llmoop_b200.package_writer import write_package
    from llmoop_b200.synth import ModelSpec

    spec = ModelSpec(name="mix_fp8", hidden=256, layers=2, q_heads=q_heads, kv_heads=kv_heads, head_dim=head, ffn=256, vocab=256, max_positions=256,
                     quant="fp8", std=0.08, seed=31)
    directory = write_package(spec, tmp_path / spec.name)
    package = nb.Package(directory, capacity_tokens=128, page_tokens=16, max_streams=4, max_lanes=96, verify_level=0)
    engine = nb.Engine(package)
    engine.set_prefill_chunk(48)

    def run(prompts):
        for i, prompt in enumerate(prompts):
            engine.add_stream(i, speculative_draft_tokens=2)
            engine.enqueue_input_event(i, prompt, 12)
        outputs, _ = engine.run_until_idle()
        logits = [engine.debug_target_logits(i, [5])[0] for i in range(len(prompts))]
        for i in range(len(prompts)):
            engine.remove_stream(i)
        return [([t for sid, t, _, _ in outputs if sid == i], row.tobytes()) for i, row in enumerate(logits)]

    for lengths in ((7, 7, 7), (3, 9, 1, 12), (26, 40, 17)):
        prompts = _prompts(spec.vocab, lengths, head + q_heads)
        together = run(prompts)
        for prompt, got in zip(prompts, together):
            assert run([prompt]) == [got], lengths
    engine.close()
    package.unmount()


@pytest.mark.parametrize("quant,std", [("int4", 0.02), ("bf16", 0.05)])
@pytest.mark.parametrize("lengths,drafts", [((5, 6), (3, 3)), ((30, 45), (3, 3)), ((7, 60), (3, 3)), ((6, 5), (1, 5)), ((20, 4), (4, 2)), ((3, 3, 3), (0, 4, 1))])
def test_streams_of_eight_lanes_together_and_alone(tmp_path, quant, std, lengths, drafts):
    """Streams that decode in eight lanes together, in one cycle or in several: tokens and logits are those of each stream
    alone, bit for bit, whatever the prompts."""
    import llmoop_b200 as nb
    from llmoop_b200.package_writer import write_package
    from llmoop_b200.synth import ModelSpec

    spec = ModelSpec(name=f"mix_{quant}", hidden=512, layers=2, q_heads=4, kv_heads=2, head_dim=128, ffn=512, vocab=256, max_positions=256, quant=quant,
                     std=std, seed=41)
    directory = write_package(spec, tmp_path / spec.name)
    package = nb.Package(directory, capacity_tokens=128, page_tokens=16, max_streams=4, max_lanes=128, verify_level=0)
    engine = nb.Engine(package)
    engine.set_prefill_chunk(128)

    def run(prompts, drafts):
        for i, prompt in enumerate(prompts):
            engine.add_stream(i, speculative_draft_tokens=drafts[i])
            engine.enqueue_input_event(i, prompt, 16)
        outputs, _ = engine.run_until_idle()
        logits = [engine.debug_target_logits(i, [5])[0] for i in range(len(prompts))]
        for i in range(len(prompts)):
            engine.remove_stream(i)
        return [([t for sid, t, _, _ in outputs if sid == i], row.tobytes()) for i, row in enumerate(logits)]

    prompts = _prompts(spec.vocab, lengths, sum(lengths))
    together = run(prompts, drafts)
    assert [run([prompt], [count])[0] for prompt, count in zip(prompts, drafts)] == together
    engine.close()
    package.unmount()


def test_fork_of_more_streams_than_one_launch_copies_pages_for():
    import llmoop_b200 as nb

    forks = 1040
    package = nb.Package(GOLDEN / "cfg1_bf16_mtp", capacity_tokens=32, page_tokens=16, max_streams=forks + 1, max_lanes=forks + 1, verify_level=0)
    engine = nb.Engine(package)
    context, question = _prompts(256, (5, 1), 3)
    engine.add_stream(0)
    engine.submit_input_event_until_idle(0, context, 0)
    for i in range(1, forks + 1):  # every fork writes the page it shares with the others
        engine.fork_stream(0, i)
        engine.enqueue_input_event(i, question, 3)
    outputs, _ = engine.run_until_idle()
    answers = [[] for _ in range(forks + 1)]
    for stream, token, _, _ in outputs:
        answers[stream].append(token)
    assert len(answers[1]) == 3 and all(answer == answers[1] for answer in answers[1:])
    alone, _ = engine.submit_input_event_until_idle(0, question, 3)
    assert alone == answers[1]
    engine.close()
    package.unmount()
