"""Closing ticks that wait for the next step's batch (an event's last token is fed back together with the other streams'
next windows): with a limit on the batches of a run, with windows of different lengths in one cycle, and when the step that
should have run them fails."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def package(tmp_path_factory):
    from llmoop_b200.package_writer import write_package
    from llmoop_b200.synth import ModelSpec

    spec = ModelSpec(name="closing_ticks", hidden=512, layers=3, q_heads=8, kv_heads=2, head_dim=64, ffn=1408, vocab=1024, max_positions=512,
                     quant="int4", std=0.01, seed=7)
    directory = tmp_path_factory.mktemp("packages") / spec.name
    write_package(spec, directory)
    return directory, spec


def _mount(directory):
    import llmoop_b200 as nb

    mounted = nb.Package(directory, capacity_tokens=128, page_tokens=16, max_streams=4, max_lanes=64, verify_level=0)
    return nb.Engine(mounted), mounted


def test_failed_step_keeps_the_closing_tick(package):
    """Two streams finish their events in one step; the callback stops one of them, whose closing tick then is a control step
    of its own, and arms a barrier timeout for it.  The other stream, whose closing tick waited for the batch behind, must
    still take its next event."""
    import llmoop_b200 as nb

    directory, spec = package
    rng = np.random.default_rng(8)
    prompts = [[int(t) for t in rng.integers(0, spec.vocab, size=4)] for _ in range(2)]
    engine, mounted = _mount(directory)

    def generate(stream, with_failure):
        engine.add_stream(stream)
        engine.enqueue_input_event(stream, prompts[0], 3)
        tokens = []
        if with_failure:
            engine.add_stream(9)
            engine.enqueue_input_event(9, prompts[1], 3)

            def on_output(sid, token, tick, index):
                if sid == stream:
                    tokens.append(token)
                elif index == 2:
                    engine.stop_stream_after_current(9)
                    engine.inject_barrier_timeouts(1)

            with pytest.raises(nb.NerveError, match="gave up waiting at a grid barrier"):
                engine.run_until_idle(on_output=on_output)
        else:
            tokens += [token for _, token, _, _ in engine.run_until_idle()[0]]
        engine.enqueue_input_event(stream, prompts[1], 4)
        outputs, _ = engine.run_until_idle()
        tokens += [token for sid, token, _, _ in outputs if sid == stream]
        return tokens, engine.stream_tick(stream)

    want = generate(1, False)
    assert len(want[0]) == 7 and want[1] == 4 + 3 + 4 + 4
    assert generate(2, True) == want
    assert engine.stream_tick(9) == 4 + 3 and engine.snapshot()["idle"]  # its closing tick has run, too
    engine.close()
    mounted.unmount()


@pytest.mark.parametrize("drafts", [0, 2])
def test_stopping_a_stream_at_its_last_token(package, drafts):
    """A callback stops a stream whose event it has just seen the last token of: the closing tick runs as a control step, once,
    the run reports that the scheduler had given the activation up, and both streams take their next events."""
    import llmoop_b200 as nb

    directory, spec = package
    rng = np.random.default_rng(9)
    prompts = [[int(t) for t in rng.integers(0, spec.vocab, size=4)] for _ in range(2)]
    engine, mounted = _mount(directory)
    for stream in (1, 2):
        engine.add_stream(stream, speculative_draft_tokens=drafts)
        engine.enqueue_input_event(stream, prompts[0], 3)
    with pytest.raises(nb.NerveError, match="activation"):
        engine.run_until_idle(on_output=lambda sid, token, tick, index: engine.stop_stream_after_current(2) if sid == 2 and index == 2 else None)
    engine.run_until_idle()
    assert [engine.stream_tick(stream) for stream in (1, 2)] == [7, 7]
    for stream in (1, 2):
        engine.enqueue_input_event(stream, prompts[1], 3)
    outputs, _ = engine.run_until_idle()
    tokens = [[token for sid, token, _, _ in outputs if sid == stream] for stream in (1, 2)]
    assert tokens[0] == tokens[1] and len(tokens[0]) == 3
    assert [engine.stream_tick(stream) for stream in (1, 2)] == [14, 14]
    engine.close()
    mounted.unmount()


def test_failed_control_step_is_repeated(package):
    """A stream is stopped between two runs and the batch of its closing tick fails: the next run repeats it, and the stream
    takes its next event."""
    import llmoop_b200 as nb

    directory, spec = package
    prompt = [int(t) for t in np.random.default_rng(10).integers(0, spec.vocab, size=4)]
    engine, mounted = _mount(directory)
    engine.add_stream(1)
    engine.enqueue_input_event(1, prompt, 8)
    first, _ = engine.run(2)
    emitted = len(first)
    engine.stop_stream_after_current(1)
    engine.inject_barrier_timeouts(1)
    with pytest.raises(nb.NerveError, match="gave up waiting at a grid barrier"):
        engine.run_until_idle()
    engine.enqueue_input_event(1, prompt, 3)
    outputs, _ = engine.run_until_idle()
    assert len(outputs) == 3 and engine.stream_tick(1) == 4 + emitted + 4 + 3
    engine.close()
    mounted.unmount()


@pytest.mark.parametrize("drafts", [0, 2])
def test_bounded_runs_end_with_their_closing_ticks(package, drafts):
    """Runs of one batch each: a run that has emitted an event's last token has run its closing tick, too; the tokens are those
    of one unbounded run."""
    directory, spec = package
    rng = np.random.default_rng(12)
    prompts = [[int(t) for t in rng.integers(0, spec.vocab, size=3)] for _ in range(2)]
    lengths = (3, 8)
    engine, mounted = _mount(directory)

    def start(first):
        for i, (prompt, length) in enumerate(zip(prompts, lengths)):
            engine.add_stream(first + i, speculative_draft_tokens=drafts)
            engine.enqueue_input_event(first + i, prompt, length)

    start(1)
    outputs, _ = engine.run_until_idle()
    want = [[token for sid, token, _, _ in outputs if sid == stream] for stream in (1, 2)]
    assert [len(tokens) for tokens in want] == list(lengths)
    start(11)
    got = [[], []]
    for _ in range(40):
        outputs, report = engine.run(1)
        for sid, token, _, _ in outputs:
            got[sid - 11].append(token)
        for i, (tokens, length) in enumerate(zip(got, lengths)):
            if len(tokens) == length:
                assert engine.stream_tick(11 + i) == len(prompts[i]) + length
                counts = engine.scheduler_stream_counts(11 + i)
                assert counts["in_flight_activation_count"] == 0 and counts["completed_input_event_count"] == 1, counts
        if report.idle:
            break
    assert got == want
    engine.close()
    mounted.unmount()
