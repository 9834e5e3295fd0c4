"""The one-launch forward of small dense bf16 models.

Its linears run on tensor cores in tiles of 16 rows and eight lanes, its attention with a warp per (lane, head), a CTA per
stream; wider batches than 32 lanes a stream, fewer than 64 columns and what does not fit its shared memory stay with the
kernels of the single operations.  Widths at the tiles' edges and beyond the last one that it takes, contexts at a page's
edge and around the end of the window (64 tokens), longer ones in a test of their own, each head width; against the oracle and the other route, a lane of any
width equal to the lane alone.

Bars: two faithful orders of summation differ by single bf16 roundings of the hidden state, 2^-8 of a value of order one
each.  Two of them in every column are 2 x 2^-8 x sqrt(hidden) x 0.02 in a logit: 1.2e-3 to 1.8e-3 RMS for 64 to 128
columns, which gives the 2e-3 (mean) and, at some 10 sigma for the largest of all, the 2e-2 of the other tests."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WINDOW = 64
SHAPES = {
    # name: hidden, layers, q heads, kv heads, head width, ffn, vocab
    "hd8": (64, 3, 8, 2, 8, 96, 272),
    "hd16": (64, 2, 4, 2, 16, 128, 256),
    "hd32": (64, 1, 2, 1, 32, 160, 512),
    "large": (96, 1, 4, 4, 32, 160, 512),  # two layers do not fit: the single operations' kernels
    "few_columns": (32, 2, 4, 2, 16, 64, 256),  # too few: the single operations' kernels
}


def _write(name, directory, **options):
    from llmoop_b200.package_writer import write_package
    from llmoop_b200.synth import ModelSpec

    hidden, layers, q_heads, kv_heads, head, ffn, vocab = SHAPES[name]
    spec = ModelSpec(name=f"small_{name}", hidden=hidden, layers=layers, q_heads=q_heads, kv_heads=kv_heads, head_dim=head, ffn=ffn, vocab=vocab, seed=23, **options)
    write_package(spec, directory / spec.name)
    return spec, directory / spec.name


@pytest.fixture(scope="module", params=sorted(SHAPES))
def package(request, tmp_path_factory):
    import llmoop_b200 as nb

    spec, directory = _write(request.param, tmp_path_factory.mktemp("packages"))
    mounted = nb.Package(directory, capacity_tokens=WINDOW, page_tokens=16, max_streams=4, max_lanes=64, verify_level=0)
    yield mounted, directory, spec
    mounted.unmount()


@pytest.mark.parametrize("context", [0, 15, 16, 31, 40, WINDOW - 1, WINDOW + 9])
def test_widths_agree_with_one_lane_and_with_the_oracle(package, context):
    import llmoop_b200 as nb
    from oracle.nerve_oracle import Oracle, OraclePackage, OracleStream

    mounted, directory, spec = package
    rng = np.random.default_rng(context)
    history = [int(t) for t in rng.integers(0, spec.vocab, size=context)]
    probe = [int(t) for t in rng.integers(0, spec.vocab, size=33)]
    engine = nb.Engine(mounted)
    engine.add_stream(1)
    if history:
        engine.submit_input_event_until_idle(1, history, 0)
    oracle_package = OraclePackage(directory)
    oracle = Oracle(oracle_package)
    alone = None
    for lanes in (1, 2, 7, 8, 9, 16, 31, 32, 33):
        stream = OracleStream(oracle_package, WINDOW)
        for i in range(context):
            oracle.target_forward(stream, history[i : i + 1], i, want_logits=False)
        _, expected = oracle.target_forward(stream, probe[:lanes], context, want_logits=True)
        routes = []
        for one_launch in (True, False):
            engine.set_decode_stack(one_launch)
            routes.append(engine.debug_target_logits(1, probe[:lanes])[0])
        # a pass over the window's end overwrites tokens that its first ticks still see in the oracle
        for other in [routes[1]] + ([expected] if lanes == 1 or context + lanes <= WINDOW else []):
            difference = np.abs(routes[0] - other)
            assert difference.max() <= 2e-2 and difference.mean() <= 2e-3, (lanes, difference.max(), difference.mean())
        if spec.name.startswith("small_hd") and lanes <= 32 and context + lanes <= WINDOW:
            alone = routes[0][0].copy() if alone is None else alone
            assert np.array_equal(routes[0][0], alone), (lanes, np.abs(routes[0][0] - alone).max())
    engine.close()


@pytest.mark.parametrize("name, capacity, page_tokens", [("hd8", 624, 16), ("hd16", 1071, 1), ("hd32", 320, 16)])
def test_contexts_of_several_rounds_and_of_many_pages(name, capacity, page_tokens, tmp_path):
    """A thread of the attention takes four tokens at a time (two for heads of 32), a warp 128 (64): contexts at the end of the
    first round, in the second and at the end of the largest windows that are taken; more than 512 pages of a stream's, which
    the kernel reads from global memory.  A window a page larger is left to the kernels of the single operations."""
    import llmoop_b200 as nb
    from oracle.nerve_oracle import Oracle, OraclePackage, OracleStream

    spec, directory = _write(name, tmp_path, max_positions=16384)
    oracle_package = OraclePackage(directory)
    oracle, stream = Oracle(oracle_package), OracleStream(oracle_package, capacity)
    rng = np.random.default_rng(17)
    contexts = [context for context in (63, 64, 126, 127, 129, 500, capacity - 8) if context + 8 <= capacity]
    tokens = [int(t) for t in rng.integers(0, spec.vocab, size=capacity)]
    launches = {}
    for window in (capacity, capacity + 16):
        mounted = nb.Package(directory, capacity_tokens=window, page_tokens=page_tokens, max_streams=2, max_lanes=512, verify_level=0)
        engine = nb.Engine(mounted)
        engine.add_stream(1)
        at = 0
        for context in contexts if window == capacity else ():
            engine.submit_input_event_until_idle(1, tokens[at:context], 0)
            oracle.target_forward(stream, tokens[at:context], at, want_logits=False)
            at = context
            probe = [int(t) for t in rng.integers(0, spec.vocab, size=8)]
            _, expected = oracle.target_forward(stream, probe, context, want_logits=True)  # (overwritten by what follows)
            alone = None
            for lanes in (1, 2, 5, 8):
                engine.set_decode_stack(True)
                got = engine.debug_target_logits(1, probe[:lanes])[0]
                engine.set_decode_stack(False)
                for other in (expected[:lanes], engine.debug_target_logits(1, probe[:lanes])[0]):
                    difference = np.abs(got - other)
                    assert difference.max() <= 2e-2 and difference.mean() <= 2e-3, (context, lanes, difference.max(), difference.mean())
                alone = got[0].copy() if alone is None else alone
                assert np.array_equal(got[0], alone), (context, lanes)
        for route in (True, False):
            engine.set_decode_stack(route)
            engine.add_stream(2)
            engine.enqueue_input_event(2, tokens[:8], 4)
            launches[window, route] = engine.run_until_idle()[1].kernel_launches
            engine.remove_stream(2)
        engine.close()
        mounted.unmount()
    assert 2 * launches[capacity, True] < launches[capacity, False] and launches[capacity + 16, True] == launches[capacity + 16, False], launches


@pytest.mark.parametrize("sampled", [(), (2,), (0, 1, 2, 3)])
def test_streams_beside_one_another_answer_as_alone(package, sampled):
    """Drafts, acceptance and the next tokens of four streams, each also alone, none, one or all of them sampled: a CTA per
    stream shares no value with others.  The kernels of the single operations take many times the launches."""
    import llmoop_b200 as nb

    sampler = {"method": 1, "temperature": 0.8, "top_p": 0.95, "min_p": 0.0, "top_k": 40}
    mounted, _, spec = package
    rng = np.random.default_rng(3)
    questions = [[int(t) for t in rng.integers(0, spec.vocab, size=size)] for size in (1, 9, 17, 30)]
    answers, launches = {}, {}
    for name, groups in (("alone", [[0], [1], [2], [3]]), ("together", [[0, 1, 2, 3]]), ("single operations", [[0, 1, 2, 3]])):
        engine = nb.Engine(mounted)
        engine.set_decode_stack(name != "single operations")
        answers[name], launches[name] = {i: [] for i in range(4)}, 0
        for group in groups:
            for i in group:
                engine.add_stream(i, seed=i, speculative_draft_tokens=i % 2 + 1 if spec.mtp else 0, sampler=sampler if i in sampled else None)
                engine.enqueue_input_event(i, questions[i], 12)
            outputs, report = engine.run_until_idle()
            launches[name] += report.kernel_launches
            for stream, token, _, _ in outputs:
                answers[name][stream].append(token)
        engine.close()
    if spec.name.startswith("small_hd"):
        assert answers["alone"] == answers["together"]
        assert 2 * launches["together"] < launches["single operations"], launches
    else:
        assert launches["together"] == launches["single operations"], launches
