"""The kernel-per-operator attention at the edges of its tiles against the CPU oracle, through prefill chunks and verify
batches of a small INT4 package with 128- and 64-wide heads: chunk rows (lanes x query heads per kv head) around the
96-row switch between its two forms and around 128-row blocks, contexts around the 64-token tiles and over more than one
split.  Logits of the chunk's last lanes within the bars of the other engine tests."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LOGIT_MAX, LOGIT_MEAN = 2e-2, 2e-3


@pytest.fixture(scope="module", params=[(128, 4, 1), (64, 8, 2)], ids=["hd128_g4", "hd64_g4"])
def package(request, tmp_path_factory):
    from llmoop_b200.package_writer import write_package
    from llmoop_b200.synth import ModelSpec

    head, q_heads, kv_heads = request.param
    spec = ModelSpec(name=f"attention_{head}", hidden=512, layers=2, q_heads=q_heads, kv_heads=kv_heads, head_dim=head, ffn=256, vocab=512,
                     max_positions=1024, quant="int4", std=0.01, seed=5, mtp=False)
    directory = tmp_path_factory.mktemp("packages") / spec.name
    write_package(spec, directory)
    return directory, spec


@pytest.mark.parametrize("context,chunk", [(0, 24), (0, 25), (63, 9), (64, 33), (65, 64), (300, 65), (511, 97), (700, 129)])
def test_chunk_logits_match_oracle(package, context, chunk):
    import llmoop_b200 as nb
    from oracle.nerve_oracle import Oracle, OraclePackage, OracleStream

    directory, spec = package
    rng = np.random.default_rng(context * 131 + chunk)
    tokens = [int(t) for t in rng.integers(0, spec.vocab, size=context + chunk)]
    opkg = OraclePackage(directory)
    oracle, ostream = Oracle(opkg), OracleStream(opkg, 1024)
    mounted = nb.Package(directory, capacity_tokens=1024, page_tokens=16, max_streams=1, max_lanes=256, verify_level=0)
    engine = nb.Engine(mounted)
    engine.set_decode_stack(False)
    engine.set_prefill_chunk(256)
    engine.add_stream(1)
    if context:
        engine.submit_input_event_until_idle(1, tokens[:context], 0)
        oracle.target_forward(ostream, tokens[:context], 0, want_logits=False)
    logits, _ = engine.debug_target_logits(1, tokens[context:])
    _, want = oracle.target_forward(ostream, tokens[context:], context, want_logits=True)
    difference = np.abs(logits[-8:] - np.asarray(want)[-8:])
    assert difference.max() <= LOGIT_MAX and difference.mean() <= LOGIT_MEAN, (difference.max(), difference.mean())
    engine.close()
    mounted.unmount()
