"""A parallel block: one RMSNorm feeds q/k/v and, behind o, the gate/up pair too.  Its readers stand on both sides of
another INT4 linear's input, so above eight lanes the norm's operand form has to be prepared again for the second ones.
Logits against the CPU oracle around the eight-lane switch; synthetic weights, tokens uniform over the vocabulary."""

import json

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LOGIT_MAX, LOGIT_MEAN = 2e-2, 2e-3


@pytest.fixture(scope="module")
def package(tmp_path_factory):
    from llmoop_b200.package_writer import write_package
    from llmoop_b200.synth import ModelSpec

    spec = ModelSpec(name="parallel_block", hidden=256, layers=2, q_heads=4, kv_heads=2, head_dim=64, ffn=384, vocab=256, max_positions=256,
                     quant="int4", std=0.05, seed=11, mtp=False)
    directory = write_package(spec, tmp_path_factory.mktemp("packages") / spec.name)
    path = directory / "vulkan_resident_package.json"
    manifest = json.loads(path.read_text())
    moved = 0
    for component in manifest["circuit_graph"]["components"]:
        for nodes in ("nodes", "semantic_execution_nodes"):
            for node in component["circuit"].get(nodes, []):
                if node["id"] in ("ffn_gate_projection", "ffn_up_projection"):
                    assert node["inputs"] == ["ffn_norm_out"]
                    node["inputs"] = ["operator_norm_out"]
                    moved += 1
    assert moved >= 2 * spec.layers
    path.write_text(json.dumps(manifest))
    return directory, spec


@pytest.mark.parametrize("lanes", [8, 9, 24])
def test_readers_on_both_sides_of_another_linear(package, lanes):
    import llmoop_b200 as nb
    from oracle.nerve_oracle import Oracle, OraclePackage, OracleStream

    directory, spec = package
    tokens = [int(t) for t in np.random.default_rng(lanes).integers(0, spec.vocab, size=lanes)]
    opkg = OraclePackage(directory)
    _, want = Oracle(opkg).target_forward(OracleStream(opkg, 64), tokens, 0, want_logits=True)
    mounted = nb.Package(directory, capacity_tokens=64, page_tokens=16, max_streams=1, max_lanes=32, verify_level=0)
    engine = nb.Engine(mounted)
    engine.add_stream(1)
    logits, _ = engine.debug_target_logits(1, tokens)
    difference = np.abs(logits - np.asarray(want))
    assert difference.max() <= LOGIT_MAX and difference.mean() <= LOGIT_MEAN, (difference.max(), difference.mean())
    engine.close()
    mounted.unmount()
