"""A draft adapter whose projection is INT4 and takes more columns (twice the hidden size) than any INT4 matrix of the layers:
the buffer of the GEMM's operand form has to hold it.  Prompts of more than eight lanes run the adapter through the GEMM; tokens
and acceptance must follow the CPU oracle, up to near-ties (the 1e-3 rule of the other engine tests)."""

import json

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def package(tmp_path_factory):
    from llmoop_b200.package_writer import write_package
    from llmoop_b200.safetensors_io import write_safetensors
    from llmoop_b200.synth import ModelSpec, quantize_int4_group

    spec = ModelSpec(name="int4_adapter", hidden=512, layers=1, q_heads=4, kv_heads=2, head_dim=128, ffn=256, vocab=256, max_positions=256, quant="int4",
                     std=0.02, seed=51)
    directory = write_package(spec, tmp_path_factory.mktemp("packages") / spec.name)
    path = directory / "vulkan_resident_package.json"
    manifest = json.loads(path.read_text())
    index_path = directory / manifest["tensor_index_path"]
    index = json.loads(index_path.read_text())
    packed, scales = quantize_int4_group(np.random.default_rng(3).standard_normal((spec.hidden, 2 * spec.hidden), dtype=np.float32) * np.float32(0.04))
    tensors = {"mtp.fc.weight_packed": ("I32", np.ascontiguousarray(packed).view(np.uint32)), "mtp.fc.weight_scale": ("BF16", scales)}
    like = {"mtp.fc.weight_packed": "model.layers.0.self_attn.q_proj.weight_packed", "mtp.fc.weight_scale": "model.layers.0.self_attn.q_proj.weight_scale"}
    for i, (name, (dtype, data)) in enumerate(tensors.items()):
        file = f"weights/adapter_{i}.safetensors"
        write_safetensors(directory / file, {name: (dtype, data.shape, data)})
        entry = dict(index["tensors"][like[name]], dtype=dtype, shape=list(data.shape), data_offsets=[0, data.nbytes], parameter_count=int(data.size),
                     byte_count=data.nbytes, source_file=file)
        entry.pop("data_sha256", None)
        if name.endswith("packed"):
            entry["logical_shape"] = [spec.hidden, 2 * spec.hidden]
            entry["quantization"] = dict(entry["quantization"], scales="mtp.fc.weight_scale")
        index["tensors"][name] = entry
    index_path.write_text(json.dumps(index))
    moved = 0
    for component in manifest["speculative_decoders"][0]["circuit_graph"]["components"]:
        refs = component["circuit"]["parameters"]["refs"]
        if "input_projection" in refs:
            refs["input_projection"]["tensor"] = "mtp.fc.weight_packed"
            moved += 1
    assert moved == 1
    path.write_text(json.dumps(manifest))
    return directory, spec


@pytest.mark.parametrize("length", [5, 23, 60])
def test_int4_adapter_follows_the_oracle(package, length):
    import llmoop_b200 as nb
    from oracle.nerve_oracle import Oracle, OraclePackage, OracleStream
    from oracle.parity import follow_generation

    directory, spec = package
    prompt = [int(t) for t in np.random.default_rng(length).integers(0, spec.vocab, size=length)]
    mounted = nb.Package(directory, capacity_tokens=128, page_tokens=16, max_streams=1, max_lanes=64, verify_level=0)
    engine = nb.Engine(mounted)
    engine.set_prefill_chunk(64)
    engine.set_cycle_logging(True)
    engine.add_stream(1, speculative_draft_tokens=2)
    tokens, _ = engine.submit_input_event_until_idle(1, prompt, 10)
    opkg = OraclePackage(directory)
    report = follow_generation(Oracle(opkg), OracleStream(opkg, 128), prompt, tokens, engine.cycle_log(), 2)
    assert report["tokens_compared"] == len(tokens) == 10 and not report["violations"] and report["accepted_equal"], report["violations"]
    engine.close()
    mounted.unmount()
