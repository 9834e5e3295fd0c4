"""What the framework's users have it do, as cases that can be timed: conversations run through the engine's public
calls (fork_stream / add_stream, enqueue_input_event, run_until_idle, debug_target_logits, remove_stream), and the INT4
linear through its operator-level entry point.

A turn is one request of one or several streams: `streams` streams start from a shared context of `context` tokens that
is already in the KV cache (0: fresh streams), each takes a question of `question` tokens of its own (prefill), answers
with `answer` greedy or sampled tokens, `drafts` speculated per cycle (decode), and one stream's next-token logits are
read, as by a client that wants log-probabilities.

Models, written as compiled packages with synthetic weights:
  8b    the benchmark's configuration: 32 layers, hidden 4096, 32 q / 8 kv heads of 128, FFN 14336, vocabulary 128256,
        INT4 g128 weights, bf16 embedding and lm_head, one MTP layer;
  moe   four layers of the sparse-expert configuration: hidden 2048, 32 q / 4 kv heads of 128, 128 experts of 768, top
        8, FP8 e4m3 weights with 128x128 block scales, vocabulary 151936, one MTP layer;
  tiny  the smallest configuration: 2 layers, hidden 64, 4 q / 2 kv heads of 16, FFN 128, vocabulary 256, bf16, one MTP
        layer.
Layer weights are N(0, std).  Embedding and lm_head are made so that a token's successor wins by a margin that
rounding cannot turn, as a trained model's mostly does: embedding(t) = scale x v(t), lm_head(next(t)) = 0.02 x v(t) with
`next` a random permutation.  v(t) lives in the first half of the columns for seven tokens of ten, in the second half
for the others; the MTP adapter hands on the first half only, so that seven drafts of ten are accepted.
"""

import ctypes
import itertools
import math
import os
import shutil
import tempfile
from pathlib import Path

import numpy as np
import torch

import llmoop_b200 as nb
from llmoop_b200.package_writer import write_package
from llmoop_b200.synth import LLAMA3_8B_INT4, ModelSpec, iter_checkpoint_torch

EASY = 0.7  # share of the tokens whose successor the MTP layer predicts

# name -> (shape, scale of the embedding against the layers' contributions, mount options, prefill chunk)
MODELS = {
    "8b": (ModelSpec(name="perf_8b_int4", seed=0, **LLAMA3_8B_INT4), 12.0,
           dict(capacity_tokens=10240, page_tokens=16, max_streams=48, max_lanes=2048), 2048),
    "moe": (ModelSpec(name="perf_moe_fp8_4l", hidden=2048, layers=4, q_heads=32, kv_heads=4, head_dim=128, ffn=768, vocab=151936,
                      max_positions=4096, rope_theta=1000000.0, quant="fp8", std=0.05, experts=128, experts_per_token=8, moe_ffn=768,
                      qk_norm=True, seed=1), 6.0,
            dict(capacity_tokens=4096, page_tokens=16, max_streams=48, max_lanes=2048), 2048),
    "tiny": (ModelSpec(name="perf_tiny_bf16", hidden=64, layers=2, q_heads=4, kv_heads=2, head_dim=16, ffn=128, vocab=256, quant="bf16",
                       std=0.08, seed=2), 2.0,
             dict(capacity_tokens=256, page_tokens=16, max_streams=48, max_lanes=256), 256),
}


def listed():
    def turn(name, model, streams, context, question, answer, drafts, sampled=False):
        return {"name": name, "model": model, "streams": streams, "context": context, "question": question, "answer": answer,
                "drafts": drafts, "sampled": sampled}

    return [
        # the smallest calls: one short exchange with the tiny model, all latency and launches
        turn("tiny_exchange", "tiny", 1, 0, 16, 32, 1),
        # the benchmark: one user's answer, speculative, behind a 512-token prompt
        turn("chat", "8b", 1, 512, 1, 64, 3),
        # the same without speculation: one token per step
        turn("chat_no_drafts", "8b", 1, 300, 1, 32, 0),
        # sampled with temperature, top-k and top-p, speculative
        turn("chat_sampled", "8b", 1, 1100, 1, 48, 3, True),
        # time to the first tokens of a short question
        turn("short_question", "8b", 1, 0, 37, 4, 3),
        # the benchmark's prompt
        turn("prompt", "8b", 1, 0, 512, 1, 3),
        # a follow-up turn of a long conversation: ragged prefill at a long context, then decoding there
        turn("long_conversation", "8b", 1, 8000, 713, 24, 3),
        # eight users of one document at once: 32 verify lanes per cycle
        turn("eight_streams", "8b", 8, 700, 9, 24, 3),
        # thirty-two users: 160 verify lanes per cycle
        turn("thirty_two_streams", "8b", 32, 450, 21, 16, 4),
        # eight users of the sparse-expert model, two drafts
        turn("moe_eight_streams", "moe", 8, 1024, 5, 32, 2),
        # the sparse-expert model's prompt
        turn("moe_prompt", "moe", 1, 0, 1024, 1, 2),
        # one linear of the largest configuration's layers (hidden 8192, FFN 28672) at its 160 verify lanes
        {"name": "linear_int4_wide", "model": "linear", "lanes": 160, "n": 28672, "k": 8192},
    ]


def _log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    limit = max(_cost(case) for case in listed())
    while True:
        model = rng.choices(["8b", "moe", "tiny", "linear"], [6, 2, 1, 1])[0]
        if model == "linear":  # the layers' matrices of the 8B and 70B configurations
            n, k = rng.choice([(4096, 4096), (1024, 4096), (14336, 4096), (4096, 14336), (8192, 8192), (28672, 8192), (8192, 28672)])
            case = {"model": model, "lanes": _log_uniform(rng, 1, 512), "n": n, "k": k}
        else:
            largest = {"8b": 8192, "moe": 2048, "tiny": 96}[model]
            case = {
                "model": model,
                "streams": rng.choice([1, 1, 1, _log_uniform(rng, 2, 32)]),
                "context": rng.choice([0, _log_uniform(rng, 16, largest)]),
                "question": _log_uniform(rng, 1, min(1500, largest)),
                "answer": _log_uniform(rng, 1, 64),
                "drafts": rng.choice([0, 1, 2, 3, 3, 4]),
                "sampled": rng.random() < 0.25,
            }
            if case["streams"] * case["question"] > 2048:
                continue
        if _cost(case) <= limit:
            return case


# ---- what a pass cannot do without


def _layer(spec):
    """(weights outside the experts, weights of one expert, bytes per weight) of one layer."""
    h, q, kv = spec.hidden, spec.q_heads * spec.head_dim, spec.kv_heads * spec.head_dim
    attention = h * (q + 2 * kv) + q * h
    per = {"int4": 0.5 + 2 / 128, "fp8": 1.0, "bf16": 2.0}[spec.quant]
    if spec.experts:
        return attention + spec.experts * h, 3 * h * spec.moe_ffn, per
    return attention + 3 * h * spec.ffn, 0, per


def _forward(spec, layers, lanes, logits, attended, history):
    """(bytes, flops) of `lanes` lanes through `layers` layers; `logits` lanes go through the lm_head; `attended` tokens are
    attended by the lanes in all, `history` tokens of KV are read."""
    dense, expert, per = _layer(spec)
    touched = min(spec.experts, lanes * spec.experts_per_token)
    bytes_ = layers * (per * (dense + touched * expert) + 4 * spec.kv_heads * spec.head_dim * history)
    flops = layers * (2 * lanes * (dense + spec.experts_per_token * expert) + 4 * spec.q_heads * spec.head_dim * attended)
    if logits:
        bytes_ += 2 * spec.vocab * spec.hidden + 4 * logits * spec.vocab
        flops += 2 * logits * spec.vocab * spec.hidden
    return bytes_, flops


def work(case):
    if case["model"] == "linear":
        lanes, n, k = case["lanes"], case["n"], case["k"]
        return {"bytes": n * (k / 2 + 2 * k / 128) + 2 * lanes * (n + k), "flops": 2 * lanes * n * k}
    spec = MODELS[case["model"]][0]
    streams, context, question, answer, drafts = (case[key] for key in ("streams", "context", "question", "answer", "drafts"))
    parts = []

    def draft(lanes, logits, attended, history):
        bytes_, flops = _forward(spec, 1, lanes, logits, attended, history)
        adapter = 2 * spec.hidden * spec.hidden
        parts.append((bytes_ + 2 * adapter, flops + 2 * lanes * adapter))

    # the questions: every stream's in one pass over the weights
    lanes, attended, history = streams * question, streams * question * (context + (question + 1) / 2), context + streams * question
    parts.append(_forward(spec, spec.layers, lanes, streams, attended, history))
    draft(lanes, 0, attended, history)
    # the answer: cycles of drafts, one verify of drafts + 1 lanes per stream and the MTP layer's own state steps
    per_cycle = sum(EASY ** i for i in range(drafts + 1))
    cycles = math.ceil((answer - 1) / per_cycle)
    history = context + streams * (question + answer / 2)
    for _ in range(cycles):
        for _ in range(drafts):
            draft(streams, streams, streams * (context + question + answer / 2), history)
        lanes = streams * (drafts + 1)
        attended = lanes * (context + question + answer / 2)
        parts.append(_forward(spec, spec.layers, lanes, lanes, attended, history))
        draft(lanes, 0, attended, history)
    # the logits of one more token
    history = context + question + answer
    parts.append(_forward(spec, spec.layers, 1, 1, history, history))
    return {"bytes": sum(b for b, _ in parts), "flops": sum(f for _, f in parts)}


def _cost(case):
    needed = work(case)
    return needed["bytes"] / 6.0e12 + needed["flops"] / 1.0e15


def tolerance(case):
    if case["model"] == "linear":
        return {"rel": 3e-3, "max": 0.03}  # one f32 sum rounded to bf16 once
    # Logits behind a bf16 residual stream of 64 (8b) additions, each rounded by up to 2^-9 of its value: two orders of
    # the f32 sums that are both right part by 1.5 % to 1.7 %.  A route of moe that turns on a near-tie weighs as much.
    # The tokens win by wide margins.
    return {"rel": 1e-2 if case["model"] == "tiny" else 2.5e-2, "max": 0.3, "differ": 0.0}


# ---- packages


def _bf16(values):
    return values.to(torch.bfloat16).view(torch.int16).cpu().numpy().view(np.uint16)


def _vocabulary(spec, scale):
    """embedding, lm_head and MTP adapter (see the module's docstring)."""
    generator = torch.Generator(device="cuda")
    generator.manual_seed(1000 + spec.seed)
    h = spec.hidden
    v = torch.randn((spec.vocab, h), generator=generator, device="cuda") * math.sqrt(2.0)
    easy = torch.rand((spec.vocab, 1), generator=generator, device="cuda") < EASY
    first = torch.arange(h, device="cuda")[None, :] < h // 2
    v *= easy == first
    embedding = _bf16(v * scale)
    lm_head = torch.empty_like(v)
    lm_head[torch.randperm(spec.vocab, generator=generator, device="cuda")] = v * 0.02
    adapter = torch.randn((h, 2 * h), generator=generator, device="cuda") * 0.02
    adapter[:, :h] = torch.diag(4.0 * first[0].float())
    return {"model.embed_tokens.weight": embedding, "lm_head.weight": _bf16(lm_head), "mtp.fc.weight": _bf16(adapter)}


def _sparse_expert_tensors(spec):
    """The FP8 sparse-expert layers, experts packed [expert, row, column]; weights quantised per 128x128 block."""
    generator = torch.Generator(device="cuda")
    generator.manual_seed(spec.seed)

    def normal(*shape):
        return torch.randn(shape, generator=generator, device="cuda") * spec.std

    def fp8(name, scale_name, *shape):
        w = normal(*shape)
        tiles = w.view(*shape[:-2], shape[-2] // 128, 128, shape[-1] // 128, 128)
        scale = (tiles.abs().amax(dim=(-3, -1)) / 448.0).to(torch.bfloat16)
        quantised = (tiles / scale.float()[..., :, None, :, None]).clamp(-448, 448).to(torch.float8_e4m3fn).view(torch.uint8)
        yield name, "F8_E4M3", shape, quantised.reshape(shape).cpu().numpy()
        yield scale_name, "BF16", tuple(scale.shape), scale.view(torch.int16).cpu().numpy().view(np.uint16)

    def bf16(name, values):
        return name, "BF16", tuple(values.shape), _bf16(values)

    h = spec.hidden
    for name in ("model.embed_tokens.weight", "lm_head.weight", "mtp.fc.weight"):
        yield name, "BF16", ((h, 2 * h) if name == "mtp.fc.weight" else (spec.vocab, h)), None
    for name in ("model.norm", "mtp.norm", "mtp.pre_fc_norm_embedding", "mtp.pre_fc_norm_hidden"):
        yield bf16(name + ".weight", torch.ones(h))
    for prefix in [f"model.layers.{i}" for i in range(spec.layers)] + ["mtp.layers.0"]:
        for name, width in (("input_layernorm", h), ("post_attention_layernorm", h), ("self_attn.q_norm", spec.head_dim), ("self_attn.k_norm", spec.head_dim)):
            yield bf16(f"{prefix}.{name}.weight", torch.ones(width))
        q, kv = spec.q_heads * spec.head_dim, spec.kv_heads * spec.head_dim
        for name, n, k in (("q_proj", q, h), ("k_proj", kv, h), ("v_proj", kv, h), ("o_proj", h, q)):
            base = f"{prefix}.self_attn.{name}.weight"
            yield from fp8(base, base + "_scale_inv", n, k)
        yield bf16(f"{prefix}.mlp.gate.weight", torch.randn((spec.experts, h), generator=generator, device="cuda") * 0.06)
        base = f"{prefix}.mlp.experts."
        yield from fp8(base + "gate_up_proj", base + "gate_up_proj_scale_inv", spec.experts, 2 * spec.moe_ffn, h)
        yield from fp8(base + "down_proj", base + "down_proj_scale_inv", spec.experts, h, spec.moe_ffn)


def _package_directory(spec, scale):
    """Writes the package once per machine (the 8B one is about 6 GB)."""
    directory = Path(tempfile.gettempdir()) / f"nerve_b200_perf_{os.getuid()}" / spec.name
    if (directory / "vulkan_resident_package.json").exists():
        return directory
    staging = directory.with_name(f"{spec.name}.tmp{os.getpid()}")
    shutil.rmtree(staging, ignore_errors=True)
    own = _vocabulary(spec, scale)
    tensors = _sparse_expert_tensors(spec) if spec.experts else iter_checkpoint_torch(spec, "cuda")
    write_package(spec, staging, tensors=((name, dtype, shape, own.get(name, data)) for name, dtype, shape, data in tensors), hash_tensors=False)
    try:
        staging.rename(directory)
    except OSError:
        shutil.rmtree(staging, ignore_errors=True)  # another process was first
    return directory


_engines = {}
_ids = itertools.count(1)


def _engine(model):
    """The mounted model and its engine, which a program keeps for all its conversations."""
    if model not in _engines:
        spec, scale, options, chunk = MODELS[model]
        engine = nb.Engine(nb.Package(_package_directory(spec, scale), verify_level=0, **options))
        engine.set_prefill_chunk(chunk)
        torch.cuda.empty_cache()
        _engines[model] = engine
    return _engines[model]


class _Conversation:
    """A context in the KV cache (a stream of its own) and the questions that will be asked about it."""

    def __init__(self, case, seed):
        self.case, self.seed, self.engine, self.base = case, seed, _engine(case["model"]), None
        vocab = MODELS[case["model"]][0].vocab
        rng = np.random.default_rng(seed)
        self.questions = [[int(t) for t in rng.integers(0, vocab, size=case["question"])] for _ in range(case["streams"])]
        if case["context"]:
            self.base = next(_ids)
            self.engine.add_stream(self.base, **self._stream_options())
            self.engine.submit_input_event_until_idle(self.base, [int(t) for t in rng.integers(0, vocab, size=case["context"])], 0)

    def _stream_options(self):
        sampler = {"method": 1, "temperature": 0.8, "top_p": 0.95, "min_p": 0.0, "top_k": 40} if self.case["sampled"] else None
        return {"seed": self.seed & 0xFFFF, "speculative_draft_tokens": self.case["drafts"], "sampler": sampler}

    def turn(self):
        ids = []
        for question in self.questions:
            stream = next(_ids)
            if self.base is None:
                self.engine.add_stream(stream, **self._stream_options())
            else:
                self.engine.fork_stream(self.base, stream, seed=(self.seed + len(ids)) & 0xFFFF)
            self.engine.enqueue_input_event(stream, question, self.case["answer"])
            ids.append(stream)
        outputs, _ = self.engine.run_until_idle()
        answers = {stream: [] for stream in ids}
        for stream, token, _, _ in outputs:
            answers[stream].append(token)
        logits, _ = self.engine.debug_target_logits(ids[-1], answers[ids[-1]][-1:])
        for stream in ids:
            self.engine.remove_stream(stream)
        return {"tokens": np.array([answers[stream] for stream in ids], dtype=np.int64), "logits": logits}

    def __del__(self):
        if self.base is not None:
            self.engine.remove_stream(self.base)


class _Linear:
    """One INT4 g128 matrix, activations and an output buffer on the device."""

    def __init__(self, case, seed):
        generator = torch.Generator(device="cuda")
        generator.manual_seed(seed)
        self.lanes, self.n, self.k = case["lanes"], case["n"], case["k"]
        self.x = torch.randn((self.lanes, self.k), generator=generator, device="cuda").to(torch.bfloat16)
        # four-bit values of a normal distribution cut at 3 sigma, eight to a word; scales as absmax / 7 of such a group
        normal = torch.randn((self.n, self.k // 8), generator=generator, device="cuda")
        self.weight = torch.zeros((self.n, self.k // 8), dtype=torch.int32, device="cuda")
        for nibble in range(8):
            self.weight |= ((normal.normal_(generator=generator) * 2.33).round().clamp(-8, 7).to(torch.int32) + 8) << (4 * nibble)
        self.scales = (torch.rand((self.n, self.k // 128), generator=generator, device="cuda") * 0.004 + 0.006).to(torch.bfloat16)
        self.y = torch.empty((self.lanes, self.n), dtype=torch.bfloat16, device="cuda")

    def turn(self):
        pointer = lambda tensor: ctypes.c_void_p(tensor.data_ptr())  # noqa: E731
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        status = nb.library().nerve_b200_op_linear_int4(pointer(self.x), pointer(self.weight), pointer(self.scales), pointer(self.y), None,
                                                        self.lanes, self.n, self.k, 128, stream)
        if status != 0:
            raise RuntimeError(nb.library().nerve_b200_last_error().decode())
        return self.y


def prepare(case, seed):
    return _Linear(case, seed) if case["model"] == "linear" else _Conversation(case, seed)


def run(state):
    return state.turn()
