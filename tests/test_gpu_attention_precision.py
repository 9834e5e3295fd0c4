"""The attention kernels of the kernel-per-operator path against 64-bit arithmetic, launch by launch: the tiled form (16, 32
and 128 query rows) and the scalar f32 form of layers that feed FP8, heads of 64 and 128, 1 to 8 query heads per KV head,
several streams with equal and with different numbers of lanes, a ring that has wrapped.

The f32 partials of the splits, merged in 64 bits, must come within 2^-20 of the output's 2-norm.  A probability enters with
its 24 bits and a tile's sums join by f32 multiply-adds, so the relative error of an output is a few 2^-24 (f32 sums of
1024 tokens in order: 2^-20.7); probabilities of 16 bits leave 2^-19.2 and more.  The bf16 outputs must come within
half a unit of the last place, and what f32 leaves at a tie, of the reference."""

import ctypes
import math
import subprocess
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

HERE = Path(__file__).resolve().parent
PAGE = 16


@pytest.fixture(scope="module")
def launch(tmp_path_factory):
    library = tmp_path_factory.mktemp("attention") / "attention_partials.so"
    command = ["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC,-fvisibility=hidden", "-shared",
               "-o", str(library), str(HERE / "attention_partials.cu")]
    result = subprocess.run(command, capture_output=True, text=True)
    assert result.returncode == 0, result.stderr
    return ctypes.CDLL(str(library)).attention_partials


def _reference(q, pool, positions, slots, scale, capacity):
    """softmax(q K) V of every lane over the ticks (position - capacity, position] of its stream's ring, in 64 bits."""
    import torch

    lanes, q_heads, _ = q.shape
    pages, kv_heads = capacity // PAGE, pool.shape[2]
    out = torch.empty(q.shape, dtype=torch.float64, device="cuda")
    for lane in range(lanes):
        position, slot = int(positions[lane]), int(slots[lane])
        ring = torch.arange(max(0, position + 1 - capacity), position + 1, device="cuda") % capacity
        own = pool[slot * pages : (slot + 1) * pages].double()
        keys, values = (own[:, half].permute(1, 0, 2, 3).reshape(kv_heads, capacity, -1)[:, ring] for half in (0, 1))
        query = q[lane].double().view(kv_heads, q_heads // kv_heads, -1)
        out[lane] = (torch.softmax(query @ keys.transpose(1, 2) * scale, -1) @ values).reshape(q_heads, -1)
    return out


# lanes of each stream, tokens in front of them (None: the ring has wrapped), tokens per split
CASES = [([1], 0, 128), ([4, 4, 4], 60, 128), ([5, 5], 700, 128), ([24], 1000, 128), ([9], 2040, 512), ([130], 70, 256), ([129], 1900, 1024), ([1, 1], None, 128),
         ([3, 17, 1, 40], 33, 64), ([7, 200], 120, 128)]


@pytest.mark.parametrize("scalar", [False, True], ids=["tiled", "scalar_f32"])
@pytest.mark.parametrize("head", [64, 128])
@pytest.mark.parametrize("group", [1, 2, 4, 8])
def test_partials_against_64_bits(launch, head, group, scalar):
    import torch

    p = lambda tensor: ctypes.c_void_p(tensor.data_ptr())  # noqa: E731
    generator = torch.Generator(device="cuda")
    generator.manual_seed(head * group)
    kv_heads = 2
    q_heads, scale = kv_heads * group, 1.0 / math.sqrt(head)
    for lanes_of, context, split in CASES:
        wrapped, lanes, widest, streams = context is None, sum(lanes_of), max(lanes_of), len(lanes_of)
        context = 777 if wrapped else context
        capacity = 512 if wrapped else (context + widest + PAGE - 1) // PAGE * PAGE
        pages = capacity // PAGE
        pool = torch.randn((streams * pages, 2, kv_heads, PAGE, head), generator=generator, device="cuda").to(torch.bfloat16)
        q = torch.randn((lanes, q_heads, head), generator=generator, device="cuda").to(torch.bfloat16)
        table = torch.arange(streams * pages, dtype=torch.int32, device="cuda")
        positions = torch.tensor([context + i for n in lanes_of for i in range(n)], dtype=torch.int32, device="cuda")
        slots = torch.tensor([s for s, n in enumerate(lanes_of) for _ in range(n)], dtype=torch.int32, device="cuda")
        splits = (min(context + widest, capacity) + split - 1) // split
        scratch = torch.zeros((lanes, q_heads, splits, head + 2), dtype=torch.float32, device="cuda")
        out = torch.zeros((lanes, q_heads, head), dtype=torch.bfloat16, device="cuda")
        ragged = (ctypes.c_int * streams)(*lanes_of)
        status = launch(p(q), p(out), p(pool), p(table), p(positions), p(slots), lanes, widest, q_heads, kv_heads, head, PAGE, pages, ctypes.c_float(scale), split,
                        splits, p(scratch), int(scalar), ragged, streams if len(set(lanes_of)) > 1 else 0)
        assert status == 0
        want = _reference(q, pool, positions, slots, scale, capacity)
        case = (lanes_of, context, split)
        if splits > 1 or scalar:
            partial = scratch.double()
            maximum, total = partial[..., head], partial[..., head + 1]
            weight = torch.where(total > 0, torch.exp(maximum - torch.where(total > 0, maximum, -math.inf).amax(-1, keepdim=True)), 0.0)
            merged = (weight[..., None] * partial[..., :head]).sum(-2) / (weight * total).sum(-1, keepdim=True)
            assert ((merged - want).norm() / want.norm()).item() <= 2.0**-20, case
        ulp = torch.exp2(torch.floor(torch.log2(want.abs().clamp_min(2.0**-100))) - 7)
        slack = 0.5 * ulp + 2.0**-18 * want.pow(2).mean().sqrt()
        assert bool(((out.double() - want).abs() <= slack).all()), case
