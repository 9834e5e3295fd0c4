"""The matrix steps of the persistent decode stack kernel against 64-bit arithmetic, one step at a time.

A layer is made so that one of its steps has inputs that are known exactly and outputs that can be read:

* the residual stream is +-1 in its first half and 0 in the second, and the norm's epsilon makes the mean square 1, so a
  normalised row is the norm's weight with the lane's sign;
* every stream has one token, so an attention output is the value projection itself;
* gates of 32 leave SiLU as they are, so a product is 32 times the up projection;
* scales of zero take the steps behind the tested one out of the residual stream, whose second half is then the output.

Row r of the tested matrix has weights only on columns below its own bound of magnitude, so that a large value in a group
does not cover what the small ones of the group add up to.  An output may be off by half a bf16 unit and by 2^-20 of the sum
of its terms' magnitudes (the f32 sums over the groups and the warps: some fifty roundings of 2^-24, and what a tie makes of
them).  A column below 2^-17 may be off by 2^-25, as an fp16 number is, where no value of its group reaches 64."""

import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = Path(__file__).resolve().parent
PAGE = 16


class _Layers(ctypes.Structure):
    _fields_ = ([("words", ctypes.c_void_p * 7), ("scales", ctypes.c_void_p * 7)] +
                [(name, ctypes.c_void_p) for name in ("input_norm", "post_norm", "rope", "hidden", "pool", "attention_out", "table", "positions", "slots")] +
                [(name, ctypes.c_int) for name in ("lanes", "lanes_per_stream", "hidden_width", "q_heads", "kv_heads", "head_width", "ffn", "page_tokens", "pages_per_slot",
                                                   "attended", "layers", "launches")] +
                [(name, ctypes.c_float) for name in ("eps", "norm_offset", "attention_scale", "milliseconds")])


@pytest.fixture(scope="module")
def launch(tmp_path_factory):
    from llmoop_b200 import build

    library = tmp_path_factory.mktemp("stack") / "stack_layers.so"
    kernels = build.BUILD / "kernels_stack.cu.o"  # (a minute's compilation: taken from the build where it is there)
    command = [build._nvcc(), *build.NVCC_FLAGS, "-shared", "-o", str(library), str(HERE / "stack_layers.cu"),
               str(kernels if kernels.exists() else build.CSRC / "kernels_stack.cu")]
    result = subprocess.run(command, capture_output=True, text=True)
    assert result.returncode == 0, result.stderr
    functions = ctypes.CDLL(str(library))
    functions.stack_layers.stream_bytes = functions.stream_bytes
    functions.stream_bytes.restype = ctypes.c_size_t
    return functions.stack_layers


def _bf16(values):
    """float64 to the nearest bf16, as float64 (finite values)."""
    bits = np.asarray(values, dtype=np.float32).view(np.uint32).astype(np.uint64)
    return (((bits + 0x7FFF + ((bits >> 16) & 1)) >> 16) << 16).astype(np.uint32).view(np.float32).astype(np.float64)


class _Layer:
    """Shape, weights (whole numbers -8 .. 7, bf16 scales per 128 columns) and norms of a layer; zeros to begin with."""

    def __init__(self, hidden, q_heads, kv_heads, head, ffn, offset=0.0):
        self.hidden, self.q_heads, self.kv_heads, self.head, self.ffn, self.offset = hidden, q_heads, kv_heads, head, ffn, offset
        rows = {"q": (q_heads * head, hidden), "k": (kv_heads * head, hidden), "v": (kv_heads * head, hidden), "o": (hidden, q_heads * head), "gate": (ffn, hidden),
                "up": (ffn, hidden), "down": (hidden, ffn)}
        self.weight = {name: np.zeros(shape, dtype=np.int64) for name, shape in rows.items()}
        self.scale = {name: np.zeros((n, k // 128)) for name, (n, k) in rows.items()}
        self.norm = {"input": np.ones(hidden) - offset, "post": np.ones(hidden) - offset}
        self.weight["gate"][:, 0], self.scale["gate"][:, 0] = 4, 8.0  # a gate of 32: column 0 is 1 in every lane

    def single(self, name, values, column=None):
        """Row r is values[r] (bf16) times one column: the lane's sign of column r + 1 (or `column`)."""
        rows = np.arange(len(values))
        columns = rows % (self.hidden // 2 - 1) + 1 if column is None else np.full(len(values), column)
        self.weight[name][rows, columns] = 1
        self.scale[name][rows, columns // 128] = values
        return columns

    def product(self, name, x):
        """Sums and sums of magnitudes in 64 bits, for rows x of [lanes, k]."""
        full = self.weight[name] * np.repeat(self.scale[name], 128, axis=1)
        largest = np.repeat(np.abs(x).reshape(len(x), -1, 128).max(-1), 128, axis=1)
        coarse = (np.abs(x) < 2.0**-17) & (largest < 64)  # where a column may be off by 2^-25, as an fp16 number is
        return x @ full.T, (np.abs(x) + 2.0**-5 * coarse) @ np.abs(full).T

    def run(self, launch, hidden, normalised_sum=0.5, positions=None, pool=None, pages=1, attended=1):
        """The residual stream and the value projections; with `pool` (a stream per lane, their pages in turn) the attention
        outputs instead, the lanes at `positions`."""
        import torch

        def device(array, dtype):
            return torch.from_numpy(np.ascontiguousarray(array.astype(dtype))).cuda()

        def bf16(array):
            return torch.from_numpy(np.ascontiguousarray(array, dtype=np.float64)).to(torch.bfloat16).cuda()

        lanes = hidden.shape[0]
        t = _Layers()
        keep = []
        for i, name in enumerate(("q", "k", "v", "o", "gate", "up", "down")):
            n, k = self.weight[name].shape
            nibbles = (self.weight[name] + 8).astype(np.uint32).reshape(n, k // 8, 8)
            keep += [device((nibbles << (4 * np.arange(8, dtype=np.uint32))).sum(-1), np.uint32).view(torch.int32), bf16(self.scale[name])]
            t.words[i], t.scales[i] = keep[-2].data_ptr(), keep[-1].data_ptr()
        named = {"input_norm": bf16(self.norm["input"]), "post_norm": bf16(self.norm["post"]), "rope": torch.full((self.head // 2,), 0x3F80, dtype=torch.int32, device="cuda"),
                 "hidden": bf16(hidden),
                 "pool": torch.zeros((lanes, 2, self.kv_heads, PAGE, self.head), dtype=torch.bfloat16, device="cuda") if pool is None else bf16(pool),
                 "attention_out": torch.zeros((8, self.q_heads * self.head), dtype=torch.bfloat16, device="cuda"),
                 "table": torch.arange(lanes * pages, dtype=torch.int32, device="cuda"),
                 "positions": device(np.zeros(lanes) if positions is None else np.asarray(positions), np.int32),
                 "slots": torch.arange(lanes, dtype=torch.int32, device="cuda")}
        for name, tensor in named.items():
            setattr(t, name, tensor.data_ptr())
        for name, value in (("lanes", lanes), ("lanes_per_stream", 1), ("hidden_width", self.hidden), ("q_heads", self.q_heads), ("kv_heads", self.kv_heads),
                            ("head_width", self.head), ("ffn", self.ffn), ("page_tokens", PAGE), ("pages_per_slot", pages), ("attended", attended), ("layers", 1), ("launches", 1)):
            setattr(t, name, value)
        t.eps, t.norm_offset, t.attention_scale = 1.0 - normalised_sum, self.offset, 1.0
        torch.cuda.synchronize()
        assert launch(ctypes.byref(t)) == 0
        if pool is not None:
            return named["attention_out"][:lanes].double().cpu().numpy()
        values = named["pool"][:, 1, :, 0].reshape(lanes, -1)
        return named["hidden"].double().cpu().numpy(), values.double().cpu().numpy()


def _hidden(rng, lanes, width):
    rows = np.zeros((lanes, width))
    rows[:, : width // 2] = rng.choice([-1.0, 1.0], size=(lanes, width // 2))
    rows[:, 0] = 1.0
    return rows


def _check(got, sums, magnitudes, where):
    unit = np.exp2(np.floor(np.log2(np.maximum(np.abs(sums), 2.0**-100))) - 7)
    excess = np.abs(got - sums) - (0.5 * unit + 2.0**-20 * magnitudes)
    assert np.isfinite(got).all() and excess.max() <= 0, (where, np.unravel_index(excess.argmax(), excess.shape), got.flat[excess.argmax()], sums.flat[excess.argmax()])


def _spread(rng, count, kind):
    """Inputs of a step, in groups that lie far apart: `outlier` has one value of 10^4 among ones of 0.05 in every group, `range`
    magnitudes from 2^-36 to 2^15; in both a group of zeros, one of ordinary values, one of large whole numbers."""
    if kind == "outlier":
        values = rng.normal(size=count) * rng.normal(size=count) * 0.05
        values[::128] = 1e4
    else:
        values = rng.choice([-1.0, 1.0], size=count) * 2.0 ** rng.uniform(-36, 15, size=count)
    values = _bf16(values)
    if count >= 512:
        values[128:256] = _bf16(rng.normal(size=128))
        values[256:384] = 0.0
        values[384:512] = rng.integers(60000, 250000, size=128) // 2048 * 2048
    return values


def _bounded(rng, layer, name, values):
    """Weights of every row on the columns below a bound of its own only."""
    n, k = layer.weight[name].shape
    magnitudes = np.abs(values)
    bounds = rng.choice(magnitudes[magnitudes > 0], size=n)
    layer.weight[name][:] = np.where(magnitudes[None, :] <= bounds[:, None], rng.integers(-8, 8, size=(n, k)), 0)
    layer.scale[name][:] = _bf16(rng.uniform(0.5, 1.0, size=(n, k // 128)))


def _step_case(step, kind, hidden_width=512, offset=0.0, heads=(16, 8, 32)):
    """(layer, hidden rows of eight lanes, what reads the step's outputs from run()'s results, sums, magnitudes)"""
    rng = np.random.default_rng(7)
    layer = _Layer(hidden_width, *heads, 768, offset)
    hidden, half = _hidden(rng, 8, hidden_width), hidden_width // 2
    if step in ("v", "up"):
        values = _spread(rng, hidden_width, kind)
        if offset:  # what the offset leaves of a bf16 weight
            values = _bf16(values - offset) + offset
            values = np.where(_bf16(values) == values, values, 1.0)
        values[0] = 1.0  # (the gates')
        layer.norm["input" if step == "v" else "post"] = values - offset
        _bounded(rng, layer, step, np.where(np.arange(hidden_width) < half, values, 0.0))
        sums, magnitudes = layer.product(step, hidden * values)
        if step == "v":
            return layer, hidden, (lambda out, got: got), sums, magnitudes
        layer.weight["down"][half + np.arange(256), np.arange(256)] = 1
        layer.scale["down"][half : half + 256, :2] = 1.0
        magnitudes += 2.0**-38 * magnitudes.max()  # (down hands them on: 2^-58 of a group's largest is the least its form holds)
        return layer, hidden, (lambda out, got: out[:, half : half + 256] / 32.0), sums[:, :256], magnitudes[:, :256]
    if step == "o":
        q_heads, kv_heads, width = heads
        values = _spread(rng, kv_heads * width, kind)
        columns = layer.single("v", values)
        head = np.arange(q_heads * width) // width // (q_heads // kv_heads) * width + np.arange(q_heads * width) % width  # of the value row, by column of o's input
        inputs = (hidden[:, columns] * values)[:, head]
        _bounded(rng, layer, "o", values[head])
    else:
        values = _spread(rng, 768, kind)
        columns = layer.single("up", values)
        inputs = hidden[:, columns] * values * 32.0
        _bounded(rng, layer, "down", values)
    sums, magnitudes = layer.product(step, inputs)
    return layer, hidden, (lambda out, got: out[:, half:]), sums[:, half:], magnitudes[:, half:]


@pytest.mark.parametrize("kind", ["outlier", "range"])
@pytest.mark.parametrize("step", ["v", "o", "up", "down"])
def test_values_far_apart_in_a_group(launch, step, kind):
    """... at every width, each lane bit for bit as alone."""
    layer, hidden, read, sums, magnitudes = _step_case(step, kind)
    alone = [read(*layer.run(launch, hidden[m : m + 1]))[0] for m in range(8)]
    for lanes in (1, 2, 3, 4, 5, 8):
        got = read(*layer.run(launch, hidden[:lanes]))
        _check(got, sums[:lanes], magnitudes[:lanes], (step, lanes))
        assert np.array_equal(got, np.stack(alone[:lanes])), lanes


def test_values_far_apart_with_a_norm_offset_and_in_windows(launch):
    """A norm that adds one to its weights; rows of 8192 columns, which five lanes and more stage in parts."""
    for hidden_width, offset, widths in ((512, 1.0, (1, 4, 8)), (8192, 0.0, (1, 4, 5, 8))):
        layer, hidden, read, sums, magnitudes = _step_case("v", "outlier", hidden_width, offset)
        for lanes in widths:
            _check(read(*layer.run(launch, hidden[:lanes])), sums[:lanes], magnitudes[:lanes], (hidden_width, lanes))


def test_query_rows_of_more_than_8192_columns(launch):
    """... whole for one lane, in windows of steps from three on."""
    layer, hidden, read, sums, magnitudes = _step_case("o", "range", heads=(72, 9, 128))
    for lanes in (1, 3, 8):
        _check(read(*layer.run(launch, hidden[:lanes])), sums[:lanes], magnitudes[:lanes], lanes)


def test_infinities_and_nans(launch):
    """A lane whose row holds one has no sums in a step that reads it - a NaN, which the rounding to bf16 (no case for NaN, as
    in the shaders) makes -0 -, the others are as without it.  An infinite product gives an infinity where down has a weight."""
    layer, hidden, read, sums, magnitudes = _step_case("v", "outlier")
    expected, others = read(*layer.run(launch, hidden[:6])), [0, 1, 3, 4, 5]
    for value in (np.inf, -np.inf, np.nan):
        rows = hidden[:6].copy()
        rows[2, 5] = value
        got = read(*layer.run(launch, rows))
        assert (np.isnan(got[2]) | (got[2] == 0)).all() and np.array_equal(got[others], expected[others])
    layer, hidden, read, _, _ = _step_case("down", "outlier")
    rows = layer.weight["up"].any(axis=1).nonzero()[0]
    infinite, column = rows[-3], layer.weight["up"][rows[-3]].nonzero()[0][0]
    layer.scale["up"][infinite] = 2.0**126  # times 32
    weights = layer.weight["down"][layer.hidden // 2 :, infinite]
    weights[:] = np.arange(len(weights)) % 16 - 8
    for lanes in (1, 3, 8):
        got = read(*layer.run(launch, hidden[:lanes]))
        signs = np.sign(hidden[:lanes, column])[:, None] * np.sign(weights)[None]
        assert np.array_equal(got, np.where(signs == 0, 0.0, np.where(signs > 0, np.inf, -np.inf))), lanes


def test_a_group_at_the_end_of_a_row_keeps_its_own_scale(launch):
    """Rows of an odd number of groups (384 columns, heads of 32): a warp has one group and threads beyond the row.  The first
    chunk of the row is a million times as large as the last group."""
    rng = np.random.default_rng(1)
    layer = _Layer(512, 12, 6, 32, 256)
    values = np.where(np.arange(192) < 4, 2.0**12, _bf16(rng.uniform(2.0**-8, 2.0**-4, size=192)))
    hidden = _hidden(rng, 4, 512)
    columns = layer.single("v", values)
    head = np.arange(384) // 32 // 2 * 32 + np.arange(384) % 32  # of the value row, by column of o's input
    inputs = (hidden[:, columns] * values)[:, head]
    layer.weight["o"][:] = rng.integers(-8, 8, size=(512, 384))
    layer.weight["o"][:, :256] = 0
    layer.scale["o"][:] = _bf16(rng.uniform(0.5, 1.0, size=(512, 3)))
    out, got = layer.run(launch, hidden)
    assert np.array_equal(got, hidden[:, columns] * values)
    sums, magnitudes = layer.product("o", inputs)
    _check(out[:, 256:], sums[:, 256:], magnitudes[:, 256:], "o")


def test_work_items_without_tokens_between_others(launch):
    """Eight streams of uneven contexts: splits are laid out for the longest, so teams meet items without tokens between ones
    that have some.  Bar: half a bf16 unit and, for probabilities in f32 that are handed on in two bf16 parts (2^-17 each),
    2^-15 of the magnitudes."""
    import torch

    rng = np.random.default_rng(2)
    positions, splits = [1099, 69, 1203, 19, 499, 1150, 129, 1023], 32
    layer = _Layer(512, 16, 8, 32, 256)
    counts = [[max(0, min(64, position + 1 - 64 * split)) for split in range(splits)] for position in positions]
    ctas, reached = torch.cuda.get_device_properties(0).multi_processor_count, 0
    for team in range(4 * ctas):
        present = [counts[item // 8 // splits][item // 8 % splits] > 0 for item in range(team, 8 * splits * 8, 4 * ctas)]  # (kv heads innermost)
        reached += any(present[a] and not present[b] and present[c] for c in range(len(present)) for b in range(c) for a in range(b))
    assert reached > 20
    hidden = _hidden(rng, 8, 512)
    values = _bf16(rng.uniform(0.5, 2.0, size=512))
    columns = layer.single("q", values)
    pages = splits * 64 // PAGE
    pool = _bf16(rng.normal(size=(8 * pages, 2, 8, PAGE, 32)))
    expected, magnitude = np.zeros((8, 16, 32)), np.zeros((8, 16, 32))
    for m, position in enumerate(positions):
        rows = pool[m * pages : (m + 1) * pages].transpose(1, 2, 0, 3, 4).reshape(2, 8, -1, 32)[:, :, : position + 1].copy()
        rows[:, :, position] = 0.0  # what this layer appends
        q = (hidden[m, columns] * values).reshape(16, 32)
        for head in range(16):
            scores = rows[0, head // 2] @ q[head]
            p = np.exp(scores - scores.max())
            expected[m, head], magnitude[m, head] = p / p.sum() @ rows[1, head // 2], p / p.sum() @ np.abs(rows[1, head // 2])
    got = layer.run(launch, hidden, positions=positions, pool=pool, pages=pages, attended=64 * splits)
    _check(got, expected.reshape(8, -1), 32.0 * magnitude.reshape(8, -1), "attention")


def test_streams_of_a_short_k_are_not_padded(launch):
    """A block of 16 x 128 nibbles and its scales is 1056 bytes; a group count that is a power of two leaves no step ragged."""
    for k in (128, 256, 512, 1024, 2048, 4096):
        for rows, pair in ((512, 0), (4096, 0), (1024, 1), (14336, 1)):
            assert launch.stream_bytes(rows, k, pair) == (1 + pair) * rows // 16 * (k // 128) * 1056, (rows, k, pair)
    assert launch.stream_bytes(1152, 9 * 128, 0) <= 1152 // 16 * 16 * 1056
