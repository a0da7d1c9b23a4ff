"""How the one-kernel decode step divides a layer's products: every weight row and column by exactly one warp, within the
matrices and within shared memory, over shapes with odd and even chunk counts, groups of one to eight and one to eight
tokens."""
import ctypes
import weakref

import pytest
import torch

SHAPES = {
    "0.5b": (896, 14, 2, 64, 4864), "1.5b": (1536, 12, 2, 128, 8960), "7b": (3584, 28, 4, 128, 18944),
    "one_chunk": (64, 2, 1, 64, 64), "odd": (192, 3, 3, 64, 576), "wide_ff": (256, 8, 1, 64, 16384), "group7": (896, 7, 1, 128, 2432),
}
UNPACED = ("1.5b", "7b")  # layers of many rings of weights: their copies are asked for behind the barriers and inside the products
WARPS, LIMIT, MAX_TILES = 16, 232448, 64


def plan(tokens, shape, ctas):
    from alofa_b200.csrc import ops

    out = (ctypes.c_int * 23)()
    taken = ops._decode_stack().alofa_decode_stack_plan(tokens, *shape, ctas, out)
    return bool(taken), list(out)


def share(phase, tiles, slices, kg, rg, cta, ctas):
    """(tiles, slices) of a CTA, as the kernel deals them."""
    if kg == 0:
        c = ctas - 1 - cta if phase == 2 else cta
        return list(range(c, tiles, ctas)), list(range(slices))
    if cta >= kg * rg:
        return [], []
    k, g = cta % kg, cta // kg
    return list(range(g * tiles // rg, (g + 1) * tiles // rg)), list(range(k * slices // kg, (k + 1) * slices // kg))


@pytest.mark.parametrize("name", list(SHAPES))
@pytest.mark.parametrize("tokens", [1, 3, 4, 7, 8])
@pytest.mark.parametrize("ctas", [148, 132])
def test_products_are_covered_once(name, tokens, ctas):
    hidden, heads, kv_heads, hd, inter = SHAPES[name]
    taken, p = plan(tokens, SHAPES[name], ctas)
    if not taken:
        assert name == "7b" and tokens > 4, "only wide operands of many tokens leave no room"
        return
    chunks, slots, x_stride, x_bytes, work_bytes, smem = p[16:22]
    paced = p[22]
    assert paced == (name not in UNPACED)
    assert slots >= 2 and smem <= LIMIT and x_bytes >= tokens * x_stride
    sizes = [((heads + 2 * kv_heads) * hd, hidden), (hidden, heads * hd), (2 * inter, hidden), (hidden, inter)]
    for phase, (rows, cols) in enumerate(sizes):
        tiles, slices, kg, rg = p[4 * phase : 4 * phase + 4]
        assert slices * chunks * 64 == cols and tiles * 16 == rows
        seen, covered = set(), set()
        for cta in range(ctas):
            own, part = share(phase, tiles, slices, kg, rg, cta, ctas)
            if not own or not part:
                continue
            assert len(own) <= MAX_TILES and 2 * len(part) * chunks * 64 + 16 <= x_stride
            pieces = [(t, s) for t in own for s in part]
            warps = min(WARPS, len(pieces))
            entries = []
            for w in range(warps):
                for u in range(w * len(pieces) // warps, (w + 1) * len(pieces) // warps):
                    assert (warps * (u + 1) - 1) // len(pieces) == w  # how an epilogue finds the warps of a tile
                    entry = w + u // len(part)
                    if (w, u // len(part)) not in entries:
                        entries.append((w, u // len(part)))
                    assert (entry + 1) * 16 * 8 * 4 + x_bytes <= work_bytes
            assert len({w + t for w, t in entries}) == len(entries)
            assert not seen & set(pieces)
            seen |= set(pieces)
            for t in own:  # two groups of eight rows: halves of a rotated head, gate and up, or neighbours
                if phase == 0:
                    first, second = t // (hd // 16) * hd + t % (hd // 16) * 8, hd // 2
                else:
                    first, second = (8 * t, inter) if phase == 2 else (16 * t, 8)
                covered |= set(range(first, first + 8)) | set(range(first + second, first + second + 8))
        assert len(seen) == tiles * slices and covered == set(range(rows))


@pytest.fixture
def small():
    """A bfloat16 model of the kernel's form on the CPU, not loaded, weights for it, and what looks at it."""
    from alofa_b200.engine.step import StepRunner
    from alofa_b200.models.qwen2 import Qwen2Config, build_spec
    from alofa_b200.parts.base import Runtime
    from alofa_b200.parts.decode_stack import DecodeStack
    from alofa_b200.parts.model import Model
    from alofa_b200.weights.loader import load_state
    from alofa_b200.weights.random_init import random_state

    rt = Runtime(torch.device("cpu"), torch.bfloat16)
    model = Model(build_spec(Qwen2Config(2, 192, 3, 3, 64, 576, 300, 1e-6, 1e4, True, 4096)), rt)
    runner = StepRunner(model, block_size=64, num_pages=4, max_requests=2, max_tokens=128, max_step_tokens=32)
    state = lambda seed: load_state(model.tensors(), random_state(model.tensors(), seed, torch.bfloat16, "cpu"), rt.dtype, rt.device)  # noqa: E731
    return model, state, DecodeStack(model, runner.storage.caches, 64)


def test_a_model_may_be_loaded_after_its_runner_was_made(small):
    model, state, stack = small
    assert stack.look() is None
    model.load(state(1))
    form = stack.look()
    assert form.sizes == (192, 3, 3, 64, 576) and len(form.layers) == 2 and form == stack.look()


def test_a_model_loaded_again_is_described_again_and_its_old_weights_go(small):
    model, state, stack = small
    model.load(state(1))
    stack.form = first = stack.look()
    old = [weakref.ref(block.mixer.out.weight) for block in model.layers] + [weakref.ref(model.layers[0].mixer.position.rotary_table()[0])]
    again = state(2)  # beside the old ones: other addresses
    model.load(again)
    assert stack.look() != first and model.loads == 2
    assert [ref() for ref in old] == [None] * len(old)


def unaligned(t):
    room = torch.empty(t.numel() + 1, dtype=t.dtype)
    room[1:] = t.flatten()
    return room[1:].view(t.shape)


@pytest.mark.parametrize("what", ["alignment", "type", "bias", "vector", "eps", "mixer", "window"])
def test_what_the_kernel_does_not_have_goes_layer_by_layer(small, what):
    """Looked at anew at every step: what changed behind the runner's back is refused, not run wrongly or raised at."""
    from alofa_b200.parts.linear import RESIDUAL, Linear

    model, state, stack = small
    model.load(state(1))
    form, block = stack.look(), model.layers[1]
    weight = block.mixer.out.weight
    if what == "alignment":
        block.mixer.out = Linear(unaligned(weight), None, RESIDUAL)
    elif what == "type":
        block.mixer.out = Linear(weight.float(), None, RESIDUAL)
    elif what == "bias":
        block.mixer.out = Linear(weight, torch.ones(192), RESIDUAL)
    elif what == "vector":
        block.mixer_norm.weight = unaligned(block.mixer_norm.weight)
    elif what == "mixer":
        block.mixer = type("Other", (type(block.mixer),), {})(block.mixer.spec, model.rt)
    elif what == "window":
        block.mixer.window = 64
    else:
        block.mixer_norm.eps = 1e-3
        assert stack.look() is not None and stack.look() != form
        return
    assert stack.look() is None


BAD = [(0, 896, 14, 2, 64, 4864), (9, 896, 14, 2, 64, 4864), (1, 0, 14, 2, 64, 4864), (1, 896, 14, 0, 64, 4864), (1, 896, 0, 2, 64, 4864), (1, 896, 14, 4, 64, 4864), (1, 896, 18, 2, 64, 4864),
       (1, 896, 14, 2, 96, 4864), (1, 896, 14, 2, 0, 4864), (1, 900, 14, 2, 64, 4864), (1, 896, 14, 2, 64, 0), (1, 896, 14, 2, 64, 4800 + 32), (1, 1 << 30, 14, 2, 64, 4864), (1, 896, 14, 2, 64, 1 << 30)]


@pytest.mark.parametrize("sizes", BAD)
def test_entries_refuse_sizes_without_a_look_at_the_device(sizes):
    from alofa_b200.csrc import ops

    lib, out = ops._decode_stack(), (ctypes.c_int * 23)()
    tokens, hidden, heads, kv_heads, hd, inter = sizes
    assert lib.alofa_decode_stack_plan(*sizes, 148, out) == 0 and not any(out)
    assert lib.alofa_decode_stack_ctas(*sizes, 64) == 0
    if tokens == 1:
        assert lib.alofa_decode_stack_layer(*[16] * 7, None, 16, 16, 1e-6, 1e-6, *sizes[1:]) == 1
    assert lib.alofa_decode_stack(16, 1, 148, tokens, hidden, heads, kv_heads, hd, inter, 64, 1, 1.0, *[16] * 15, None) == 1


def test_entries_refuse_pages_grids_and_tables():
    from alofa_b200.csrc import ops

    lib, out, good = ops._decode_stack(), (ctypes.c_int * 23)(), (8, 896, 14, 2, 64, 4864)
    assert lib.alofa_decode_stack_plan(*good, 148, out) == 1 and lib.alofa_decode_stack_plan(*good, 0, out) == 0
    for page in (0, 8, 24):
        assert lib.alofa_decode_stack_ctas(*good, page) == 0
    for layers, ctas, page, stride in ((0, 148, 64, 1), (1, 0, 64, 1), (1, 15, 64, 1), (1, 148, 0, 1), (1, 148, 24, 1), (1, 148, 64, 0)):
        assert lib.alofa_decode_stack(16, layers, ctas, *good, page, stride, 1.0, *[16] * 15, None) == 1
    assert lib.alofa_decode_stack_layer(16, None, *[16] * 5, None, 16, 16, 1e-6, 1e-6, *good[1:]) == 1


def kernel_split(lengths, kv_heads, ctas):
    """Granules a split has at most, as the kernel looks for it: all candidates from the smallest on."""
    granules = [n // 16 if n % 16 == 0 else n // 16 + 1 for n in lengths]
    per = max(16, (sum(granules) * kv_heads + ctas - 1) // ctas)
    while sum((g + per - 1) // per for g in granules) * kv_heads > ctas:
        per += 1
    return per, sum(granules) * kv_heads / ctas


@pytest.mark.parametrize("kv_heads", [1, 2, 4, 8, 16])
@pytest.mark.parametrize("most", [32, 64])
def test_long_or_uneven_keys_go_layer_by_layer(kv_heads, most):
    import random

    from alofa_b200.parts.decode_stack import keys_per_cta_fit

    rng = random.Random(kv_heads)
    seen = set()
    for _ in range(400):
        lengths = [rng.choice([1, 16, 17, 256, 257, int(2 ** rng.uniform(0, 17))]) for _ in range(rng.randint(1, 8))]
        per, even = kernel_split(lengths, kv_heads, 148)
        want = per == 16 or (per <= most and per <= 1.25 * even)
        assert keys_per_cta_fit(lengths, kv_heads, 148, most) == want, lengths
        seen.add(want)
    assert len(seen) == 2


def test_lengths_on_either_side_of_the_rule():
    from alofa_b200.parts.decode_stack import keys_per_cta_fit

    assert keys_per_cta_fit([2049] * 8, 2, 148, 32) and keys_per_cta_fit([4096] * 8, 2, 148, 32) and not keys_per_cta_fit([8192] * 8, 2, 148, 32)
    assert keys_per_cta_fit([32768], 2, 148, 32) and keys_per_cta_fit([32768] + [64] * 7, 2, 148, 32) and not keys_per_cta_fit([32768] * 4, 2, 148, 32)
    assert keys_per_cta_fit([8192] * 4, 4, 148, 64) and not keys_per_cta_fit([32768] * 4, 4, 148, 64)
    assert keys_per_cta_fit([512] * 8, 16, 148, 32) and not keys_per_cta_fit([512] * 5, 16, 148, 32) and not keys_per_cta_fit([32768] + [64] * 7, 16, 148, 32)
    assert keys_per_cta_fit([256] * 8, 16, 148, 32) and not keys_per_cta_fit([4096] * 8, 16, 148, 32)
