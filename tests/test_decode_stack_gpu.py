"""All layers of a small decode step in one kernel, against float64 and against the same step layer by layer.

Sizes go to the edges of what the kernel divides: one token to eight, heads of 64
and 128 in groups of one to eight, widths with an odd and an even number of 64-column chunks, a tile a CTA and several;
contexts of one key, on either side of a page and of a granule of sixteen keys, and of several splits."""
import numpy as np
import pytest
import torch

import plain_qwen2 as plain

pytestmark = pytest.mark.gpu

# layers, hidden, heads, kv heads, head size, inter
SHAPES = {
    "h64_odd": (2, 192, 3, 3, 64, 576),  # chunks of 64 columns, one head a group
    "h64_even": (3, 256, 4, 2, 64, 640),
    "h64_group8": (2, 512, 8, 1, 64, 2560),
    "h128": (2, 384, 3, 1, 128, 640),
    "h128_group7": (2, 896, 7, 1, 128, 2432),
}


@pytest.fixture(scope="module")
def folders(tmp_path_factory):
    from alofa_b200.models.qwen2 import NAME, Qwen2Config
    from alofa_b200.weights.random_init import write_random_model

    base = tmp_path_factory.mktemp("decode_stack_models")
    out = {}
    for i, (name, (n, h, nh, nkv, hd, f)) in enumerate(SHAPES.items()):
        out[name] = write_random_model(base / name, NAME, Qwen2Config(n, h, nh, nkv, hd, f, 300, 1e-6, 1e4, True, 4096), 40 + i, torch.bfloat16)
    return out


def decode(folder, contexts, steps, stacked, graphs=True, page=64):
    """Logits of ``steps`` decode steps behind prompts of the given lengths, and whether the one kernel ran."""
    from alofa_b200.csrc import ops
    from alofa_b200.engine.loading import load_model
    from alofa_b200.engine.step import StepEntry, StepRunner

    model, _, _ = load_model(folder, "bfloat16")
    runner = StepRunner(model, block_size=page, num_pages=sum((c + steps) // page + 1 for c in contexts) + 2, max_requests=len(contexts), max_tokens=4096, max_step_tokens=2048, cuda_graphs=graphs)
    assert runner.decode_stack is not None
    if not stacked:
        runner.decode_stack = None
    rng = np.random.default_rng(5)
    seqs = [[int(t) for t in rng.integers(0, 300, c + steps)] for c in contexts]
    slots = [runner.admit(i) for i in range(len(contexts))]
    for slot, ids, c in zip(slots, seqs, contexts):
        if c:
            for lo in range(0, c, 2048):
                runner.forward([StepEntry(slot, ids[lo : min(c, lo + 2048)])])
    out = []
    for t in range(steps):
        before = ops.launch_count()
        out.append(runner.forward([StepEntry(s, [ids[c + t]], [0]) for s, ids, c in zip(slots, seqs, contexts)]).clone())
        launched = ops.launch_count() - before
    runner.check_status()
    assert runner._stream_acc.abs().sum().item() == 0
    return torch.stack(out), launched, seqs


@pytest.mark.parametrize("name", list(SHAPES))
@pytest.mark.parametrize("contexts", [[0], [1], [63, 15], [16, 64, 17], [0, 127, 300, 1, 640, 255, 256, 257], [3000, 20, 1500, 33, 66, 99, 132]])
def test_matches_layer_by_layer(folders, name, contexts):
    got, launched, _ = decode(folders[name], contexts, 3, True)
    want, more, _ = decode(folders[name], contexts, 3, False)
    assert launched < more, "the step did not run as one kernel"
    # both round the same operands to bfloat16 (2^-9) and differ in the order of fp32 sums alone, so in which way close cases round:
    # both sides, each of the eight roundings a layer 2^-9 / sqrt(3) of its row: sqrt(2 sides * 3 layers * 8) * 2^-9 / sqrt(3) = 2^-7
    assert (got - want).norm() <= 2**-7 * want.norm()
    assert (got - want).abs().max() <= 2**-4 * want.abs().max()


def exact(model, ids, last):
    """Logits of the last tokens of a sequence from the model's own weights, in float64."""
    f = lambda t: t.double()  # noqa: E731
    norm = lambda x, n: x / torch.sqrt((x * x).mean(-1, keepdim=True) + n.eps) * f(n.weight)  # noqa: E731
    x = f(model.embedding.weight[ids])
    n = len(ids)
    for block in model.layers:
        m, ff = block.mixer, block.feed_forward
        y = norm(x, block.mixer_norm) @ f(m.qkv.weight).T + f(m.qkv.bias)
        q, k, v = (t.unflatten(1, (-1, m.hd)) for t in y.split((m.q_dim, m.kv_dim, m.kv_dim), 1))
        cos, sin = f(m.position.rotary_table()[0][:n, None]).unbind(-1)
        turn = lambda t: torch.cat([t[..., : m.hd // 2] * cos - t[..., m.hd // 2 :] * sin, t[..., m.hd // 2 :] * cos + t[..., : m.hd // 2] * sin], -1)  # noqa: B023, E731
        q, k, v = turn(q), turn(k).repeat_interleave(m.nh // m.nkv, 1), v.repeat_interleave(m.nh // m.nkv, 1)
        s = torch.einsum("qhd,khd->hqk", q, k) * m.scale + torch.full((n, n), float("-inf"), dtype=torch.float64, device=x.device).triu(1)
        x = x + torch.einsum("hqk,khd->qhd", s.softmax(-1), v).flatten(1) @ f(m.out.weight).T
        g, u = (norm(x, block.feed_forward_norm) @ f(ff.gate_up.weight).T).chunk(2, 1)
        x = x + (g * torch.sigmoid(g) * u) @ f(ff.down.weight).T
    return norm(x[-last:], model.final_norm) @ f(model.head.linear.weight).T


@pytest.mark.parametrize("sizes, tokens", [((2, 1536, 12, 2, 128, 8960), n) for n in (1, 4, 8)] + [((1, 3584, 28, 4, 128, 18944), n) for n in (1, 4)])
def test_wide_layers(sizes, tokens):
    """Layers of many rings of weights, against float64 beside the same step layer by layer: copies that are asked for behind the barriers and inside the products, a ring that wraps
    several times in one phase, many tiles a CTA."""
    import ctypes

    from alofa_b200.csrc import ops
    from alofa_b200.engine.loading import random_model
    from alofa_b200.engine.step import StepEntry, StepRunner
    from alofa_b200.models.qwen2 import NAME, Qwen2Config

    plan = (ctypes.c_int * 23)()
    assert ops._decode_stack().alofa_decode_stack_plan(tokens, *sizes[1:], 148, plan) == 1 and plan[22] == 0
    model, _, _ = random_model(NAME, Qwen2Config(*sizes, 300, 1e-6, 1e6, True, 4096), 11, generate_on_device=True)
    contexts = [100, 17, 300, 64, 1, 900, 33, 256][:tokens]
    rng = np.random.default_rng(tokens)
    seqs = [[int(t) for t in rng.integers(0, 300, c + 3)] for c in contexts]
    out = []
    for whole, graphs in ((True, True), (True, False), (False, False)):
        runner = StepRunner(model, block_size=64, num_pages=40, max_requests=tokens, max_tokens=1024, max_step_tokens=1024, cuda_graphs=graphs)
        if not whole:
            runner.decode_stack = None
        slots = [runner.admit(i) for i in range(tokens)]
        for slot, ids, c in zip(slots, seqs, contexts):
            runner.forward([StepEntry(slot, ids[:c])])
        rows = []
        for t in range(3):
            before = ops.launch_count()
            rows.append(runner.forward([StepEntry(s, [ids[c + t]], [0]) for s, ids, c in zip(slots, seqs, contexts)]).clone())
        assert graphs or (ops.launch_count() - before <= 5) == whole  # (a recorded step samples too)
        runner.check_status()
        out.append(torch.stack(rows))
    assert torch.equal(out[0], out[1])
    want = torch.stack([exact(model, ids[: c + 3], 3) for ids, c in zip(seqs, contexts)], 1)
    off = [((o.double() - want).norm() / want.norm()).item() for o in out]
    # both round as many operands to bfloat16, most of them differently: the same error but for chance, over 900 and more logits a few
    # hundredths of it (7.1e-3 and 7.3e-3 for one request of the first sizes, 7.5e-3 and 7.7e-3 for four of the last)
    assert off[0] <= 1.25 * off[2]


def test_against_plain_and_repeats_bit_for_bit(folders):
    contexts = [0, 70, 513]
    got, _, seqs = decode(folders["h64_even"], contexts, 4, True)
    again, _, _ = decode(folders["h64_even"], contexts, 4, True, graphs=False)
    assert torch.equal(got, again)
    wts, cfg = plain.load(folders["h64_even"])
    for i, (c, ids) in enumerate(zip(contexts, seqs)):
        want = torch.from_numpy(np.asarray(plain.forward(ids, wts, cfg)))[c:].float()
        have = got[:, i].cpu().float()
        assert (have - want).norm() <= 1e-2 * want.norm()  # bfloat16 operands


def test_smaller_pages(folders):
    contexts = [31, 200]
    got, _, _ = decode(folders["h128"], contexts, 2, True, page=16)
    want, _, _ = decode(folders["h128"], contexts, 2, False, page=16)
    assert (got - want).norm() <= 2**-7 * want.norm()


def test_model_loaded_again(folders):
    """The kernel's table of weights follows a model that is loaded again behind the runner's back."""
    from alofa_b200.engine.loading import load_model
    from alofa_b200.engine.step import StepEntry, StepRunner
    from alofa_b200.parts.linear import RESIDUAL, Linear

    model, _, _ = load_model(folders["h64_even"], "bfloat16")
    runner = StepRunner(model, block_size=64, num_pages=4, max_requests=1, max_tokens=128, max_step_tokens=64, cuda_graphs=False)
    first = runner.forward([StepEntry(runner.admit(1), [7], [0])]).clone()
    for block in model.layers:
        block.mixer.out = Linear(block.mixer.out.weight * 2, None, RESIDUAL)
    runner.release(0)
    changed = runner.forward([StepEntry(runner.admit(2), [7], [0])]).clone()
    runner.release(0)
    runner.decode_stack = None
    want = runner.forward([StepEntry(runner.admit(3), [7], [0])]).clone()
    assert (first - want).norm() > 0.01 * want.norm()
    assert (changed - want).norm() <= 2**-8 * want.norm()


def test_infinities_nan_and_large_numbers_of_an_embedding_reach_the_logits(folders):
    """The stream of a step as one kernel loses nothing that the same step layer by layer keeps."""
    from alofa_b200.engine.loading import load_model
    from alofa_b200.engine.step import StepEntry, StepRunner

    model, _, _ = load_model(folders["h64_even"], "bfloat16")
    with torch.no_grad():
        rows = model.embedding.weight
        rows[1, 3] = float("nan")
        rows[2, 70] = float("inf")
        rows[3] *= 2.0**40
        rows[4, 5] = -(2.0**33)
    tokens = [1, 2, 3, 4, 20]
    out = []
    for stacked in (True, False):
        runner = StepRunner(model, block_size=64, num_pages=10, max_requests=5, max_tokens=128, max_step_tokens=64, cuda_graphs=False)
        if not stacked:
            runner.decode_stack = None
        slots = [runner.admit(i) for i in range(5)]
        for _ in range(2):
            got = runner.forward([StepEntry(s, [t], [0]) for s, t in zip(slots, tokens)]).clone()
        runner.check_status()
        out.append(got[:, 10:])  # the head has the changed rows too
    got, want = out
    assert torch.equal(got.isnan(), want.isnan())
    assert want[0].isnan().all() and not want[2:].isnan().any()
    for i in (2, 3, 4):
        assert (got[i] - want[i]).norm() <= 2**-7 * want[i].norm()


def test_recorded_steps_of_a_model_loaded_again(folders):
    """A model that is loaded again decodes with the new weights, at sizes that were recorded before and at others; one that the kernel
    cannot take any more goes layer by layer."""
    from alofa_b200.csrc import ops
    from alofa_b200.engine.loading import load_model
    from alofa_b200.engine.step import StepEntry, StepRunner
    from alofa_b200.parts.linear import RESIDUAL, Linear
    from alofa_b200.weights.loader import load_state

    def make(model):
        return StepRunner(model, block_size=64, num_pages=8, max_requests=2, max_tokens=128, max_step_tokens=64)

    def steps(runner, n):
        """Logits of the last of three steps (outright, recorded, replayed) of n requests, and its launches."""
        slots = [runner.admit(i) for i in range(n)]
        for t in range(3):
            before = ops.launch_count()
            out = runner.forward([StepEntry(s, [7 + t + i], [0]) for i, s in enumerate(slots)]).clone()
        for s in slots:
            runner.release(s)
        runner.check_status()
        return out, ops.launch_count() - before

    model, _, _ = load_model(folders["h64_even"], "bfloat16")
    runner = make(model)
    first = {n: steps(runner, n)[0] for n in (1, 2)}
    state = load_state(model.tensors(), folders["h64_even"], model.rt.dtype, model.rt.device)
    for name in state:
        if name.endswith("o_proj.weight"):
            state[name] = state[name] * 3
    model.load(state)
    fresh = make(model)
    for n in (1, 2):
        got, launches = steps(runner, n)
        want, fewest = steps(fresh, n)
        assert torch.equal(got, want) and launches == fewest
        assert (got - first[n]).norm() > 0.01 * got.norm()
    # a bias, which the kernel does not have, behind the runner's back: the next size is layer by layer (recorded ones stay what they are)
    model.loads += 1
    for block in model.layers:
        block.mixer.out = Linear(block.mixer.out.weight, torch.ones(256, device="cuda"), RESIDUAL)
    got, launches = steps(runner, 2)
    fresh.decode_stack = None
    fresh._graphs.clear()
    want, layers = steps(fresh, 2)
    assert launches == layers > fewest and torch.equal(got, want)


def test_runner_made_before_its_model_is_loaded(folders):
    from alofa_b200.csrc import ops
    from alofa_b200.engine.loading import load_model
    from alofa_b200.engine.step import StepEntry, StepRunner
    from alofa_b200.parts.model import Model
    from alofa_b200.weights.loader import load_state

    loaded, _, _ = load_model(folders["h64_even"], "bfloat16")
    out, launches = [], []
    for early in (True, False):
        model = Model(loaded.spec, loaded.rt)
        load = lambda: model.load(load_state(model.tensors(), folders["h64_even"], model.rt.dtype, model.rt.device))  # noqa: E731
        if not early:
            load()
        runner = StepRunner(model, block_size=64, num_pages=4, max_requests=1, max_tokens=128, max_step_tokens=64, cuda_graphs=False)
        if early:
            load()
        slot, before = runner.admit(1), ops.launch_count()
        out.append(runner.forward([StepEntry(slot, [9], [0])]).clone())
        launches.append(ops.launch_count() - before)
    assert torch.equal(*out) and launches[0] == launches[1]


@pytest.mark.parametrize("name", ["h64_even", "h128"])
@pytest.mark.parametrize("context, pages, rows", [(40, 1, 16), (600, 7, 64)])
def test_keys_that_weigh_nothing(folders, name, context, pages, rows):
    """Scores of minus infinity, and finite ones as far below the others, over a whole granule, warp and split of keys: the others decide."""
    from alofa_b200.engine.loading import load_model
    from alofa_b200.engine.step import StepEntry, StepRunner

    model, _, _ = load_model(folders[name], "bfloat16")
    for block in model.layers:  # queries that are known: ten everywhere, turned by the position
        block.mixer.qkv.weight[: block.mixer.q_dim] = 0
        block.mixer.qkv.bias[: block.mixer.q_dim] = 10
    ids = [int(t) for t in np.random.default_rng(3).integers(0, 300, context + 1)]
    out = []
    for stacked, value in ((False, -3e38), (True, -3e38), (True, -1e32)):
        runner = StepRunner(model, block_size=64, num_pages=10, max_requests=1, max_tokens=640, max_step_tokens=640, cuda_graphs=False)
        if not stacked:
            runner.decode_stack = None
        slot = runner.admit(1)
        runner.forward([StepEntry(slot, ids[:context])])
        for kv in runner.storage.caches.values():
            k = kv.k.view(-1, 64, *kv.k.shape[1:])
            k[:pages, :rows, :, kv.k.shape[2] // 2 - 1] = value  # of the slowest pair: hardly turned
        out.append(runner.forward([StepEntry(slot, ids[context:], [0])]).clone())
        runner.check_status()
    want, got, finite = out
    assert want.isfinite().all() and got.isfinite().all()
    assert (got - want).norm() <= 2**-7 * want.norm()
    assert torch.equal(got, finite)


def test_two_runners_on_two_streams(folders):
    """Steps of two runners side by side, of shapes that want different amounts of shared memory, and beside other work that fills the
    device: the same bits as one after the other."""
    from alofa_b200.engine.loading import load_model
    from alofa_b200.engine.step import StepEntry, StepRunner

    def make(name, n):
        model, _, _ = load_model(folders[name], "bfloat16")
        runner = StepRunner(model, block_size=64, num_pages=2 * n, max_requests=n, max_tokens=128, max_step_tokens=64)
        return runner, [runner.admit(i) for i in range(n)]

    def step(pair, t):
        runner, slots = pair
        return runner.forward([StepEntry(s, [(7 * t + i) % 300], [0]) for i, s in enumerate(slots)])

    kinds, steps = [("h64_odd", 1), ("h128_group7", 8)], 12
    want = []
    for kind in kinds:
        pair = make(*kind)
        want.append([step(pair, t).clone() for t in range(steps)])
    pairs, streams, got = [make(*kind) for kind in kinds], [torch.cuda.Stream() for _ in kinds], [[], []]
    other, a = torch.cuda.Stream(), torch.ones((4096, 4096), dtype=torch.bfloat16, device="cuda")
    torch.cuda.synchronize()
    for t in range(steps):
        with torch.cuda.stream(other):
            for _ in range(4):
                a @ a
        for i, (pair, stream) in enumerate(zip(pairs, streams)):
            with torch.cuda.stream(stream):
                got[i].append(step(pair, t).clone())
    torch.cuda.synchronize()
    for i, (runner, _) in enumerate(pairs):
        runner.check_status()
        assert all(torch.equal(a, b) for a, b in zip(got[i], want[i]))


def test_more_layers_than_a_launch_takes(tmp_path):
    """A model of more layers than the kernel's parameters hold goes in several launches; also one whose last launch is a single layer."""
    from alofa_b200.models.qwen2 import NAME, Qwen2Config
    from alofa_b200.weights.random_init import write_random_model

    for layers in (48, 49, 100):
        folder = write_random_model(tmp_path / str(layers), NAME, Qwen2Config(layers, 64, 1, 1, 64, 128, 300, 1e-6, 1e4, True, 4096), 7, torch.bfloat16)
        got, launched, _ = decode(folder, [70, 3], 3, True)
        want, more, _ = decode(folder, [70, 3], 3, False)
        assert launched < more
        # as in test_matches_layer_by_layer, the roundings of all layers: sqrt(2 sides * layers * 8) * 2^-9 / sqrt(3)
        assert (got - want).norm() <= (2 * layers * 8 / 3) ** 0.5 * 2**-9 * want.norm()


def test_a_step_whose_keys_outgrow_the_kernel_goes_layer_by_layer(folders):
    """Recorded steps of one size and context bucket on either side of the line: each replay is the route of its own lengths."""
    from alofa_b200.csrc import ops
    from alofa_b200.engine.loading import load_model
    from alofa_b200.engine.step import StepEntry, StepRunner

    model, _, _ = load_model(folders["h64_odd"], "bfloat16")
    ids = [int(t) for t in np.random.default_rng(9).integers(0, 300, 4000)]
    lengths = [3000, 40, 40]
    runner = StepRunner(model, block_size=64, num_pages=80, max_requests=8, max_tokens=4096, max_step_tokens=2048)
    stack, launches, out = runner.decode_stack, [], []
    slots = [runner.admit(i) for i in range(3)]
    for s, n in zip(slots, lengths):
        for lo in range(0, n, 2000):
            runner.forward([StepEntry(s, ids[lo : min(n, lo + 2000)])])
    bucket = runner._context_bucket(3001)
    for most in (32, 0, 32, 0, 32, 0):  # the line moved, not the lengths: whether this step is on its near side
        stack.MOST_GRANULES = most
        before = ops.launch_count()
        out.append(runner.forward([StepEntry(s, [5 + i], [0]) for i, s in enumerate(slots)]).clone())
        launches.append(ops.launch_count() - before)
    runner.check_status()
    assert launches[4] == launches[2] < launches[3] == launches[5]
    assert {key for key in runner._graphs if key[2] == "decode"} == {(3, bucket, "decode", True), (3, bucket, "decode", False)}
