"""The layer sizes of the benchmarked shape (hidden 896, 14 heads on 2, head 64,
intermediate 4864, vocabulary 151936, tied head), two layers deep, against the
plain implementation: whole prompt, decoded tail, and a mixed step.  These are
the sizes the tensor-core kernels are tuned for (tiles of 128/256 with tails:
1152 = 9 x 128, 4864 = 38 x 128, 151936 = 1187 x 128)."""
import gc

import numpy as np
import pytest
import torch

import plain_qwen2 as plain

pytestmark = pytest.mark.gpu

TOL = {"float32": 1e-5, "bfloat16": 2e-2}


@pytest.fixture(scope="module")
def shaped():
    from alofa_b200.models.qwen2 import Qwen2Config, build_spec
    from alofa_b200.parts import expected_tensors
    from alofa_b200.weights.random_init import random_state

    cfg = Qwen2Config(2, 896, 14, 2, 64, 4864, 151936, 1e-6, 1e6, True, 32768)
    state = random_state(expected_tensors(build_spec(cfg)), 5, torch.bfloat16)
    wts = {k: v.to(torch.float64).numpy() for k, v in state.items()}
    pcfg = {"L": 2, "H": 896, "nh": 14, "nkv": 2, "hd": 64, "I": 4864, "V": 151936, "eps": 1e-6, "theta": 1e6, "tied": True, "window": None, "first_window_layer": 2}
    rng = np.random.default_rng(0)
    a = [int(t) for t in rng.integers(0, 151936, 150)]
    b = [int(t) for t in rng.integers(0, 151936, 70)]
    ref = {"a": plain.forward(a, wts, pcfg), "b": plain.forward(b, wts, pcfg)}
    return cfg, state, {"a": a, "b": b}, ref


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_benchmark_layer_sizes_against_plain(shaped, dtype):
    from alofa_b200.engine.loading import compute_dtype
    from alofa_b200.engine.step import StepEntry, StepRunner
    from alofa_b200.models.qwen2 import build_spec
    from alofa_b200.parts.base import Runtime
    from alofa_b200.parts.model import Model
    from alofa_b200.weights.loader import load_state

    cfg, state, toks, ref = shaped
    model = Model(build_spec(cfg), Runtime(torch.device("cuda"), compute_dtype(dtype)))
    model.load(load_state(model.tensors(), state, model.rt.dtype, model.rt.device))
    runner = StepRunner(model, block_size=64, num_pages=8, max_requests=4, max_tokens=512, max_step_tokens=256)
    a, b = toks["a"], toks["b"]
    sa, sb = runner.admit(1), runner.admit(2)
    got = {"a": [], "b": []}
    got["a"].append(runner.forward([StepEntry(sa, a[:130], list(range(130)))]).cpu().numpy())  # a prompt portion past one 128-token tile
    mixed = runner.forward([StepEntry(sa, a[130:131], [0]), StepEntry(sb, b[:67], list(range(67)))]).cpu().numpy()  # a decoded token beside a prompt
    got["a"].append(mixed[:1])
    got["b"].append(mixed[1:])
    for i in range(131, 150):  # decoded one by one (CUDA graph of batch 1 in bfloat16)
        got["a"].append(runner.forward([StepEntry(sa, a[i : i + 1], [0])]).cpu().numpy())
    both = runner.forward([StepEntry(sb, b[67:68], [0])]).cpu().numpy()
    got["b"].append(both)
    got["b"].append(runner.forward([StepEntry(sb, b[68:], [0, 1])]).cpu().numpy())
    runner.check_status()
    for rid in ("a", "b"):
        mine = np.concatenate(got[rid]).astype(np.float64)
        want = ref[rid]
        bound = TOL[dtype] * max(1.0, float(np.abs(want).max()))
        diff = np.abs(mine - want)
        assert diff.max() <= bound, f"{dtype} request {rid}: position {int(np.argmax(diff.max(axis=1) > bound))} differs by {diff.max():.3e} > {bound:.3e}"
        assert (mine.argmax(axis=1) == want.argmax(axis=1)).mean() > 0.9


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_the_benchmarked_prompt_step_against_plain(shaped, dtype):
    """The benchmark's own prompt step at its real widths, two layers deep: one
    2,048-token prompt in one step, and in portions of 512, logits wanted at
    the first row, either side of a 128-token tile edge and the last row.
    This is where the persistent gate/up kernel has more tiles than SMs, the
    tensor-core attention runs several waves and the down product splits its
    depth."""
    from alofa_b200.engine.loading import compute_dtype
    from alofa_b200.engine.step import StepEntry, StepRunner
    from alofa_b200.models.qwen2 import build_spec
    from alofa_b200.parts.base import Runtime
    from alofa_b200.parts.model import Model
    from alofa_b200.weights.loader import load_state

    cfg, state, _, _ = shaped
    wts = {k: v.to(torch.float64).numpy() for k, v in state.items()}
    pcfg = {"L": 2, "H": 896, "nh": 14, "nkv": 2, "hd": 64, "I": 4864, "V": 151936, "eps": 1e-6, "theta": 1e6, "tied": True, "window": None, "first_window_layer": 2}
    toks = [int(t) for t in np.random.default_rng(7).integers(0, 151936, 2048)]
    rows = [0, 127, 128, 2047]
    want = plain.forward(toks, wts, pcfg, rows=rows)
    model = Model(build_spec(cfg), Runtime(torch.device("cuda"), compute_dtype(dtype)))
    model.load(load_state(model.tensors(), state, model.rt.dtype, model.rt.device))
    runner = StepRunner(model, block_size=64, num_pages=70, max_requests=2, max_tokens=4096, max_step_tokens=2112)
    bound = TOL[dtype] * max(1.0, float(np.abs(want).max()))
    whole = runner.admit(1)
    got = runner.forward([StepEntry(whole, toks, rows)]).cpu().numpy().astype(np.float64)
    assert np.abs(got - want).max() <= bound, f"{dtype} whole: {np.abs(got - want).max():.3e} > {bound:.3e}"
    cut = runner.admit(2)
    parts = []
    for lo in range(0, 2048, 512):
        local = [r - lo for r in rows if lo <= r < lo + 512]
        out = runner.forward([StepEntry(cut, toks[lo : lo + 512], local)])
        if local:
            parts.append(out.cpu().numpy().astype(np.float64))
    got = np.concatenate(parts)
    runner.check_status()
    assert np.abs(got - want).max() <= bound, f"{dtype} portions of 512: {np.abs(got - want).max():.3e} > {bound:.3e}"
    assert (got.argmax(axis=1) == want.argmax(axis=1)).all()


def test_steps_allocate_nothing(shaped):
    """Every buffer a step needs comes from the runner's arena: once a step of
    a shape has run, prompt steps, mixed steps and decode steps leave the
    device memory the tensor library holds exactly as it was."""
    from alofa_b200.engine.loading import compute_dtype
    from alofa_b200.engine.step import StepEntry, StepRunner
    from alofa_b200.models.qwen2 import build_spec
    from alofa_b200.parts.base import Runtime
    from alofa_b200.parts.model import Model
    from alofa_b200.weights.loader import load_state

    cfg, state, toks, _ = shaped
    model = Model(build_spec(cfg), Runtime(torch.device("cuda"), compute_dtype("bfloat16")))
    model.load(load_state(model.tensors(), state, model.rt.dtype, model.rt.device))
    runner = StepRunner(model, block_size=64, num_pages=16, max_requests=4, max_tokens=512, max_step_tokens=256, cuda_graphs=False)
    a, b = toks["a"], toks["b"]

    def steps():
        sa, sb = runner.admit(1), runner.admit(2)
        runner.forward([StepEntry(sa, a[:130], [129])])
        runner.forward([StepEntry(sa, a[130:131], [0]), StepEntry(sb, b[:67], [66])])
        for k in range(3):  # both decode, three steps
            runner.forward([StepEntry(sa, a[131 + k : 132 + k], [0]), StepEntry(sb, b[67 + k : 68 + k], [0])])
        runner.release(sa)
        runner.release(sb)

    steps()  # kernels loaded, the arena grown to what these shapes need
    gc.collect()  # what other tests left in reference cycles does not go in between
    torch.cuda.synchronize()
    grown = runner.arena.grown
    before = torch.cuda.memory_allocated()
    peak = torch.cuda.max_memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    steps()
    torch.cuda.synchronize()
    assert torch.cuda.memory_allocated() == before and torch.cuda.max_memory_allocated() == before
    assert runner.arena.grown == grown
    runner.check_status()


@pytest.mark.parametrize("n, whole", [(8, True), (8, False), (12, False), (40, False)])
def test_decode_steps_on_the_accumulator_stream_give_the_same_bits_every_run(shaped, n, whole):
    """Requests decoded together (eight: all layers in one kernel, and the
    five-kernel layer in its place; twelve: the five-kernel layer; forty: the
    layer of larger steps), whose residual products add their split sums with
    atomic integer adds in whatever order their CTAs finish: two runs from the
    same state must give the same logits bit for bit, and the accumulators are
    zero between steps."""
    from alofa_b200.csrc import ops
    from alofa_b200.engine.loading import compute_dtype
    from alofa_b200.engine.step import StepEntry, StepRunner
    from alofa_b200.models.qwen2 import build_spec
    from alofa_b200.parts.base import Runtime
    from alofa_b200.parts.model import Model
    from alofa_b200.weights.loader import load_state

    cfg, state, _, _ = shaped
    model = Model(build_spec(cfg), Runtime(torch.device("cuda"), compute_dtype("bfloat16")))
    model.load(load_state(model.tensors(), state, model.rt.dtype, model.rt.device))
    rng = np.random.default_rng(11)
    prompts = [[int(t) for t in rng.integers(0, 151936, int(k))] for k in rng.integers(20, 200, n)]
    feed = rng.integers(0, 151936, size=(4, n))
    runs = []
    for graphs in (True, True, False):
        runner = StepRunner(model, block_size=64, num_pages=5 * n, max_requests=n, max_tokens=512, max_step_tokens=256, cuda_graphs=graphs)
        assert runner._stream_acc is not None and n <= runner.STREAM_TOKENS
        if not whole and n <= ops.DECODE_STACK_TOKENS:
            runner.decode_stack = None
        slots = [runner.admit(i) for i in range(n)]
        for s, p in zip(slots, prompts):
            runner.forward([StepEntry(s, p, [])])
        rows = []
        for step in feed:
            before = ops.launch_count()
            rows.append(runner.forward([StepEntry(s, [int(t)], [0]) for s, t in zip(slots, step)]).clone())
            assert int(runner._stream_acc.abs().sum()) == 0, "an accumulator was left with a value after the step"
        assert graphs or (ops.launch_count() - before < 5 * cfg.num_hidden_layers) == whole, "the step went another way than this test says"
        runner.check_status()
        runs.append(torch.stack(rows))
    assert torch.equal(runs[0], runs[1]), "two runs of the same steps differ"
    assert torch.equal(runs[0], runs[2]), "graph replay and plain launches differ"


@pytest.mark.parametrize("design", ["qwen2", "kotutar", "darolix", "dibulix", "kikerax", "pekerax", "nugopel"])
def test_parts_take_no_more_scratch_than_they_declare(design):
    """Prompt steps of every design at its 2k benchmark sizes: what a layer's mixer and feed-forward take from the arena, the
    parts of deep products that their consumers add up among it, against ``scratch_row_bytes``; and no region grows."""
    import importlib

    import bench
    from alofa_b200.engine.loading import compute_dtype
    from alofa_b200.engine.step import StepEntry, StepRunner
    from alofa_b200.parts import expected_tensors
    from alofa_b200.parts.base import Runtime
    from alofa_b200.parts.model import Model
    from alofa_b200.weights.loader import load_state

    z = dict(bench.DESIGN_SIZES["2k"], experts=8, top=2, vocab=512)
    if design in ("qwen2", "kotutar"):
        cfg = bench.qwen2_config_like(z) if design == "qwen2" else bench.kotutar_config(z)
    else:
        sizes = dict(getattr(bench, design.upper() + "_SIZES")["2k"])
        cfg = getattr(bench, design + "_config")(z, {**sizes, **{k: v for k, v in (("groups", 2), ("keep", 1)) if k in sizes}} if design in ("kikerax", "pekerax") else sizes)
    spec = importlib.import_module(f"alofa_b200.models.{design}").build_spec(cfg)
    gen = torch.Generator(device="cuda").manual_seed(1)
    state = {}
    for name, t in expected_tensors(spec).items():
        shape = tuple(abs(n) for n in t.shape)
        x = torch.randn(shape, generator=gen, device="cuda") * 0.02
        state[name] = (x + 1 if t.init == "ones" else x + torch.eye(shape[0], device="cuda") if t.init == "identity" else x).to(torch.bfloat16)
    model = Model(spec, Runtime(torch.device("cuda"), compute_dtype("bfloat16")))
    model.load(load_state(model.tensors(), state, model.rt.dtype, model.rt.device))
    over = []

    def watched(part, run, arena):
        def forward(*args, **kwargs):
            held = lambda: sum(b.numel() for b in arena.current.blocks[: arena.current.block]) + arena.current.offset  # noqa: E731
            before, out = held(), run(*args, **kwargs)
            rows = args[2].shape[0]
            if held() - before > rows * part.scratch_row_bytes() + 64 * 256:  # each buffer starts on 256 bytes
                over.append((type(part).__name__, rows, (held() - before) // rows, part.scratch_row_bytes()))
            return out

        return forward

    for tokens in (700, 1024, 2048):
        runner = StepRunner(model, block_size=64, num_pages=80, max_requests=4, max_tokens=2048, max_step_tokens=tokens, cuda_graphs=False)
        parts = [p for block in model.layers for p in (block.mixer, block.feed_forward) if p is not None]
        for part in parts:
            part.forward = watched(part, type(part).forward.__get__(part), runner.arena)
        runner.forward([StepEntry(runner.admit(1), np.random.default_rng(0).integers(0, 512, tokens).tolist(), [tokens - 1])])
        runner.check_status()
        assert runner.arena.grown == 0
    assert not over, over
