"""A dropped model gives its weights back at once: nothing of it is in a reference cycle."""
import gc
import weakref

import pytest
import torch

import tiny
from alofa_b200.parts.linear import GATED, RESIDUAL, STORE, Linear


@pytest.fixture
def no_collector():
    gc.collect()
    gc.disable()
    yield
    gc.enable()


@pytest.mark.parametrize("epi", [STORE, RESIDUAL, GATED])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_linear_goes_with_its_last_reference(no_collector, epi, dtype):
    linear = Linear(torch.zeros((64, 64), dtype=dtype), None, epi)
    weight = weakref.ref(linear.weight)
    assert (linear._fast is not None) == (dtype == torch.bfloat16)
    del linear
    assert weight() is None


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_model_and_runner_go_with_their_last_reference(no_collector, tmp_path, dtype):
    from alofa_b200.config.registry import read_model_config
    from alofa_b200.engine.step import StepRunner
    from alofa_b200.parts.base import Runtime
    from alofa_b200.parts.model import Model
    from alofa_b200.weights.loader import load_state

    folder = tiny.write(tmp_path / "A", "A")
    arch, cfg = read_model_config(folder)
    rt = Runtime(torch.device("cpu"), dtype)
    model = Model(arch.build_spec(cfg), rt)
    model.load(load_state(model.tensors(), folder, dtype, rt.device))
    runner = StepRunner(model, block_size=16, num_pages=8, max_requests=2, max_tokens=64, max_step_tokens=32)
    held = [weakref.ref(t) for block in model.layers for t in (block.mixer.qkv.weight, block.mixer.out.weight, block.feed_forward.gate_up.weight, block.feed_forward.down.weight)]
    held += [weakref.ref(t) for t in (model.embedding.weight, runner.storage.caches[0].k)]
    del model, runner
    assert [i for i, ref in enumerate(held) if ref() is not None] == []
