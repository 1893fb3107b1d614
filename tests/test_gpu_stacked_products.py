"""The 32-bit path of every design at widths whose products leave as stacks of runs: the bits do not depend on whether a consumer
adds a stack's slices or finds the product summed (which follows from the batch), so neither does a request's result."""

import pytest
import torch

from shrike_b200.config import parse_config
from shrike_b200.engine.batch import StepEntry
from shrike_b200.engine.llm_engine import LLMEngine
from shrike_b200.shapes import shape_config
from shrike_b200.weights.random_init import random_tensors

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", ["qwen2.5-0.5b", "sadodra-1.5b", "vupitar-1.5b", "kavedra-1.5b", "setotar-1.5b", "nulazen-1.5b", "radilix-1.5b"])
def test_float32_logits_are_the_same_with_and_without_stacks(shape):
    raw = shape_config(shape)
    config = parse_config(raw)
    tensors = random_tensors(config, 1, "cuda", torch.float32)
    ids = torch.randint(0, raw.get("vocab_size") or raw["vocab"], (72,), generator=torch.Generator().manual_seed(3)).tolist()
    results = []
    for limit in (None, 0):
        engine = LLMEngine(None, block_size=16, num_blocks=24, max_running=2, dtype="float32", config=config, tensors=dict(tensors))
        runner = engine.runner
        if limit is not None:
            runner.ops.FP32_STACK_FLOATS = limit
        cache, other = runner.cache.open(), runner.cache.open()
        runner.cache.append(cache, 0, 40)
        runner.cache.append(other, 0, 3)
        logits = [runner.step([StepEntry(cache, ids[:40], 0, [0, 39])]).clone(), runner.step([StepEntry(other, ids[40:43], 0, [2])]).clone()]
        for held, length in ((cache, 40), (other, 3)):
            runner.cache.advance(held, length)
            runner.cache.append(held, length, 1)
        logits.append(runner.step([StepEntry(cache, ids[50:51], 40, [0]), StepEntry(other, ids[51:52], 3, [0])]).clone())
        runner.ops.check_status()
        assert bool(runner.ops._partials) == (limit is None), "products at these widths leave as stacks"
        results.append(torch.cat(logits))
        del engine, runner
    assert torch.isfinite(results[0]).all() and torch.equal(*results)
