"""Host-side decisions of the kernels' object that need no GPU: what it holds, and by which rules it cuts the work."""

import gc

import pytest
import torch

from shrike_b200.ops.cuda_ops import CudaOps


def bare_ops(dtype):
    """The object without its libraries: its bookkeeping runs on the CPU."""
    ops = object.__new__(CudaOps)
    ops.dtype, ops.device, ops.tensor_core_gemm_max_tokens = dtype, torch.device("cpu"), 64
    ops._partials, ops.generation = {}, 0
    return ops


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@torch.inference_mode()
def test_a_stack_lives_as_long_as_the_buffer_it_belongs_to(dtype):
    ops = bare_ops(dtype)
    kept = torch.empty(2048 * 8)
    first = ops._partial_stack(kept[: 3 * 8].view(3, 8), 4)
    where, stamp = first.data_ptr(), ops.generation
    assert first.shape == (4, 3, 8)
    for rows in range(100, 2000, 100):   # a buffer that is replaced by a larger one, prompt after prompt
        out = torch.empty(rows * 8)
        stack = ops._partial_stack(out.view(rows, 8), 16)
        assert stack.shape == (16, rows, 8) and ops._partial_stack(out.view(rows, 8), 16).data_ptr() == stack.data_ptr()
        del out, stack
        gc.collect()
        assert len(ops._partials) <= 3   # the kept one, this one, the one before it at most
    again = ops._partial_stack(kept[: 2 * 8].view(2, 8), 4)
    assert again.data_ptr() == where and ops.generation > stamp
    grown = ops._partial_stack(kept.view(2048, 8), 4)
    assert grown.shape == (4, 2048, 8)


def test_single_token_splits_where_the_places_of_a_power_of_two_would_stay_empty():
    """Every count of pairs up to the device's places: no clusters beyond two thirds of it, and splits between two powers of
    two only where they leave a CTA fewer tiles."""
    resident = 296
    for tiles in range(1, 200):
        for groups in range(1, 300):
            splits, cluster = CudaOps.single_token_splits(tiles, groups, resident)
            want = max(1, min(tiles, resident // groups))
            assert 1 <= splits <= want and splits % cluster == 0 and splits // cluster <= 32
            power = 1 << (min(want, 8).bit_length() - 1)
            if splits & (splits - 1) and cluster == 1:
                assert groups >= 24 and (splits == want or splits % 8 == 0)
                assert splits % 8 == 0 or -(-tiles // splits) < -(-tiles // power)
            if tiles <= 4 and groups >= 64:
                assert (splits, cluster) == (1, 1)
    assert CudaOps.single_token_splits(16, 24, resident) == (8, 8)      # twelve CTAs would have two tiles too
    assert CudaOps.single_token_splits(64, 24, resident) == (12, 1)     # six tiles a CTA instead of eight
    assert CudaOps.single_token_splits(8, 48, resident) == (4, 4)
    assert CudaOps.single_token_splits(16, 48, resident) == (6, 1)
    assert CudaOps.single_token_splits(16, 80, resident) == (3, 1)
    assert CudaOps.single_token_splits(4, 63, resident) == (4, 4)


@pytest.mark.parametrize("max_q_len,table_keys,max_ctx_len,head_dim,ctas,short", [
    (43, 128, 43, 64, 14, True), (43, 128, 43, 128, 12, True), (64, 128, 64, 256, 74, True),    # a short prompt
    (65, 128, 65, 64, 14, False), (43, 256, 300, 128, 12, False), (2, 256, 129, 64, 14, False),   # longer ones, longer contexts
    (36, 128, 100, 64, 14, True), (36, 128, 100, 128, 12, False), (36, 128, 0, 128, 12, False), (17, 64, 0, 128, 12, True),
    (33, 128, 64, 128, 75, False), (32, 128, 64, 128, 75, True), (64, 128, 64, 128, 148, False), (64, 128, 64, 128, 149, True),
    (64, 128, 64, 64, 112, True), (64, 128, 128, 64, 112, False), (64, 128, 128, 64, 154, True), (32, 128, 128, 64, 140, True),
])
def test_which_portions_are_short(max_q_len, table_keys, max_ctx_len, head_dim, ctas, short):
    ops = bare_ops(torch.bfloat16)
    ops.sm_count = 148
    assert ops.short_portions(max_q_len, table_keys, max_ctx_len, head_dim, ctas) is short


@pytest.mark.parametrize("dtype,lengths,start,apart", [("bfloat16", 40, 60, True), ("bfloat16", 1, 60, False), ("float32", 40, 60, False),
                                                       ("float32", 1, 60, True)])
def test_a_captured_step_holds_for_contexts_for_which_the_same_kernels_run(dtype, lengths, start, apart):
    """Two steps of the same lengths and table widths, from the start and further on."""
    from shrike_b200.config import parse_config
    from shrike_b200.engine.batch import StepEntry
    from shrike_b200.engine.runner import ModelRunner
    from shrike_b200.weights.random_init import random_tensors
    from tests.emulated_ops import EmulatedOps
    from tests.tiny_configs import TINY

    config, ops = parse_config(TINY["C"]), EmulatedOps()
    ops.context_class = bare_ops(getattr(torch, dtype)).context_class
    runner = ModelRunner(config, dict(random_tensors(config, 1)), ops, "cpu", dtype, page_size=16, num_pages=24, max_slots=4)
    keys = []
    for first in (0, start):
        cache = runner.cache.open()
        runner.cache.append(cache, 0, first + lengths)
        keys.append(runner.prepare([StepEntry(cache, [3] * lengths, first, [lengths - 1])]).key)
    assert (keys[0] != keys[1]) == apart
