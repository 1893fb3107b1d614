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
