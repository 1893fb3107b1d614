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
