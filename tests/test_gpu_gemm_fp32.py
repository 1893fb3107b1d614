"""The 32-bit product at the sizes where its work is cut differently: against float64, and bit for bit against the same
row in other batches."""

import math

import pytest
import torch

from tests.gpu_common import cuda_ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


def rnd(*shape, seed=0):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(DEV)


# k below and above the sizes from which it is cut into runs, ragged last runs and boxes; n around the row counts of a
# warp, a tile, and the matrix size from which a row is one chain
@pytest.mark.parametrize("n,k", [(7, 4), (129, 508), (130, 512), (96, 900), (1000, 4092), (257, 4100), (8, 9000), (9472, 516), (18943, 516), (18945, 516), (300, 1001)])
def test_gemm_fp32_gives_a_row_the_same_bits_in_every_batch(n, k):
    ops = cuda_ops(torch.float32)
    rows = 200
    x, w, bias = rnd(rows, k, seed=1), rnd(n, k, seed=2), rnd(n, seed=3)
    want = x.double() @ w.double().T
    # sums of k terms in float32: sqrt(k) u sum |a b| (Higham & Mary 2019), u = 2^-24
    bound = math.sqrt(k) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)
    first = None
    for m in (1, 2, 3, 5, 8, 9, 16, 17, 32, 33, 64, 65, 128, 200):
        whole = torch.empty(m, n, device=DEV)
        ops.linear(x[:m].contiguous(), w, whole)
        assert ((whole.double() - want[:m]).abs() <= bound[:m]).all(), m
        first = whole[0].clone() if first is None else first
        assert torch.equal(first, whole[0]), m
        got = ops.linear(x[:m].contiguous(), w, torch.empty(m, n, device=DEV), allow_partials=True)
        if got.dim() == 3:   # the consumer's sum
            total = got[0].clone()
            for part in got[1:]:
                total += part
            got = total
        assert torch.equal(got, whole), m
        with_bias = torch.empty(m, n, device=DEV)
        ops.linear(x[:m].contiguous(), w, with_bias, bias=bias, allow_partials=True)
        assert torch.equal(with_bias, whole + bias), m
    ops.check_status()


def test_gemm_fp32_sums_its_runs_itself_where_their_stack_would_be_too_large():
    ops = cuda_ops(torch.float32)
    m, n, k = 40, 96, 9000
    x, w = rnd(m, k, seed=1), rnd(n, k, seed=2)
    stack = ops.linear(x, w, torch.empty(m, n, device=DEV), allow_partials=True)
    assert stack.dim() == 3
    total = stack[0].clone()
    for part in stack[1:]:
        total += part
    ops.FP32_STACK_FLOATS = stack.numel()
    assert ops.linear(x, w, torch.empty(m, n, device=DEV), allow_partials=True).dim() == 3
    ops.FP32_STACK_FLOATS = stack.numel() - 1
    out = torch.empty(m, n, device=DEV)
    got = ops.linear(x, w, out, allow_partials=True)
    assert got.data_ptr() == out.data_ptr() and torch.equal(got, total)


# every height of a tile, one row below it, at it, one and half a tile above; one run, several runs added where they lie, and
# a stack of runs; n and k that end within a tile
@pytest.mark.parametrize("tile", [4, 8, 10, 12, 14, 16])
@pytest.mark.parametrize("n,k", [(257, 500), (130, 4100), (96, 900), (300, 9000)])
def test_gemm_fp32_gives_the_same_bits_at_every_tile_height(tile, n, k):
    ops = cuda_ops(torch.float32)
    x, w, bias = rnd(12 * tile + 3, k, seed=tile), rnd(n, k, seed=2), rnd(n, seed=3)
    want = torch.cat([ops.linear(part.contiguous(), w, torch.empty(len(part), n, device=DEV)) for part in x.split(16)])   # few rows
    want_stack = [ops.linear(part.contiguous(), w, torch.empty(len(part), n, device=DEV), allow_partials=True) for part in x.split(16)]
    ops.gemm_fp32_tile = tile
    for m in (8 * tile - 1, 8 * tile, 8 * tile + 1, 12 * tile + 3):
        out = torch.full((m, n), float("nan"), device=DEV)
        assert torch.equal(ops.linear(x[:m].contiguous(), w, out), want[:m]), m
        assert torch.equal(ops.linear(x[:m].contiguous(), w, out, bias=bias), want[:m] + bias), m
        stack = ops.linear(x[:m].contiguous(), w, torch.empty(m, n, device=DEV), allow_partials=True)
        assert (stack.dim() == 3) == (k > 512)
        if stack.dim() == 3:
            assert torch.equal(stack, torch.cat([s for s in want_stack], dim=1)[:, :m]), m
    ops.check_status()


# one run in small tiles, up to as many as SMs and just beyond; runs side by side and added up, with a bias, an odd width, an output that
# does not lie on 16 bytes, and without the scratch
@pytest.mark.parametrize("m,n,k", [(17, 8, 4), (65, 130, 500), (64 * 37, 256, 36), (64 * 37 + 1, 256, 36), (17, 130, 900), (200, 131, 4100), (333, 300, 9000)])
def test_gemm_fp32_plain_results_of_prompts(m, n, k):
    ops = cuda_ops(torch.float32)
    x, w, bias = rnd(m, k, seed=m), rnd(n, k, seed=2), rnd(n, seed=3)
    want = torch.cat([ops.linear(part.contiguous(), w, torch.empty(len(part), n, device=DEV)) for part in x.split(16)])   # few rows
    shifted = torch.empty(m * n + 1, device=DEV)[1:].view(m, n)
    for out in (torch.full((m, n), float("nan"), device=DEV), shifted):
        assert torch.equal(ops.linear(x, w, out), want)
        assert torch.equal(ops.linear(x, w, out, bias=bias), want + bias)
    ops.gemm_fp32_tile = 16
    assert torch.equal(ops.linear(x, w, torch.empty(m, n, device=DEV), bias=bias), want + bias)
    ops.gemm_fp32_tile, ops.FP32_STACK_FLOATS = 0, 0
    assert torch.equal(ops.linear(x, w, torch.empty(m, n, device=DEV), bias=bias), want + bias)
    ops.check_status()
