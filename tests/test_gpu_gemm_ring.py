"""The few-token tensor-core product where one CTA has an SM to itself: K around whole turns of its ring of stages."""
import math

import pytest
import torch

from tests.gpu_common import cuda_ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,stages", [(1, 11), (16, 11), (17, 10), (37, 9), (64, 8)])
def test_runs_around_whole_turns_of_the_ring(tokens, stages):
    """208 KB of stages of 64 columns of K (128 rows of w, the tokens rounded up to 16): below a turn, at it, one beyond, two
    turns and a ragged end."""
    ops = cuda_ops(torch.bfloat16)
    for kblocks, rest in ((1, 0), (stages - 1, 0), (stages, 0), (stages + 1, 8), (2 * stages, 0), (2 * stages + 1, 40), (5 * stages, 56)):
        k = kblocks * 64 + rest
        g = torch.Generator(device="cuda").manual_seed(k)
        x = torch.randn(tokens, k, device="cuda", generator=g).bfloat16()
        w = torch.randn(200, k, device="cuda", generator=g).bfloat16()
        out = torch.full((tokens, 200), float("nan"), device="cuda")
        ops.linear(x, w, out)
        want = x.double() @ w.double().T
        bound = math.sqrt(k) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)   # float32 sums of exact products
        assert ((out.double() - want).abs() <= bound).all(), (k, ((out.double() - want).abs() / bound).max())
    ops.check_status()
