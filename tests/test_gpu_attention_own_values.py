"""Portions whose keys are their own values, rows of 256, on the tcgen05 kernel: against float64."""

import pytest
import torch

from tests.gpu_common import cuda_ops
from tests.plain import plain_model as pm
from tests.test_gpu_kernels import paged_case

pytestmark = pytest.mark.gpu


# query tiles of 128 rows and key tiles of 128 in steps of 64: lengths and contexts around both, with and without several
# CTAs that share a tile's keys; tokens beside portions
@pytest.mark.parametrize("heads,page,window,splits", [(3, 16, None, 0), (12, 16, None, 2), (2, 8, 100, 0), (1, 64, 300, 3), (5, 32, None, 0)])
@pytest.mark.parametrize("ctx_lens,q_lens", [([2, 63, 64, 65], [2, 63, 64, 65]), ([127, 128, 129], [127, 128, 129]), ([257, 400, 1, 700], [256, 129, 1, 66]),
                                             ([1000], [900])])
def test_own_values_on_the_tensor_core_portions_kernel(heads, page, window, splits, ctx_lens, q_lens):
    ops = cuda_ops(torch.bfloat16)
    dim = 256
    case = paged_case(torch.bfloat16, heads, 1, dim, page, ctx_lens, q_lens, seed=heads)
    wide = torch.full((len(ctx_lens), max(case["table"].shape[1], 160 // page + 1)), -1, dtype=torch.int32, device="cuda")   # no short table
    wide[:, : case["table"].shape[1]] = case["table"]
    ops.portion_splits = splits
    out = torch.full_like(case["q"], float("nan"))
    plan = ops.attention_plan(heads, 1, dim, len(ctx_lens), wide.shape[1], page, max(q_lens), min(q_lens), sum(q_lens), list(q_lens), own_values=True)
    assert plan.tc_portions, "the case is meant for the tensor-core kernel"
    ops.paged_attention(case["q"], case["keys"], case["keys"], wide, case["q_start"], case["ctx_len"], case["seq_of"], heads, 1, dim,
                        dim ** -0.5, window, out, max_q_len=max(q_lens), max_ctx_len=max(ctx_lens), min_q_len=min(q_lens), q_lens=list(q_lens))
    ops.check_status()
    want = torch.cat([pm.causal_attention(q[len(q) - n:].double().cuda(), k.double().cuda(), k.double().cuda(), window)
                      for (q, k, _), n in zip(case["seqs"], q_lens)]).reshape(out.shape)
    # probabilities rounded to bfloat16 (2^-9 each, relative) and one rounding of outputs of order one: as for the other heads
    assert torch.isfinite(out).all() and (out.double() - want).abs().max() < 2e-2


@pytest.mark.parametrize("q_len,ctx_len,window,splits", [(700, 700, None, 1), (256, 2048, None, 2), (300, 1500, 512, 1)])
def test_own_values_are_as_close_to_float64_as_on_the_mma_kernel(q_len, ctx_len, window, splits):
    """Spread scores, of which a few keys take most of the weight.  Both kernels round a row's weights, relative to its largest,
    to bfloat16 once and their outputs once: over the million outputs here their errors agree to a part in a hundred."""
    ops = cuda_ops(torch.bfloat16)
    heads, dim, scale = 12, 256, 4.0 * 256 ** -0.5
    case = paged_case(torch.bfloat16, heads, 1, dim, 16, [ctx_len], [q_len], seed=7)
    q, k, _ = case["seqs"][0]
    q, k = q[ctx_len - q_len:].double().cuda(), k[:, 0].double().cuda()
    gap = torch.arange(ctx_len - q_len, ctx_len, device="cuda")[:, None] - torch.arange(ctx_len, device="cuda")[None]
    hidden = (gap < 0) | (gap >= (window or ctx_len))
    want = torch.stack([torch.softmax((q[:, a] @ k.T * scale).masked_fill(hidden, float("-inf")), -1) @ k for a in range(heads)], 1).reshape(q_len, -1)
    errors = {}
    for tensor_cores in (True, False):
        ops.tensor_core_attention, ops.portion_splits = tensor_cores, splits
        plan = ops.attention_plan(heads, 1, dim, 1, case["table"].shape[1], 16, q_len, q_len, q_len, [q_len], own_values=True)
        assert bool(plan.tc_portions) == tensor_cores
        out = torch.full_like(case["q"], float("nan"))
        ops.paged_attention(case["q"], case["keys"], case["keys"], case["table"], case["q_start"], case["ctx_len"], case["seq_of"], heads, 1,
                            dim, scale, window, out, max_q_len=q_len, max_ctx_len=ctx_len, min_q_len=q_len, q_lens=[q_len])
        ops.check_status()
        errors[tensor_cores] = float((out.double() - want).norm() / want.norm())
    assert errors[True] <= 1.01 * errors[False], errors


# what the launch accepts beside a window, each where a step of 64 keys, a tile of 128 and the last query tile end; the oracle in float64
@pytest.mark.parametrize("kv_heads,heads", [(1, 3), (2, 4)])
@pytest.mark.parametrize("options", [{}, {"sinks": True}, {"softcap": 5.0}, {"slopes": True}, {"window": 70, "keep_first": 5},
                                     {"window": 130, "keep_first": 129, "sinks": True}, {"chunk": 96}, {"softcap": 3.0, "slopes": True, "window": 200}])
@pytest.mark.parametrize("ctx_lens,q_lens,splits", [([129, 66, 1], [129, 65, 1], 0), ([400], [300], 3)])
def test_own_values_with_everything_a_score_can_have(kv_heads, heads, options, ctx_lens, q_lens, splits):
    ops = cuda_ops(torch.bfloat16)
    dim, page = 256, 16
    options = dict(options)
    window, keep, chunk, cap = options.get("window"), options.get("keep_first", 0), options.get("chunk"), options.get("softcap")
    generator = torch.Generator().manual_seed(heads)
    sinks = torch.randn(heads, generator=generator).cuda() if options.pop("sinks", False) else None
    slopes = torch.rand(heads, generator=generator).mul(0.05).cuda() if options.pop("slopes", False) else None
    case = paged_case(torch.bfloat16, heads, kv_heads, dim, page, ctx_lens, q_lens, seed=heads + len(ctx_lens))
    ops.portion_splits = splits
    plan = ops.attention_plan(heads, kv_heads, dim, len(ctx_lens), case["table"].shape[1], page, max(q_lens), min(q_lens), sum(q_lens), list(q_lens),
                              keep_first=keep, own_values=True, max_ctx_len=max(ctx_lens))
    assert plan.tc_portions, "the case is meant for the tensor-core kernel"
    out = torch.full_like(case["q"], float("nan"))
    options.pop("window", None)
    ops.paged_attention(case["q"], case["keys"], case["keys"], case["table"], case["q_start"], case["ctx_len"], case["seq_of"], heads, kv_heads, dim,
                        dim ** -0.5, window, out, max_q_len=max(q_lens), max_ctx_len=max(ctx_lens), min_q_len=min(q_lens), q_lens=list(q_lens),
                        sinks=sinks, slopes=slopes, **options)
    ops.check_status()
    want = []
    for (q, k, _), n in zip(case["seqs"], q_lens):
        total = len(q)
        position, key = torch.arange(total - n, total, device="cuda")[:, None], torch.arange(total, device="cuda")[None]
        hidden = key > position
        if window:
            hidden = hidden | ((position - key >= window) & (key >= keep))
        if chunk:
            hidden = hidden | (position // chunk != key // chunk)
        rows = []
        for a in range(heads):
            held = k[:, a * kv_heads // heads].double().cuda()
            score = q[total - n:, a].double().cuda() @ held.T * dim ** -0.5
            if cap:
                score = cap * torch.tanh(score / cap)
            if slopes is not None:
                score = score - slopes[a].double() * (position - key)
            score = score.masked_fill(hidden, float("-inf"))
            if sinks is not None:
                score = torch.cat([score, sinks[a].double().expand(n, 1)], dim=1)
            rows.append(torch.softmax(score, dim=1)[:, :total] @ held)
        want.append(torch.stack(rows, dim=1).reshape(n, heads * dim))
    # probabilities rounded to bfloat16 (2^-9 each, relative) and one rounding of outputs of order one, as above
    assert torch.isfinite(out).all() and (out.double() - torch.cat(want)).abs().max() < 2e-2
