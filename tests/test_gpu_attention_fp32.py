"""The 32-bit path's attention: a token's bits are the same in a prompt, alone and beside a portion, and close to float64."""

import numpy as np
import pytest
import torch

from tests.gpu_common import cuda_ops
from tests.plain import plain_model as pm
from tests.test_gpu_kernels import paged_case

pytestmark = pytest.mark.gpu
DEV = "cuda"


def rnd(*shape, seed=0):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(DEV)


def attention(ops, case, rows, q_start, ctx_len, seq_of, table, heads, kv_heads, dim, q_lens, **options):
    out = torch.full((rows.shape[0], heads * dim), float("nan"), device=DEV)
    ops.paged_attention(rows, case["keys"], case["values"], table, q_start, ctx_len, seq_of, heads, kv_heads, dim, dim ** -0.5,
                        options.pop("window", None), out, max_q_len=max(q_lens), max_ctx_len=int(ctx_len.max()), min_q_len=min(q_lens),
                        q_lens=list(q_lens), **options)
    return out


# contexts around a tile of 32 and a chunk of 64 keys; shared heads below, at and above the 16 and 64 rows of a CTA
@pytest.mark.parametrize("heads,kv_heads,dim,page", [(7, 1, 128, 16), (16, 1, 64, 16), (17, 1, 48, 5), (66, 1, 16, 8), (4, 2, 256, 16)])
@pytest.mark.parametrize("options", [{}, {"window": 40}, {"window": 40, "keep_first": 5}, {"chunk": 48}, {"softcap": 3.0, "sinks": True}])
def test_fp32_attention_gives_a_token_the_same_bits_in_a_prompt_and_alone(heads, kv_heads, dim, page, options):
    ops = cuda_ops(torch.float32)
    options = dict(options)
    if options.pop("sinks", False):
        options["sinks"] = rnd(heads, seed=9)
    ctx_lens = [1, 31, 32, 33, 63, 64, 65, 127, 128, 129, 300, 517]
    case = paged_case(torch.float32, heads, kv_heads, dim, page, ctx_lens, ctx_lens, seed=heads)
    whole = attention(ops, case, case["q"], case["q_start"], case["ctx_len"], case["seq_of"], case["table"], heads, kv_heads, dim, ctx_lens, **options)
    assert torch.isfinite(whole).all()
    # the last token of every sequence alone, in a batch of single tokens (keys on CTAs of their own) and beside a portion
    last = (case["q_start"][1:] - 1).long()
    count = len(ctx_lens)
    index = torch.arange(count + 1, dtype=torch.int32, device=DEV)
    alone = attention(ops, case, case["q"][last].contiguous(), index, case["ctx_len"], index[:count], case["table"], heads, kv_heads, dim,
                      [1] * count, **options)
    assert torch.equal(alone, whole[last])
    # lengths that the caller does not know: the shortest alone, or none at all; and rows that do not lie on 16 bytes
    for known in ({"max_q_len": 1}, {}):
        shifted = torch.empty(count * heads * dim + 1, device=DEV)
        rows = shifted[1:].view(count, heads * dim)
        rows.copy_(case["q"][last])
        out = torch.empty(count * heads * dim + 1, device=DEV)[1:].view(count, heads * dim)
        given = dict(options)
        ops.paged_attention(rows, case["keys"], case["values"], case["table"], index, case["ctx_len"], index[:count], heads, kv_heads, dim,
                            dim ** -0.5, given.pop("window", None), out, **known, **given)
        assert torch.equal(out, alone)
    rows = torch.cat([case["q"][last[:-1]], case["q"][last[-1] - 9:]]).contiguous()
    q_lens = [1] * (count - 1) + [10]
    starts = torch.tensor(np.cumsum([0] + q_lens), dtype=torch.int32, device=DEV)
    seq_of = torch.repeat_interleave(torch.arange(count), torch.tensor(q_lens)).to(torch.int32).to(DEV)
    mixed = attention(ops, case, rows, starts, case["ctx_len"], seq_of, case["table"], heads, kv_heads, dim, q_lens, **options)
    assert torch.equal(mixed[: count - 1], whole[last[:-1]]) and torch.equal(mixed[count - 1:], whole[last[-1] - 9: last[-1] + 1])
    # a warp a row
    ops.fp32_attention_form = 2
    assert torch.equal(attention(ops, case, case["q"], case["q_start"], case["ctx_len"], case["seq_of"], case["table"], heads, kv_heads, dim, ctx_lens,
                                 **options), whole)
    assert torch.equal(attention(ops, case, rows, starts, case["ctx_len"], seq_of, case["table"], heads, kv_heads, dim, q_lens, **options), mixed)
    if set(options) <= {"window"}:
        want = torch.cat([pm.causal_attention(q.double().to(DEV), k.double().to(DEV), v.double().to(DEV), options.get("window"))
                          for q, k, v in case["seqs"]]).reshape(whole.shape)
        assert (whole.double() - want).abs().max() < 2e-5


def test_fp32_attention_keeps_a_later_tokens_values_out():
    ops = cuda_ops(torch.float32)
    case = paged_case(torch.float32, 2, 1, 64, 16, [40], [40], seed=3)
    args = (case["q_start"], case["ctx_len"], case["seq_of"], case["table"], 2, 1, 64, [40])
    want = attention(ops, case, case["q"], *args)
    page = int(case["table"][0, 2])
    case["values"][page, 7] = float("inf")   # the value of position 39
    got = attention(ops, case, case["q"], *args)
    assert torch.equal(got[:39], want[:39]) and not torch.isfinite(got[39]).all()


def test_fp32_attention_takes_pages_that_do_not_lie_on_16_bytes():
    """Views into a larger array, one element behind a 16-byte border: plain loads in place of wide ones, the same bits."""
    ops = cuda_ops(torch.float32)
    heads, kv_heads, dim, lens = 6, 2, 48, [70, 1, 33]
    case = paged_case(torch.float32, heads, kv_heads, dim, 16, lens, lens, seed=5)
    shifted = dict(case)
    for name in ("keys", "values"):
        room = torch.empty(case[name].numel() + 1, device=DEV)
        shifted[name] = room[1:].view(case[name].shape)
        shifted[name].copy_(case[name])
    last = (case["q_start"][1:] - 1).long()
    index = torch.arange(len(lens) + 1, dtype=torch.int32, device=DEV)
    for which in (("keys",), ("values",), ("keys", "values")):
        moved = dict(case, **{name: shifted[name] for name in which})
        whole = [attention(ops, c, c["q"], c["q_start"], c["ctx_len"], c["seq_of"], c["table"], heads, kv_heads, dim, lens) for c in (case, moved)]
        assert torch.equal(*whole)
        alone = [attention(ops, c, c["q"][last].contiguous(), index, c["ctx_len"], index[: len(lens)], c["table"], heads, kv_heads, dim, [1] * len(lens))
                 for c in (case, moved)]
        assert torch.equal(*alone) and torch.equal(alone[0], whole[0][last])


def test_fp32_attention_reads_lengths_that_kernels_of_the_stream_just_wrote():
    """One request that grows by a token a round: its length is written by a kernel, the store of its newest key and value and
    the attention follow directly, round after round."""
    ops = cuda_ops(torch.float32)
    heads, kv_heads, dim, page, n = 6, 2, 64, 16, 130
    case = paged_case(torch.float32, heads, kv_heads, dim, page, [n], [n], seed=8)
    want = attention(ops, case, case["q"], case["q_start"], case["ctx_len"], case["seq_of"], case["table"], heads, kv_heads, dim, [n])
    q, k, v = (t.to(DEV).reshape(n, -1).contiguous() for t in case["seqs"][0])
    keys, values = torch.full_like(case["keys"], float("nan")), torch.full_like(case["values"], float("nan"))
    table = case["table"].long()[0]
    slots = (table[torch.arange(n, device=DEV) // page] * page + torch.arange(n, device=DEV) % page).to(torch.int32)
    q_start, seq_of = torch.tensor([0, 1], dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    ctx_len, out = torch.zeros(1, dtype=torch.int32, device=DEV), torch.full((n, heads * dim), float("nan"), device=DEV)
    torch.cuda.synchronize()
    for i in range(n):
        ctx_len.add_(1)
        ops.kv_write(k[i: i + 1], v[i: i + 1], keys, values, slots[i: i + 1])
        ops.paged_attention(q[i: i + 1], keys, values, case["table"], q_start, ctx_len, seq_of, heads, kv_heads, dim, dim ** -0.5, None,
                            out[i: i + 1], max_q_len=1, min_q_len=1)
    assert torch.equal(out, want)


def test_fp32_attention_of_more_sequences_than_a_grid_has_places():
    ops = cuda_ops(torch.float32)
    count, heads, dim, page = 65600, 2, 16, 4
    keys, values = rnd(count, page, 1, dim, seed=1), rnd(count, page, 1, dim, seed=2)
    q = rnd(count, heads * dim, seed=3)
    table = torch.randperm(count, generator=torch.Generator().manual_seed(4)).to(torch.int32).to(DEV).view(count, 1)
    ctx_len = torch.randint(1, page + 1, (count,), generator=torch.Generator().manual_seed(5)).to(torch.int32).to(DEV)
    index = torch.arange(count + 1, dtype=torch.int32, device=DEV)
    case = {"keys": keys, "values": values}
    whole = attention(ops, case, q, index, ctx_len, index[:count], table, heads, 1, dim, [1] * count)
    few = attention(ops, case, q[-300:].contiguous(), index[:301].clone(), ctx_len[-300:].contiguous(), index[:300], table[-300:].contiguous(), heads, 1,
                    dim, [1] * 300)
    assert torch.isfinite(whole).all() and torch.equal(whole[-300:], few)


# the batches that a rule sends to a warp a row, beside ones just short of it: many pairs of one or two heads, few keys, many short entries
@pytest.mark.parametrize("heads,kv_heads,q_lens,ctx_lens", [
    (32, 32, [1] * 32, list(range(1, 33))), (32, 32, [1] * 3, [5, 128, 33]), (32, 32, [1] * 4, [5, 128, 33, 64]), (32, 32, [1] * 7, [5, 256, 33, 64, 65, 1, 127]),
    (32, 32, [1] * 8, [5, 256, 33, 64, 65, 1, 127, 31]), (16, 8, [1] * 128, [300 - i for i in range(128)]),
    (6, 2, [1] * 3, [8, 3, 1]), (6, 2, [1] * 3, [9, 3, 1]), (4, 4, [2, 5, 1, 3], [70, 5, 1, 33]), (4, 2, [3, 3], [40, 3]), (4, 2, [3, 4], [40, 4])])
def test_fp32_attention_by_either_form_gives_the_same_bits(heads, kv_heads, q_lens, ctx_lens):
    ops = cuda_ops(torch.float32)
    case = paged_case(torch.float32, heads, kv_heads, 48, 16, ctx_lens, q_lens, seed=heads + len(q_lens))
    args = (case["q"], case["q_start"], case["ctx_len"], case["seq_of"], case["table"], heads, kv_heads, 48, q_lens)
    outs = []
    for form in (0, 1, 2):
        ops.fp32_attention_form = form
        outs.append(attention(ops, case, *args))
    assert torch.isfinite(outs[0]).all() and torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])


# windows and kept keys whose chunks meet, touch and lie apart; the chunks on CTAs of their own against one warp that walks them all
@pytest.mark.parametrize("options", [{"window": 1}, {"window": 64}, {"window": 65, "keep_first": 1}, {"window": 100, "keep_first": 64}, {"window": 30, "keep_first": 130},
                                     {"window": 500, "keep_first": 65}, {"chunk": 64}, {"chunk": 200}])
def test_fp32_single_tokens_walk_the_chunks_that_a_window_reaches(options):
    ops = cuda_ops(torch.float32)
    heads, kv_heads, dim, ctx_lens = 6, 2, 48, [1, 63, 64, 65, 128, 129, 190, 193, 257, 700, 1025]
    case = paged_case(torch.float32, heads, kv_heads, dim, 16, ctx_lens, [1] * len(ctx_lens), seed=11)
    wide = torch.full((len(ctx_lens), 160), -1, dtype=torch.int32, device=DEV)   # tables far wider than what is held
    wide[:, : case["table"].shape[1]] = case["table"]
    outs = []
    for form, table in ((2, case["table"]), (1, case["table"]), (1, wide)):
        ops.fp32_attention_form = form
        outs.append(attention(ops, case, case["q"], case["q_start"], case["ctx_len"], case["seq_of"], table, heads, kv_heads, dim, [1] * len(ctx_lens), **options))
    assert torch.isfinite(outs[0]).all() and torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
