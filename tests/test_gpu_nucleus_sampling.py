"""Nucleus sampling over a cluster of CTAs: the token that the definition gives, at the sizes where a row is cut differently."""

import math

import pytest
import torch

from shrike_b200.sampling.rng import gumbel_noise_host
from tests.gpu_common import cuda_ops
from tests.plain import plain_model as pm

pytestmark = pytest.mark.gpu
DEV = "cuda"


def rnd(*shape, seed=0):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(DEV)


# rows of fewer entries than a cluster's threads, exactly as many, one more; a real vocabulary; more than fits a cluster
@pytest.mark.parametrize("vocab", [1, 5, 127, 1023, 1024, 1025, 9000, 152064, 420000])
def test_nucleus_sampling_draws_the_token_the_definition_gives(vocab):
    ops = cuda_ops(torch.float32)
    rows = 6
    logits = rnd(rows, vocab, seed=vocab) * 2.0
    temperature = [0.8, 1.0, 0.5, 2.0, 0.8, 0.0]
    top_p = [0.95, 0.5, 0.9, 0.99, 1e-6, 0.5]
    seeds = [11 + 1000003 * r for r in range(rows)]
    out = torch.full((rows,), -1, dtype=torch.int32, device=DEV)
    ops.sample(logits, torch.tensor(temperature, device=DEV), torch.tensor(top_p, device=DEV), torch.tensor(seeds, dtype=torch.int64, device=DEV), out)
    ops.check_status()
    host = logits.cpu()
    assert int(out[5]) == int(host[5].argmax())
    for r in range(rows - 1):
        probs = pm.softmax_with_temperature(host[r], temperature[r])
        score = host[r].double() / temperature[r] + torch.from_numpy(gumbel_noise_host(seeds[r], vocab)).double()
        # a float32 sum of the mass is good to about 1e-5: the kept set lies between the sets of top_p -+ that
        sets = [pm.top_p_keep(probs, min(max(top_p[r] + d, 1e-9), 1.0)) for d in (-1e-5, 1e-5)]
        allowed = {int(torch.where(kept, score, torch.tensor(-math.inf, dtype=torch.float64)).argmax()) for kept in sets}
        assert int(out[r]) in allowed, (r, int(out[r]), allowed)


# one token has all of the mass in 32 bits: it alone is kept, also where logits over a tiny temperature no longer tell tokens
# apart (10 / 2e-38 is infinite); all of the mass on two equal logits; both forms of the kernel
@pytest.mark.parametrize("vocab", [5, 1025, 152064, 420000])
def test_nucleus_of_tokens_that_hold_all_of_the_mass(vocab):
    ops = cuda_ops(torch.float32)
    temperature = [2e-38, 1e-9, 1e-3, 0.5, 2e-38, 1e-9]
    top_p = [0.5, 0.95, 0.999, 0.9, 1e-6, 0.9]
    rows, best = len(temperature), vocab - 2
    logits = 10.0 + rnd(rows, vocab, seed=vocab).abs().clamp(max=8.0)
    logits[:, best] = 19.0
    logits[3, best] = 1000.0
    logits[5, 1] = 19.0
    out = torch.full((rows,), -1, dtype=torch.int32, device=DEV)
    for seed in range(4):
        seeds = torch.arange(rows, dtype=torch.int64, device=DEV) + 100 * seed
        ops.sample(logits, torch.tensor(temperature, device=DEV), torch.tensor(top_p, device=DEV), seeds, out)
        ops.check_status()
        assert out[:5].tolist() == [best] * 5 and int(out[5]) in (1, best)


# around the vocabularies and batches from which a row is a cluster's and not a block's: a row's token does not depend on which
@pytest.mark.parametrize("vocab,sizes", [(1535, (1, 8)), (1536, (1, 8, 9)), (2049, (8, 9)), (4095, (8, 9)), (4096, (8, 128, 129)), (11999, (128, 129)),
                                         (12000, (1, 129))])
def test_nucleus_sampling_by_a_cluster_or_a_block_draws_the_same_token(vocab, sizes):
    ops = cuda_ops(torch.float32)
    rows = max(sizes) + 1
    logits = rnd(rows, vocab, seed=vocab) * 2.0
    temperature = 0.5 + torch.rand(rows, generator=torch.Generator().manual_seed(1)).to(DEV)
    top_p = torch.rand(rows, generator=torch.Generator().manual_seed(2)).clamp(0.05, 0.99).to(DEV)
    seeds = torch.arange(rows, dtype=torch.int64, device=DEV) * 1000003 + 7
    outs = []
    for count in sizes:
        out = torch.full((count,), -1, dtype=torch.int32, device=DEV)
        ops.sample(logits[:count].contiguous(), temperature[:count].contiguous(), top_p[:count].contiguous(), seeds[:count].contiguous(), out)
        outs.append(out)
    ops.check_status()
    probs = torch.softmax(logits.double() / temperature.double()[:, None], -1)
    for out in outs:
        assert torch.equal(out[: min(sizes)], outs[0][: min(sizes)]) and torch.equal(out, outs[-1][: len(out)])
        # a kept token: the mass above it is less than top_p (float32 sums: 1e-5)
        mine = probs[: len(out)].gather(1, out.long()[:, None])
        above = torch.where(probs[: len(out)] > mine, probs[: len(out)], torch.zeros((), dtype=torch.float64, device=DEV)).sum(1)
        assert (above < top_p[: len(out)].double() + 1e-5).all()


# around those from which two threads share a place's entries
@pytest.mark.parametrize("vocab,sizes", [(5999, (12, 13)), (6000, (12, 13)), (29999, (12, 13, 64)), (30000, (1, 64, 65)), (89999, (64, 65)), (90000, (12, 65))])
def test_nucleus_sampling_by_one_or_two_threads_a_place_draws_the_same_token(vocab, sizes):
    test_nucleus_sampling_by_a_cluster_or_a_block_draws_the_same_token(vocab, sizes)
