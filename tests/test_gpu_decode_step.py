"""All layers of a decode step as one kernel, against the layer-by-layer path and the plain implementation."""

import ctypes

import numpy as np
import pytest
import torch

from shrike_b200.config import parse_config
from shrike_b200.engine.batch import StepEntry
from shrike_b200.engine.runner import ModelRunner
from shrike_b200.ops import build
from shrike_b200.ops.cuda_ops import KernelError
from shrike_b200.weights.random_init import random_tensors
from tests.gpu_common import TOL, cuda_ops
from tests.helpers import random_tokens
from tests.plain import plain_model as pm

pytestmark = pytest.mark.gpu


def shape(width, heads, kv_heads, dim, inter, layers=2):
    return dict(architectures=["Qwen2ForCausalLM"], hidden_size=width, intermediate_size=inter, num_hidden_layers=layers,
                num_attention_heads=heads, num_key_value_heads=kv_heads, head_dim=dim, vocab_size=777, rms_norm_eps=1e-6,
                rope_theta=1000000.0, tie_word_embeddings=True, max_position_embeddings=32768, eos_token_id=776)


# rows of a CTA of one and two tiles of 16, ring stages that end short, rows of the activation that do not fit and come in halves
SHAPES = {
    "d64": shape(896, 14, 2, 64, 4864),
    "d64 one kv head": shape(384, 8, 1, 64, 1280, layers=3),
    "d64 sixteen to a kv head": shape(256, 16, 1, 64, 1408),
    "d128": shape(1536, 12, 2, 128, 8960),
    "d128 every head its own": shape(512, 4, 4, 128, 1280),
    "d128 wide": shape(3584, 28, 4, 128, 18944, layers=1),
}


def decode(raw, lengths, page_size, whole, steps=3):
    """Logits of `steps` decode steps of sequences that hold `lengths` tokens, the pools after them, launches of the last step."""
    config = parse_config(raw)
    weights = {k: (v.to(torch.bfloat16) if v.dim() >= 2 else v) for k, v in random_tensors(config, 3, "cuda", torch.float32).items()}
    ops = cuda_ops(torch.bfloat16)
    pages = sum(-(-(n + steps) // page_size) for n in lengths)
    runner = ModelRunner(config, weights, ops, "cuda", "bfloat16", page_size=page_size, num_pages=pages, max_slots=len(lengths))
    sequences = [random_tokens(raw["vocab_size"], n + steps, 50 + i) for i, n in enumerate(lengths)]
    caches = [runner.cache.open() for _ in lengths]
    for cache, ids, n in zip(caches, sequences, lengths):
        if n:
            runner.cache.append(cache, 0, n)
            runner.step([StepEntry(cache, ids[:n], 0, [])])
    ops.whole_steps = whole
    rows = []
    for step in range(steps):   # eager, captured, replayed
        for cache, n in zip(caches, lengths):
            runner.cache.append(cache, n + step, 1)
        before = ops.launches
        out = runner.step([StepEntry(cache, [ids[n + step]], n + step, [0]) for cache, ids, n in zip(caches, sequences, lengths)])
        launches = ops.launches - before
        rows.append(out.float().cpu().numpy().copy())
    ops.check_status()
    return np.stack(rows), [pool.float().cpu() for pool in runner.storage.kv], launches, weights, sequences


# runs of one, two and more tiles of keys (64 or 128), the new key first, last and alone in its tile, lengths that share no page border
@pytest.mark.parametrize("page_size", [16, 5])
@pytest.mark.parametrize("key,lengths", [
    ("d64", (97,)), ("d64", (127, 128, 129, 0)), ("d64", (1, 255, 511, 30, 2)), ("d64 one kv head", (63, 700, 5, 64, 128, 256, 17, 1)),
    ("d64 sixteen to a kv head", (40, 2600)), ("d128", (0,)), ("d128", (63, 64, 65)), ("d128", (517, 127)), ("d128 every head its own", (3, 700, 128)),
    ("d128 wide", (77, 1300))])
def test_a_step_as_one_kernel_gives_the_logits_and_cache_rows_of_the_layers_one_by_one(key, lengths, page_size):
    raw = SHAPES[key]
    got, got_pools, launches, weights, sequences = decode(raw, lengths, page_size, True)
    want, want_pools, one_by_one, _, _ = decode(raw, lengths, page_size, False)
    assert launches < 6 < one_by_one, "the step was meant to run as one kernel"
    scale = max(1.0, float(np.abs(want).max()))
    assert np.isfinite(got).all() and np.abs(got - want).max() <= TOL["bfloat16"] * scale
    for a, b in zip(got_pools, want_pools):   # rows of earlier tokens the same, the steps' own within bfloat16's rounding of like sums
        assert (a - b).abs().max() <= TOL["bfloat16"] * max(1.0, float(b.abs().max()))
    for i, (ids, n) in enumerate(zip(sequences, lengths)):
        plain = pm.forward(raw, weights, ids, dtype=torch.float64, rounding=pm.ROUNDING_POINTS).cpu().numpy()[n:]
        assert np.abs(got[:, i] - plain).max() <= TOL["bfloat16"] * max(1.0, float(np.abs(plain).max())), i


def test_other_sizes_and_more_sequences_keep_the_layers_one_by_one():
    ops = cuda_ops(torch.bfloat16)
    for raw, tokens, served in (("d64", 4, True), ("d64", 8, False), ("d128", 4, True), ("d128", 5, False), ("d128 wide", 2, True),
                                ("d128 wide", 3, False), ("d64 one kv head", 8, True)):
        config = parse_config(SHAPES[raw])
        mixer, ffn = config.layers[0].mixer, config.layers[0].feed_forward
        from shrike_b200.ops.build import decode_step_library
        assert bool(decode_step_library().shrike_decode_step_serves(tokens, len(config.layers), mixer.width, mixer.num_heads, mixer.num_kv_heads,
                                                                    mixer.head_dim, ffn.intermediate)) == served
    for raw in (shape(448, 7, 1, 64, 1280), shape(512, 4, 2, 128, 1376), shape(512, 32, 16, 32, 1280), dict(SHAPES["d64"], use_sliding_window=True,
                sliding_window=64, max_window_layers=0)):
        config = parse_config(raw)
        weights = {k: (v.to(torch.bfloat16) if v.dim() >= 2 else v) for k, v in random_tensors(config, 3, "cuda", torch.float32).items()}
        runner = ModelRunner(config, weights, ops, "cuda", "bfloat16", page_size=16, num_pages=8, max_slots=2)
        assert runner.model._whole_step is None


def runner_of(raw, requests, page_size=16, tokens=700, ops=None):
    config = parse_config(raw)
    weights = {k: (v.to(torch.bfloat16) if v.dim() >= 2 else v) for k, v in random_tensors(config, 3, "cuda", torch.float32).items()}
    return ModelRunner(config, weights, ops or cuda_ops(torch.bfloat16), "cuda", "bfloat16", page_size=page_size,
                       num_pages=requests * -(-tokens // page_size), max_slots=requests)


def opened(runner, ids, count):
    """A request whose cache holds the first `count` of `ids` and has room for one token more."""
    cache = runner.cache.open()
    if count:
        runner.cache.append(cache, 0, count)
        runner.step([StepEntry(cache, ids[:count], 0, [])])
    runner.cache.append(cache, count, 1)
    return cache


def test_nothing_is_read_beyond_a_sequences_row_of_the_block_table():
    """A context longer than the row: keys beyond it count as zeros, whatever stands in the next sequence's row."""
    raw, lengths = SHAPES["d64"], (230, 90, 150)
    runner = runner_of(raw, 3, page_size=5)
    sequences = [random_tokens(raw["vocab_size"], n + 1, 50 + i) for i, n in enumerate(lengths)]
    caches = [opened(runner, ids, n) for ids, n in zip(sequences, lengths)]
    seen = []
    with torch.inference_mode():
        for other in (1, 2):   # the row behind the first one's
            entries = [StepEntry(caches[i], [sequences[i][-1]], lengths[i], [0]) for i in (0, other)]
            ctx = runner.builder.build(entries)
            view = ctx.groups[0]
            view.max_blocks = 32   # of the 47 blocks that the first one's context spans
            view.block_table = view.block_table[:, :32].contiguous()
            before = runner.ops.launches
            logits, _ = runner._run(ctx, False)
            assert runner.ops.launches - before < 6
            seen.append(logits[0].float().cpu().numpy().copy())
    runner.ops.check_status()
    assert np.isfinite(seen[0]).all() and np.array_equal(seen[0], seen[1])


def test_where_the_device_will_not_run_all_ctas_together_the_layers_run_one_by_one():
    raw, n = SHAPES["d64"], 40
    ids = random_tokens(raw["vocab_size"], n + 1, 9)
    seen = []
    for refused in (False, True):
        runner = runner_of(raw, 1)
        program = runner.model._whole_step
        if refused:
            runner.ops.whole_steps = True
            program.lib = type("Refuses", (), {"__getattr__": lambda _, name, real=program.lib: getattr(real, name),
                                               "shrike_decode_step": staticmethod(lambda args, stream: program.NOT_TOGETHER)})()
        else:
            runner.ops.whole_steps = False
        cache = opened(runner, ids, n)
        for _ in range(3):   # eager, captured, replayed
            seen.append(runner.step([StepEntry(cache, [ids[n]], n, [0])]).float().cpu().numpy().copy())
        runner.ops.check_status()
    assert all(np.array_equal(seen[0], other) for other in seen[1:])


def test_a_wait_that_runs_out_ends_the_step_with_its_code_and_the_next_step_is_right():
    """A build whose waits for other CTAs' words give up at the first look that finds them missing: the kernel runs to its end,
    says so in the status word, and leaves the exchanges fit for the next launch."""
    raw, n = SHAPES["d64"], 300
    ids = random_tokens(raw["vocab_size"], n + 1, 9)
    runner = runner_of(raw, 1)
    runner.use_graphs = False
    program = runner.model._whole_step
    cache = opened(runner, ids, n)
    patient, impatient = program.lib, build.load_library("shrike_decode_step_impatient", ["decode_step.cu"], {"SHRIKE_STEP_POLL_LIMIT": 1})
    impatient.shrike_decode_step.argtypes, impatient.shrike_decode_step.restype = patient.shrike_decode_step.argtypes, ctypes.c_int

    class Impatient:
        shrike_decode_step = staticmethod(impatient.shrike_decode_step)

        def __getattr__(self, name):
            return getattr(patient, name)

    def step():
        return runner.step([StepEntry(cache, [ids[n]], n, [0])]).float().cpu().numpy().copy()

    want = step()
    runner.ops.check_status()
    for _ in range(2):
        program.lib = Impatient()
        step()
        with pytest.raises(KernelError, match="wait for another CTA's values ran out"):
            runner.ops.check_status()
        program.lib = patient
        assert np.array_equal(step(), want)
        runner.ops.check_status()


def follow(raw, seed, whole, script, lengths):
    """Logits of a script's steps on one runner, and the launches of each.  A step is a list of (request, its count of tokens);
    None: the cache pool is replaced by a copy."""
    config = parse_config(raw)
    weights = {k: (v.to(torch.bfloat16) if v.dim() >= 2 else v) for k, v in random_tensors(config, seed, "cuda", torch.float32).items()}
    ops = cuda_ops(torch.bfloat16)
    room = [n + 200 for n in lengths]
    runner = ModelRunner(config, weights, ops, "cuda", "bfloat16", page_size=16, num_pages=sum(-(-n // 16) for n in room), max_slots=len(lengths))
    ids = [random_tokens(raw["vocab_size"], n, 70 + i) for i, n in enumerate(room)]
    ops.whole_steps = whole
    caches, at, rows, launches = [], list(lengths), [], []
    for i, n in enumerate(lengths):
        caches.append(runner.cache.open())
        runner.cache.append(caches[i], 0, room[i])
        runner.step([StepEntry(caches[i], ids[i][:n], 0, [])])
    for step in script:
        if step is None:
            held = runner.storage
            pages = [group.shape[2] for group in held.kv]
            runner.storage = runner.builder.storage = type(held)(held.groups, 16, pages, {}, len(lengths), torch.bfloat16, runner.device)
            for new, old in zip(runner.storage.kv, held.kv):
                new.copy_(old)
                old.fill_(float("nan"))
            runner._graphs.clear()   # a captured step belongs to the pool it was captured with
            continue
        before = ops.launches
        out = runner.step([StepEntry(caches[i], ids[i][at[i]: at[i] + count], at[i], [count - 1]) for i, count in step])
        launches.append(ops.launches - before)
        rows.append(out.float().cpu().numpy().copy())
        for i, count in step:
            at[i] += count
    ops.check_status()
    return rows, launches


def singles(*requests):
    return [(i, 1) for i in requests]


@pytest.mark.parametrize("seed", [3, 4])   # the second engine of a process finds what the first has freed
def test_steps_of_different_counts_and_kinds_in_one_engine(seed):
    """The words that CTAs exchange lie elsewhere for every count of sequences, and the numbers in them go on through captured
    launches, prompts, steps that the layers take one by one and a new cache pool."""
    raw, lengths = SHAPES["d64"], (40, 333, 90, 1, 700, 128, 127, 64, 500, 12)
    script = [singles(0)] * 3 + [singles(0, 1, 2, 3)] * 3 + [singles(2, 3)] * 2 + [[(4, 70), (0, 1), (1, 1)]]
    script += [singles(*range(9))] * 2 + [singles(0, 1, 2, 3), singles(5), singles(8, 9, 0), singles(4, 5, 6, 7, 8)] * 2
    script += [singles(6), None] + [singles(0), singles(3, 2, 1, 0), singles(4, 9)] * 3 + [[(7, 33)], singles(7), singles(4)]
    got, launches = follow(raw, seed, True, script, lengths)
    want, _ = follow(raw, seed, False, script, lengths)
    steps = [step for step in script if step is not None]
    for step, a, b, count in zip(steps, got, want, launches):
        assert np.isfinite(a).all() and np.abs(a - b).max() <= TOL["bfloat16"] * max(1.0, float(np.abs(b).max())), step
        assert (count < 6) == (len(step) <= 5 and max(n for _, n in step) == 1), (step, count)


@pytest.mark.parametrize("lengths", [(9000,), (20000, 130), (3, 12000, 700, 64)])
def test_long_contexts(lengths):
    """Runs of many tiles of keys, up to the contexts that are left to the layers one by one."""
    raw = SHAPES["d64"]
    script = [singles(*range(len(lengths)))] * 3
    got, launches = follow(raw, 3, True, script, lengths)
    want, _ = follow(raw, 3, False, script, lengths)
    assert max(launches) < 6
    for a, b in zip(got, want):
        assert np.isfinite(a).all() and np.abs(a - b).max() <= TOL["bfloat16"] * max(1.0, float(np.abs(b).max()))


def test_a_batch_that_grows_beyond_the_longest_context_goes_on_layer_by_layer():
    """Eight kv heads, eight sequences: the line lies low.  Captured launches of one way are not replayed for the other."""
    raw = shape(512, 8, 8, 64, 1280)
    line = build.decode_step_library().shrike_decode_step_keys(8, 2, 512, 8, 8, 64, 1280)
    lengths = (line - 4, 300, 20, 1, 130, 64, 800, 500)
    script = [singles(*range(8))] * 8
    got, launches = follow(raw, 3, True, script, lengths)
    want, _ = follow(raw, 3, False, script, lengths)
    assert 500 < line < 5000 and [count < 6 for count in launches] == [True] * 4 + [False] * 4
    for a, b in zip(got, want):
        assert np.isfinite(a).all() and np.abs(a - b).max() <= TOL["bfloat16"] * max(1.0, float(np.abs(b).max()))
