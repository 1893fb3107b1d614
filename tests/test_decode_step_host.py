"""The one-kernel decode step's exchanges, walked through on the host: CTAs hand values on as words that carry the number of the
exchange, and a reader that comes after its words were written again would wait for a number that is gone."""

import ctypes
from types import SimpleNamespace

import pytest
import torch

from shrike_b200.cache.manager import CacheManager, KVGroupSpec
from shrike_b200.engine.batch import BatchBuilder, StepEntry
from shrike_b200.ops import build
from shrike_b200.ops.decode_step import DecodeStep

CTAS = 148
WIDTHS = {   # width, heads, kv heads, head size, intermediate
    "0.5b": (896, 14, 2, 64, 4864), "1.5b": (1536, 12, 2, 128, 8960), "3b": (2048, 16, 2, 128, 11008), "7b": (3584, 28, 4, 128, 18944),
    "one kv head": (384, 8, 1, 64, 1280), "every head its own": (512, 4, 4, 128, 1280),
}
ROWS = (1, 2, 4, 8)   # bits of a CTA's role: it has rows (units) of q/k/v, output, gate/up, down
READS = 16            # it reads the residual words in part 0


def roles_of(sizes, ctas=CTAS):
    roles = (ctypes.c_int * ctas)()
    assert build.decode_step_library().shrike_decode_step_roles(ctas, *sizes, roles) == 0
    return list(roles)


def cta_of_row(sizes, ctas=CTAS):
    """Which CTA writes a row of q/k/v: equal shares, rounded up to four."""
    _width, heads, kv_heads, dim, _inter = sizes
    each = -(-(-(-(heads + 2 * kv_heads) * dim // ctas)) // 4) * 4
    return lambda row: row // each


def walk(sizes, roles, tokens, runs, slow, layers=3):
    """Runs the layers' exchanges with CTA `slow` held up: it goes one step on only when no other can.  Returns the CTAs that
    found a word already written again, and whether all came to the end."""
    _width, heads, kv_heads, dim, _inter = sizes
    ctas, group, owner = len(roles), heads // kv_heads, cta_of_row(sizes)
    pairs = [(t, h, r) for t in range(tokens) for h in range(kv_heads) for r in range(runs)]
    assert len(pairs) <= ctas
    words = {name: [-1] * ctas for name in ("residual", "qkv", "sums", "heads", "activation")}
    has = [[c for c in range(ctas) if roles[c] & bit] for bit in ROWS]

    def qkv_owners(h, last):
        rows = list(range(h * group * dim, (h + 1) * group * dim))
        if last:   # the run that holds the step's own key and value
            for plane in (0, 1):
                first = (heads + plane * kv_heads + h) * dim
                rows += range(first, first + dim)
        return sorted({owner(row) for row in rows})

    def cta(c):
        def put(name, number):
            words[name][c] = number

        if roles[c] & 2:
            put("residual", 0)
        for layer in range(layers):
            number = 2 * layer
            if roles[c] & READS:
                yield "residual", has[1], number
            if roles[c] & 1:
                put("qkv", number)
            if c < len(pairs):
                _t, h, r = pairs[c]
                yield "qkv", qkv_owners(h, r == runs - 1), number
                if runs > 1:
                    put("sums", number)
                    yield "sums", range(c - r, c - r + runs), number
                put("heads", number)
            yield "heads", range(len(pairs)), number
            if roles[c] & 2:
                put("residual", number + 1)
            yield "residual", has[1], number + 1
            put("activation", number + 1)
            if roles[c] & 8:
                yield "activation", range(ctas), number + 1
                put("residual", number + 2)
        return

    agents = {c: cta(c) for c in range(ctas)}
    waits = {}
    for c in range(ctas):
        if c != slow:
            waits[c] = next(agents[c], None)
    missed, held = [], True   # `held`: the slow one has not begun
    while waits and not missed:
        moved = False
        for c in sorted(waits):
            if c == slow:
                continue
            while waits[c] is not None and all(words[waits[c][0]][o] == waits[c][2] for o in waits[c][1]):
                moved = True
                waits[c] = next(agents[c], None)
            if waits[c] is None:
                del waits[c]
            elif any(words[waits[c][0]][o] > waits[c][2] for o in waits[c][1]):
                missed.append(c)
        if moved:
            continue
        if held:
            held = False
            waits[slow] = next(agents[slow], None)
        elif slow in waits and all(words[waits[slow][0]][o] == waits[slow][2] for o in waits[slow][1]):
            waits[slow] = next(agents[slow], None)
        elif slow in waits and any(words[waits[slow][0]][o] > waits[slow][2] for o in waits[slow][1]):
            missed.append(slow)
        else:
            break
        if slow in waits and waits[slow] is None:
            del waits[slow]
    return missed, not waits


@pytest.mark.parametrize("tokens,runs", [(1, 1), (1, 16), (2, 3)])
@pytest.mark.parametrize("key", list(WIDTHS))
def test_no_cta_finds_its_words_written_again_whichever_is_held_up(key, tokens, runs):
    sizes = WIDTHS[key]
    roles = roles_of(sizes)
    pairs = tokens * runs * sizes[2]
    without = [c for c in range(CTAS) if not roles[c] & 1]
    assert all(role & 4 for role in roles)   # every CTA has a gated unit: most of the order rests on it
    for slow in sorted({0, pairs - 1, pairs, CTAS // 2, CTAS - 1, *without[:1], *without[-1:]}):
        assert walk(sizes, roles, tokens, runs, slow) == ([], True), slow


def test_a_reader_of_the_residual_that_writes_no_rows_would_miss_it():
    """What the roles are for: with every CTA reading the residual in part 0, one without q/k/v rows and without a pair finds the
    next number there when it is held up."""
    sizes = WIDTHS["0.5b"]
    roles = [role | READS for role in roles_of(sizes)]
    idle = [c for c in range(CTAS) if not roles[c] & 1]
    assert idle and walk(sizes, roles, 1, 1, idle[0]) == ([idle[0]], False)


def held(manager, count):
    cache = manager.open()
    manager.append(cache, 0, count)
    return cache


@pytest.mark.parametrize("groups", [1, 2])
def test_entries_that_share_a_page_with_a_new_token_are_left_to_the_layers_one_by_one(groups):
    """Such an entry may read the key that another of the same step stores: the layers one by one store all keys first."""
    manager = CacheManager([KVGroupSpec((g,), 2, 64, None) for g in range(groups)], 4, 64, 16)
    builder = BatchBuilder(4, groups, "cpu", None)
    builder.watches_pages = True
    step = object.__new__(DecodeStep)
    step.ops = SimpleNamespace(whole_steps=True)
    step._most_keys, step._refused = {n: 1000 for n in range(1, 9)}, False
    a, b, c = held(manager, 12), held(manager, 9), held(manager, 12)

    def taken(*entries, pad_to=0):
        staged = builder.stage([StepEntry(cache, [1] * count, start, [0]) for cache, start, count in entries], pad_to=pad_to)
        assert step.takes(staged) == step.takes(builder.context(staged))   # what a captured step goes by, and the step
        return step.takes(staged)

    assert taken((a, 11, 1)) and taken((a, 11, 1), (b, 8, 1), (c, 11, 1)) and taken((a, 11, 1), (b, 8, 1), pad_to=8)
    assert not taken((a, 10, 1), (a, 11, 1))                    # neighbours on one page
    assert not taken((a, 8, 1), (a, 7, 1))                      # across a page's border
    assert not taken((a, 3, 1), (b, 8, 1), (a, 11, 1))          # pages apart, which the later one reads all the same
    assert not taken((a, 11, 1), (a, 11, 1))
    assert not taken((a, 10, 2), (b, 8, 1))                     # no step of single tokens
    shared = held(manager, 4)                                   # another request, whose first page is a's
    for table, other in zip(shared.tables, a.tables):
        table.pages[0] = other.pages[0]
    assert taken((a, 11, 1), (shared, 3, 1)) is False and taken((b, 8, 1), (shared, 3, 1))
    builder.watches_pages = False                               # a runner asks only where it matters
    assert taken((a, 11, 1)) and not taken((a, 11, 1), (b, 8, 1))
    builder.watches_pages = True
    many = [(held(manager, 1), 0, 1) for _ in range(9)]
    assert taken(*many[:8]) and not taken(*many)
    assert torch.equal(builder.build([StepEntry(a, [1], 11, [0])]).ctx_len, torch.tensor([12], dtype=torch.int32))


def test_the_longest_context_a_step_is_served_with_follows_the_sizes():
    """Within a quarter of where the two ways were measured to be equal (at 148 SMs), fewer keys with more sequences where kv heads
    are many, and none where the sizes themselves are not served."""
    keys = build.decode_step_library().shrike_decode_step_keys
    for sizes, measured in ((WIDTHS["1.5b"], {1: 13700, 2: 13400, 3: 11800, 4: 11000}), (WIDTHS["3b"], {1: 13000, 2: 12800, 3: 11900, 4: 9500}),
                            (WIDTHS["7b"], {1: 11000, 2: 12000}), (WIDTHS["0.5b"], {1: 25300, 2: 31000}),
                            ((896, 14, 14, 64, 4864), {1: 16700, 2: 6900, 3: 3460, 4: 1580}), ((512, 8, 8, 64, 1280), {5: 3260, 8: 1720}),
                            ((1536, 12, 12, 128, 8960), {1: 14500, 2: 3050, 3: 1480})):
        for tokens, equal in measured.items():
            assert 0.75 * equal <= keys(tokens, 28, *sizes) <= 1.15 * equal, (sizes, tokens, keys(tokens, 28, *sizes))
    for heads in (6, 12):
        line = [keys(tokens, 28, 1536, 12, heads, 128, 8960) for tokens in (1, 2, 3, 4)]
        assert line == sorted(line, reverse=True) and 4 * line[3] < line[0], line
    assert all(0 <= keys(tokens, 2, width, heads, heads, 64, 1280) <= 65536 for tokens in range(1, 9)
               for width, heads in ((256, 4), (384, 6), (512, 2)))
    assert keys(5, 28, *WIDTHS["1.5b"]) == keys(3, 28, *WIDTHS["7b"]) == keys(9, 24, *WIDTHS["0.5b"]) == keys(1, 200, *WIDTHS["0.5b"]) == 0


def test_a_context_beyond_that_is_left_to_the_layers_one_by_one():
    manager = CacheManager([KVGroupSpec((0,), 2, 64, None)], 4, 64, 16)
    builder = BatchBuilder(4, 1, "cpu", None)
    builder.watches_pages = True
    step = object.__new__(DecodeStep)
    step.ops, step._refused, step._most_keys = SimpleNamespace(whole_steps=True), False, {1: 30, 2: 20}
    a, b = held(manager, 40), held(manager, 9)
    taken = lambda *starts: step.takes(builder.stage([StepEntry(c, [1], start, [0]) for c, start in zip((a, b), starts)]))
    assert taken(29) and not taken(30) and taken(19, 8) and not taken(20, 8)
