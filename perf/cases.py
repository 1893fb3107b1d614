"""The work whose speed is followed: steps of the engine on random weights of the package's own shapes.

A case is one call of `ModelRunner.step`, the one path to the model that generation, trace replay and the benchmark
all take: entries of (a request's cache, its next tokens, the position of the first, the wanted places) in, float32
logits out, keys and values (or recurrent states) written to the cache.  The fields of a case:

  shape    a file of `shrike_b200/shapes`; dtype: the engine's type
  kind     "decode":  `batch` requests that hold about `context` tokens each take one token more, all sampled
           "prefill": one prompt of `tokens` tokens, a new request every pass, the last token's logits
           "mixed":   a portion of `tokens` tokens of a prompt that has `context` tokens behind it, and `batch`
                      requests of up to `context` tokens that decode meanwhile: a step under the token budget
  top_p    below 1: sampled at temperature 0.8, else greedy
"""

import math

import torch

import shrike_b200.models  # noqa: F401  (registers the architectures)
from shrike_b200.config import parse_config
from shrike_b200.engine.batch import StepEntry
from shrike_b200.engine.llm_engine import LLMEngine
from shrike_b200.shapes import shape_config
from shrike_b200.weights.random_init import random_tensors

PAGE = 16
TYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}


def case(name, shape, kind, dtype="bfloat16", batch=0, context=0, tokens=0, top_p=1.0):
    given = {"shape": shape, "kind": kind, "dtype": dtype, "batch": batch, "context": context, "tokens": tokens, "top_p": top_p}
    return given if name is None else {"name": name, **given}


def listed():
    return [
        # one user on the smallest model, a short chat: launches and latency
        case("decode_0.5b_b1", "qwen2.5-0.5b", "decode", batch=1, context=97),
        # one user on a small model, in the middle of an answer
        case("decode_1.5b_b1", "qwen2.5-1.5b", "decode", batch=1, context=517),
        # the headline: eight users at 1,024 tokens
        case("decode_7b_b8", "qwen2.5-7b", "decode", batch=8, context=1024),
        # the large batch of the headline, sampled as a chat service samples
        case("decode_7b_b64", "qwen2.5-7b", "decode", batch=64, context=1024, top_p=0.95),
        # a batch in the middle of the mixed workload: an odd count of requests of uneven lengths
        case("decode_1.5b_b37", "qwen2.5-1.5b", "decode", batch=37, context=801),
        # a short question to the smallest model
        case("prefill_0.5b_43", "qwen2.5-0.5b", "prefill", tokens=43),
        # the headline's long prompt
        case("prefill_7b_2048", "qwen2.5-7b", "prefill", tokens=2048),
        # a step of the mixed workload under its 512-token budget: a portion beside decoding requests
        case("mixed_1.5b_512", "qwen2.5-1.5b", "mixed", batch=37, context=640, tokens=475),
        # the 32-bit path: a prompt, and a few requests decoding
        case("prefill_fp32_0.5b_333", "qwen2.5-0.5b", "prefill", dtype="float32", tokens=333),
        case("decode_fp32_1.5b_b3", "qwen2.5-1.5b", "decode", dtype="float32", batch=3, context=200),
        # another of the designs served: linear attention with a state beside latent attention over wide page rows
        case("prefill_kavedra_1.5b_2048", "kavedra-1.5b", "prefill", tokens=2048),
        case("decode_kavedra_1.5b_b8", "kavedra-1.5b", "decode", batch=8, context=700),
    ]


def _between(rng, low, high):
    """A whole number, evenly spread over its logarithm."""
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high + 1)))))))


def draw(rng):
    what = rng.choice(["decode"] * 4 + ["prefill"] * 3 + ["mixed"] + ["fp32"] * 2 + ["kavedra"] * 2)
    if what == "fp32":
        if rng.random() < 0.5:
            return case(None, rng.choice(["qwen2.5-0.5b", "qwen2.5-1.5b"]), "prefill", "float32", tokens=_between(rng, 9, 400))
        return case(None, rng.choice(["qwen2.5-0.5b", "qwen2.5-1.5b"]), "decode", "float32", batch=_between(rng, 1, 16),
                    context=_between(rng, 16, 400))
    if what == "kavedra":
        if rng.random() < 0.5:
            return case(None, "kavedra-1.5b", "prefill", tokens=_between(rng, 100, 2048))
        return case(None, "kavedra-1.5b", "decode", batch=_between(rng, 1, 32), context=_between(rng, 64, 1024))
    if what == "mixed":
        singles = _between(rng, 4, 64)
        return case(None, rng.choice(["qwen2.5-0.5b", "qwen2.5-1.5b"]), "mixed", batch=singles, context=_between(rng, 100, 1024),
                    tokens=512 - singles)
    shape = rng.choice(["qwen2.5-0.5b", "qwen2.5-1.5b", "qwen2.5-3b", "qwen2.5-7b"])
    if what == "prefill":
        return case(None, shape, "prefill", tokens=_between(rng, 17, 2048))
    return case(None, shape, "decode", batch=_between(rng, 1, 64), context=_between(rng, 32, 1500),
                top_p=rng.choice([1.0, 1.0, 0.95]))


# ---- inputs --------------------------------------------------------------------------------------------------

def _requests(case, seed):
    """[(token ids the cache holds, the next token ids)] of a case, the portion first.  The ids follow from the seed, the
    lengths from the case alone: up to a twentieth below the context (mixed: from a fifth of it up)."""
    raw = shape_config(case["shape"])
    vocab = raw.get("vocab_size") or raw["vocab"]
    source = torch.Generator().manual_seed(1000003 * int(seed) + 17)
    spread = torch.Generator().manual_seed(case["batch"] + 100 * case["context"])

    def ids(count):
        return torch.randint(0, vocab, (count,), generator=source).tolist()

    found = []
    if case["kind"] == "prefill":
        return [([], ids(case["tokens"]))]
    low = 0.95
    if case["kind"] == "mixed":
        found.append((ids(case["context"]), ids(case["tokens"])))
        low = 0.2
    for _ in range(case["batch"]):
        share = low + (1.0 - low) * float(torch.rand((), generator=spread))
        found.append((ids(max(1, int(case["context"] * share) - 1)), ids(1)))
    return found


def _weights(case, seed):
    """Seeded random weights.  In a trained decoder every branch moves the residual a little; with N(0, 0.02)
    everywhere the first layer overwrites the embedding, and 28 layers make several percent of one rounding.  So the
    Qwen2 shapes get an embedding of order one and branches scaled down, by powers of two."""
    config = parse_config(shape_config(case["shape"]))
    tensors = random_tensors(config, int(seed), "cuda", TYPES[case["dtype"]])
    for name, tensor in tensors.items():
        if name == "model.embed_tokens.weight":
            tensor.mul_(32.0)
        elif name.endswith(("self_attn.o_proj.weight", "mlp.down_proj.weight")):
            tensor.mul_(0.125)
    return config, tensors


class State:
    """An engine with its requests' caches filled up to the pass."""

    def __init__(self, case, seed):
        self.kind = case["kind"]
        config, tensors = _weights(case, seed)
        self.requests = _requests(case, seed)
        pages = sum(-(-(len(held) + len(new)) // PAGE) for held, new in self.requests)
        self.engine = LLMEngine(None, block_size=PAGE, num_blocks=pages, max_running=len(self.requests),
                                max_tokens_per_step=4096, dtype=case["dtype"], config=config, tensors=tensors)
        self.runner = self.engine.runner
        self.sampling = (0.8, case["top_p"], int(seed)) if case["top_p"] < 1.0 else (0.0, 1.0, 0)
        self.caches = []
        if self.kind == "prefill":
            return
        waiting, count = [], 0
        for held, new in self.requests:
            cache = self.runner.cache.open()
            self.runner.cache.append(cache, 0, len(held))
            if waiting and count + len(held) > 4096:
                self.runner.step(waiting)
                waiting, count = [], 0
            waiting.append(StepEntry(cache, held, 0, []))
            count += len(held)
            self.caches.append(cache)
        self.runner.step(waiting)
        for cache, (held, new) in zip(self.caches, self.requests):
            self.runner.cache.append(cache, len(held), len(new))


def prepare(case, seed):
    return State(case, seed)


def run(state):
    """One step.  A prompt is a new request every pass; requests that decode take the same token again, at the same
    position (a recurrent state goes one token further with each pass).  Drawn tokens are not among the outputs: with
    random weights the two largest of 152,000 bfloat16-computed logits often lie closer than two correct sums of them."""
    runner = state.runner
    if state.kind == "prefill":
        prompt = state.requests[0][1]
        cache = runner.cache.open()
        runner.cache.append(cache, 0, len(prompt))
        logits = runner.step([StepEntry(cache, prompt, 0, [len(prompt) - 1])])
        runner.cache.free(cache)
    else:
        logits, _tokens = runner.step([StepEntry(cache, new, len(held), [len(new) - 1], state.sampling)
                                       for cache, (held, new) in zip(state.caches, state.requests)], sample=True)
    return {"logits": logits, "pages": list(runner.storage.kv), "states": [v for _, v in sorted(runner.storage.state.items())]}


# ---- what a pass cannot do without ---------------------------------------------------------------------------

def work(case):
    """Weights and the cached tokens read once, the new tokens' cache rows and the logits written once."""
    raw = shape_config(case["shape"])
    config = parse_config(raw)
    size = 4 if case["dtype"] == "float32" else 2
    lengths = _requests(case, 0)
    new = sum(len(n) for _, n in lengths)
    rows = len(lengths)
    pairs = sum(len(n) * len(h) + len(n) * (len(n) + 1) / 2 for h, n in lengths)   # (query, key) pairs of one layer
    cached, held_requests = sum(len(h) for h, _ in lengths), sum(1 for h, _ in lengths if h)
    if "hidden_size" in raw:
        hidden, heads, kv = raw["hidden_size"], raw["num_attention_heads"], raw["num_key_value_heads"]
        dim, layers, vocab = raw["head_dim"], raw["num_hidden_layers"], raw["vocab_size"]
        matrices = layers * (hidden * (heads + 2 * kv) * dim + heads * dim * hidden + 3 * hidden * raw["intermediate_size"])
        per_token = layers * 2 * kv * dim * size
        flops = 2.0 * new * matrices + layers * 4.0 * heads * dim * pairs
        bytes_ = matrices * size + (cached + new) * per_token
    else:
        hidden, vocab = raw["width"], raw["vocab"]
        flops, bytes_ = 0.0, 0.0
        seen = set()
        for run_ in config.order:
            entry = raw["layers"][run_.layer]
            m, kind = entry["mixer"], entry["type"]
            heads, dim = m["heads"], m["dim"]
            matrices = 3 * hidden * entry["mlp"]["ff"]
            if kind == "lightning":
                matrices += 5 * hidden * heads * dim
                flops += new * heads * 6.0 * dim * dim
                bytes_ += heads * dim * dim * 4 * (rows + held_requests)
            elif kind == "attention":
                matrices += 2 * hidden * (heads + m["kv_heads"]) * dim
                flops += 4.0 * heads * dim * pairs
                bytes_ += (cached + new) * 2 * m["kv_heads"] * dim * size
            else:
                rank, turned = m["kv_rank"], m["rot_dim"]
                matrices += hidden * (heads * (dim + turned) + rank + turned + 2 * heads * dim) + 2 * heads * dim * rank
                flops += 2.0 * heads * (dim + turned + dim) * pairs
                bytes_ += (cached + new) * (rank + turned) * size
            if run_.enter is not None:
                flops += 2.0 * new * 2 * hidden * hidden
                if "enter" not in seen:
                    bytes_ += 2 * hidden * hidden * size
                    seen.add("enter")
            flops += 2.0 * new * matrices
            if run_.layer not in seen:   # a layer that runs twice is read once
                bytes_ += matrices * size
                seen.add(run_.layer)
    flops += 2.0 * rows * hidden * vocab
    bytes_ += hidden * vocab * size + rows * vocab * 4 + new * hidden * size
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    """Relative errors of two correct implementations at the same precision, over the layers' depth; measured against
    64 bits and stated with a factor of about four."""
    if case["dtype"] == "float32":   # 7e-7 (0.5B) to 1.6e-6 (1.5B)
        return {"rel": 1e-5, "max": 4e-4}
    if case["shape"] in ("qwen2.5-7b", "kavedra-1.5b"):   # 1.0e-2 and 1.2e-2
        return {"rel": 0.03, "max": 0.5}
    return {"rel": 0.015, "max": 0.3}   # 2e-3 (0.5B) to 5e-3 (3B)


# ---- the same in 64 bits -------------------------------------------------------------------------------------

def exact(case, seed):
    if work(case)["flops"] + _context_flops(case) > 1.5e14:   # over about 20 seconds
        return None
    with torch.no_grad():
        raw = shape_config(case["shape"])
        _config, weights = _weights(case, seed)
        requests = [(held + new, len(new)) for held, new in _requests(case, seed)]
        return (_exact_qwen2 if "hidden_size" in raw else _exact_kavedra)(raw, weights, requests, case)


def _context_flops(case):
    """What computing the held tokens anew costs."""
    raw = shape_config(case["shape"])
    if "hidden_size" in raw:
        h = raw["hidden_size"]
        per_layer = 2 * h * h + 2 * h * raw["num_key_value_heads"] * raw["head_dim"] + 3 * h * raw["intermediate_size"]
        per_token = 2.0 * raw["num_hidden_layers"] * per_layer
    else:
        per_token = 2.0 * 28 * 60e6
    return per_token * sum(len(held) for held, _ in _requests(case, 0))


def _rms(x, eps):
    return x / torch.sqrt(x.square().mean(-1, keepdim=True) + eps)


def _causal(q, k, v, scale, sink=None, window=None):
    """q [n, H, D], k [n, G, D], v [n, G, V] of one whole sequence; query head a reads key/value head a // (H / G)."""
    n, heads, groups = q.shape[0], q.shape[1], k.shape[1]
    gap = torch.arange(n, device=q.device)[:, None] - torch.arange(n, device=q.device)[None, :]
    hidden = gap < 0
    if window is not None:
        hidden = hidden | (gap >= window)
    out = torch.empty(n, heads, v.shape[-1], dtype=q.dtype, device=q.device)
    for a in range(heads):
        g = a * groups // heads
        s = ((q[:, a] @ k[:, g].T) * scale).masked_fill_(hidden, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[a].expand(n, 1)], dim=1)
        out[:, a] = torch.softmax(s, dim=1)[:, :n] @ v[:, g]
    return out


def _pages_of(rows, ends):
    """rows [tokens, ...] of the requests one after another -> [pages, PAGE, ...] in the order in which a fresh pool
    hands its pages out: first what every request holds, then the page that its new tokens begin, where they begin one."""
    pages, later, at = [], [], 0
    for total, first in ends:
        padded = torch.zeros(-(-total // PAGE) * PAGE, *rows.shape[1:], dtype=rows.dtype, device=rows.device)
        padded[:total] = rows[at: at + total]
        split = -(-first // PAGE)
        whole = padded.view(-1, PAGE, *rows.shape[1:])
        pages.append(whole[:split])
        later.append(whole[split:])
        at += total
    return torch.cat(pages + later)


def _exact_qwen2(raw, weights, requests, case):
    d = torch.float64
    heads, kv, dim, eps = raw["num_attention_heads"], raw["num_key_value_heads"], raw["head_dim"], raw["rms_norm_eps"]
    ids = torch.tensor([t for seq, _ in requests for t in seq], device="cuda")
    lengths = [len(seq) for seq, _ in requests]
    positions = torch.cat([torch.arange(n, device="cuda") for n in lengths])
    # the model's definition forms the rotation's angles in 32 bits
    frequency = 1.0 / (raw["rope_theta"] ** (torch.arange(0, dim, 2).float() / dim))
    angle = (positions.float()[:, None] * frequency.to("cuda")[None, :]).to(d)
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]

    def turned(x):
        a, b = x[..., : dim // 2], x[..., dim // 2:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], dim=-1)

    x = weights["model.embed_tokens.weight"][ids].to(d)
    count = x.shape[0]
    kept = []
    for layer in range(raw["num_hidden_layers"]):
        def w(name):
            return weights["model.layers.%d.%s" % (layer, name)].to(d)
        h = _rms(x, eps) * w("input_layernorm.weight")
        q = turned((h @ w("self_attn.q_proj.weight").T + w("self_attn.q_proj.bias")).view(count, heads, dim))
        k = turned((h @ w("self_attn.k_proj.weight").T + w("self_attn.k_proj.bias")).view(count, kv, dim))
        v = (h @ w("self_attn.v_proj.weight").T + w("self_attn.v_proj.bias")).view(count, kv, dim)
        ends = [(len(seq), len(seq) - new) for seq, new in requests]
        kept.append(torch.stack([_pages_of(k, ends), _pages_of(v, ends)]))
        o = torch.cat([_causal(a, b, c, dim ** -0.5) for a, b, c in zip(q.split(lengths), k.split(lengths), v.split(lengths))])
        x = x + o.reshape(count, -1) @ w("self_attn.o_proj.weight").T
        h = _rms(x, eps) * w("post_attention_layernorm.weight")
        gate = h @ w("mlp.gate_proj.weight").T
        x = x + (gate * torch.sigmoid(gate) * (h @ w("mlp.up_proj.weight").T)) @ w("mlp.down_proj.weight").T
    last = torch.tensor(lengths, device="cuda").cumsum(0) - 1
    hidden = _rms(x[last], eps) * weights["model.norm.weight"].to(d)
    head = weights.get("lm_head.weight", weights["model.embed_tokens.weight"])
    logits = torch.cat([hidden @ part.to(d).T for part in head.split(16384)], dim=1)
    return {"logits": logits, "pages": [torch.stack(kept)], "states": []}


def _pair_angles(rot, positions):
    """cos and sin of neighbouring pairs' rotation, with stretched frequencies where the shape asks for them."""
    dims, base = rot["dims"], rot["base"]
    freq, gain = [base ** (-2.0 * i / dims) for i in range(dims // 2)], 1.0
    stretch = rot.get("scaling")
    if stretch:
        def border(turns):
            return dims * math.log(stretch["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))
        low = max(math.floor(border(stretch["fast"])), 0)
        high = min(math.ceil(border(stretch["slow"])), dims - 1)
        ramp = [min(max((i - low) / max(high - low, 0.001), 0.0), 1.0) for i in range(dims // 2)]
        freq = [f / stretch["factor"] * r + f * (1.0 - r) for f, r in zip(freq, ramp)]
        gain = 0.1 * math.log(stretch["factor"]) + 1.0
    angle = positions.double()[:, None, None] * torch.tensor(freq, dtype=torch.float64, device=positions.device)
    return angle.cos() * gain, angle.sin() * gain


def _turn_pairs(x, angles, dims):
    cos, sin = angles
    out = x.clone()
    even, odd = x[..., 0:dims:2], x[..., 1:dims:2]
    out[..., 0:dims:2] = even * cos - odd * sin
    out[..., 1:dims:2] = odd * cos + even * sin
    return out


def _evens_first(x, dims):
    """The order in which the cache holds the rotated dimensions: one of each pair, then the others."""
    order = list(range(0, dims, 2)) + list(range(1, dims, 2))
    return x[..., order + list(range(dims, x.shape[-1]))]


def _exact_kavedra(raw, weights, requests, case):
    d = torch.float64
    eps = raw["norm"]["eps"]
    ids = torch.tensor([t for seq, _ in requests for t in seq], device="cuda")
    lengths = [len(seq) for seq, _ in requests]
    ends = [(len(seq), len(seq) - new) for seq, new in requests]
    positions = torch.cat([torch.arange(n, device="cuda") for n in lengths])
    count = len(ids)
    embedded = weights["embed"][ids].to(d)
    loop, layers = raw["loop"], raw["layers"]
    order = [(i, None) for i in range(loop["start"])]
    for turn in range(loop["times"]):
        order += [(i, turn if i == loop["start"] else None) for i in range(loop["start"], loop["stop"])]
    order += [(i, None) for i in range(loop["stop"], len(layers))]

    def silu(z):
        return z * torch.sigmoid(z)

    x, states, latents, keys_values = embedded.clone(), [], [], []
    for index, opens in order:
        entry, name = layers[index], "l%d" % index
        m, kind = entry["mixer"], entry["type"]
        heads, dim, vdim = m["heads"], m["dim"], m["vdim"]

        def w(local):
            return weights["%s.%s" % (name, local)].to(d)
        if opens is not None:
            x = torch.cat([x, embedded], dim=-1) @ weights["loop.in"].to(d).T + weights["loop.step"].to(d)[opens]
        h = _rms(x, eps) * (1.0 + w("norm1"))
        if kind == "lightning":
            q, k = (silu(h @ w("mix." + p).T).view(count, heads, dim) for p in "qk")
            v = silu(h @ w("mix.v").T).view(count, heads, vdim)
            decay = torch.tensor(m["decay"], dtype=d, device="cuda")
            out, held = [], []
            for a, b, c in zip(q.split(lengths), k.split(lengths), v.split(lengths)):
                n = a.shape[0]
                gap = (torch.arange(n, device="cuda")[:, None] - torch.arange(n, device="cuda")[None, :])
                one = torch.empty(n, heads, vdim, dtype=d, device="cuda")
                state = torch.empty(heads, dim, vdim, dtype=d, device="cuda")
                for e in range(heads):
                    fade = (decay[e] ** gap.clamp(min=0)).masked_fill(gap < 0, 0.0)
                    one[:, e] = ((a[:, e] @ b[:, e].T) * fade) @ c[:, e]
                    state[e] = (b[:, e] * fade[-1][:, None]).T @ c[:, e]
                out.append(one)
                held.append(state)
            states.append(torch.stack(held))
            o = _rms(torch.cat(out).reshape(count, heads * vdim), eps) * w("mix.norm") * torch.sigmoid(h @ w("mix.g").T)
        elif kind == "attention":
            angles = _pair_angles(m["rot"], positions)
            q, k, v = ((h @ w("mix." + p).T + w("mix." + p + ".b")).view(count, -1, dim) for p in "qkv")
            q, k = _turn_pairs(q, angles, m["rot"]["dims"]), _turn_pairs(k, angles, m["rot"]["dims"])
            keys_values.append(torch.stack([_pages_of(_evens_first(k, m["rot"]["dims"]), ends), _pages_of(v, ends)]))
            o = torch.cat([_causal(a, b, c, m["scale"], sink=w("mix.sink"))
                           for a, b, c in zip(q.split(lengths), k.split(lengths), v.split(lengths))]).reshape(count, -1)
        else:
            rank, turned = m["kv_rank"], m["rot_dim"]
            angles = _pair_angles(m["rot"], positions)
            q = (h @ w("mix.q").T).view(count, heads, dim + turned)
            q = torch.cat([q[..., :dim], _turn_pairs(q[..., dim:], angles, turned)], dim=-1)
            down = h @ w("mix.dkv").T
            latent = _rms(down[:, :rank], eps) * w("mix.dkv.norm")
            shared = _turn_pairs(down[:, None, rank:], angles, turned)
            k = torch.cat([(latent @ w("mix.uk").T).view(count, heads, dim), shared.expand(count, heads, turned)], dim=-1)
            v = (latent @ w("mix.uv").T).view(count, heads, vdim)
            rows = torch.cat([latent, _evens_first(shared[:, 0], turned)], dim=-1)[:, None, :]
            latents.append(_pages_of(rows, ends)[None])
            window = (m.get("mask") or {}).get("size")
            o = torch.cat([_causal(a, b, c, m["scale"], window=window)
                           for a, b, c in zip(q.split(lengths), k.split(lengths), v.split(lengths))]).reshape(count, -1)
            o = o * torch.sigmoid(h @ w("mix.g").T)
        x = x + o @ w("mix.o").T
        h = _rms(x, eps) * (1.0 + w("norm2"))
        x = x + (silu(h @ w("mlp.gate").T) * (h @ w("mlp.up").T)) @ w("mlp.down").T
    last = torch.tensor(lengths, device="cuda").cumsum(0) - 1
    hidden = _rms(x[last], eps) * (1.0 + weights["final.norm"].to(d))
    logits = torch.cat([hidden @ part.to(d).T for part in weights["head"].split(16384)], dim=1) * raw["logit_scale"]
    # one pool of latent rows and one of keys and values, in the order in which the layers first ask for them
    return {"logits": logits, "pages": [torch.stack(latents), torch.stack(keys_values)], "states": states}
