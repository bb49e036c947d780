"""The work this engine is measured on: requests in the shapes that its users bring, through its
public entry points (``load_lm``, ``generate_batch``, the step function ``ModelRunner.step`` with
the cache manager's ``open`` / ``fork`` / ``close``).

Kinds of work:

``decode``    requests that hold a context get a continuation each: every context is forked, the
              forks take ``steps`` tokens one by one, all of them together, and are closed.  The
              logits of every step come back.  The tokens are given, as in a trace replay, so that
              every implementation computes the same numbers.
``prompt``    requests open, their whole prompts run (in steps of at most 2,048 tokens), the logits
              of each last token come back; with ``score`` the logits of every token.
``portions``  a long prompt runs in portions of ``portion`` tokens, each beside one token of every
              decoding request: what the scheduler makes of a request that arrives while others
              are being served.
``turn``      whole requests: prompts, then ``steps`` tokens one by one, then the end.
``generate``  ``generate_batch``: scheduler, step function and sampling together, greedy.

Weights are random (N(0, 0.02) and the like, the tables' and matrices' usual initialisation) and
belong to the program, not to a request: a model is loaded once and serves every input, as in a
user's program.  Contexts, prompts and given tokens are drawn anew from every seed.
"""
import math
import shutil
import tempfile
import weakref
import zlib

import torch

from pretrained_rstr_b200 import generate_batch, load_lm
from pretrained_rstr_b200.config.registry import named_size
from pretrained_rstr_b200.engine.batch import Entry
from pretrained_rstr_b200.weights.loader import write_model_folder

STEP_TOKENS = 2048                      # tokens a step takes at most (load_lm's default)
POSITIONS = 1024
#: the most requests that decode together in a case of a model
REQUESTS = {"small": 64, "medium": 32, "xl": 16, "musilorn-small": 16}
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}


# ------------------------------------------------------------------------------- the cases
def listed():
    def case(name, kind, model, requests, tokens, steps=0, ragged=True, dtype="bfloat16",
             portion=0, score=False):
        return dict(name=name, kind=kind, model=model, dtype=dtype, requests=requests, tokens=tokens,
                    steps=steps, ragged=ragged, portion=portion, score=score)

    return [
        # one user at a chat or a completion prompt: the smallest step, latency counts
        case("one_user", "decode", "small", 1, 640, steps=16),
        # the benchmark's headline: a small batch near the longest context
        case("batch_8", "decode", "small", 8, 1000, steps=16),
        # a loaded server, contexts of 500 to 1,000 tokens
        case("batch_64", "decode", "small", 64, 1000, steps=8),
        # an odd number of requests of unequal length at the next size
        case("medium_23", "decode", "medium", 23, 777, steps=8),
        # the largest model at a small batch: weights come from memory
        case("xl_8", "decode", "xl", 8, 900, steps=4),
        # time to first token of one ordinary prompt
        case("first_token", "prompt", "small", 1, 137),
        # the benchmark's prompt step
        case("prompts_2x1024", "prompt", "small", 2, 1024, ragged=False),
        # a batch of documents through the largest model (summaries, embeddings of prompts)
        case("xl_prompts", "prompt", "xl", 3, 731),
        # evaluation: the logits of every token of some texts, in 32-bit
        case("score_float32", "prompt", "small", 3, 301, dtype="float32", score=True),
        # a request of 1,000 tokens arrives while 24 others decode
        case("arrival", "portions", "small", 24, 1000, portion=256),
        # generation as the API's examples call it, in 32-bit (reproducible tokens)
        case("generate_float32", "generate", "small", 8, 96, steps=24, dtype="float32"),
        # another design: short convolutions, grouped keys, retention, a looped span
        case("musilorn_turn", "turn", "musilorn-small", 6, 500, steps=16),
    ]


def _between(rng, low, high):
    """A whole number from low to high, spread over its logarithm."""
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "prompt", "prompt", "portions", "turn", "generate"])
    model = rng.choice(["small", "small", "medium", "xl"])
    dtype = "bfloat16"
    requests, tokens, steps, portion, score = 1, 1, 0, 0, False
    if kind == "decode":
        if model == "small" and rng.random() < 0.15:
            dtype = "float32"
        requests = _between(rng, 1, 8 if dtype == "float32" else REQUESTS[model] if model != "xl" else 8)
        tokens = _between(rng, 16, POSITIONS - 16)
        steps = rng.randint(2, 4 if model == "xl" else 8)
    elif kind == "prompt":
        if model == "small" and rng.random() < 0.25:
            dtype = "float32"
        score = model != "xl" and rng.random() < 0.3
        requests = _between(rng, 1, 8)
        most = 1000 if score or dtype == "float32" else 2100
        tokens = _between(rng, 5, min(POSITIONS, max(8, most // requests)))
    elif kind == "portions":
        model = rng.choice(["small", "medium"])
        requests = _between(rng, 2, REQUESTS[model])
        tokens = _between(rng, 100, 1000)
        portion = rng.choice([64, 100, 128, 256, 512])
    elif kind == "turn":
        model = "musilorn-small"
        requests = _between(rng, 1, REQUESTS[model])
        tokens = _between(rng, 8, 700)
        steps = rng.randint(2, 16)
    else:
        model, dtype = "small", "float32"
        requests = _between(rng, 1, 8)
        tokens = _between(rng, 4, 128)
        steps = rng.randint(4, 24)
    return dict(kind=kind, model=model, dtype=dtype, requests=requests, tokens=tokens, steps=steps,
                ragged=rng.random() < 0.8, portion=portion, score=score)


def lengths(case):
    """Tokens each request holds (or brings): all the case's, or spread between half and all."""
    n = case["tokens"]
    if not case["ragged"]:
        return [n] * case["requests"]
    return [max(1, n - (i * 7919) % (n // 2 + 1)) for i in range(case["requests"])]


# ---------------------------------------------------------------------------------- weights
def _weights(model, dtype):
    """Names and values of a model's tensors, on the GPU in the element type it runs in."""
    arch, cfg = named_size(model)
    layers = getattr(cfg, "n_layer", 0)
    out = {}
    for name, want in arch.expected_tensors(cfg).items():
        g = torch.Generator(device="cuda")
        g.manual_seed(zlib.crc32(name.encode("utf-8")))
        std, mean = 0.02, 0.0
        if layers:                                        # GPT-2's rule
            if name.endswith("c_proj.weight"):
                std = 0.02 / math.sqrt(2.0 * layers)
            elif ".ln_" in name and name.endswith("weight") or name == "ln_f.weight":
                mean = 1.0
        elif name == "embed":
            std = 1.0
        elif name.endswith(".b"):
            std = 0.1
        elif len(want.shape) == 1:
            std, mean = 0.1, 1.0
        elif name.endswith(".conv"):
            std = 0.5
        else:
            std = 1.0 / math.sqrt(want.shape[-1])
        t = torch.randn(tuple(want.shape), generator=g, device="cuda", dtype=torch.float32)
        out[name] = (t * std + mean).to(DTYPES[dtype])
    return cfg, out


_loaded = {}


def _model(name, dtype):
    """The program's model: loaded from a model folder once, then serving every request."""
    key = (name, dtype)
    if key not in _loaded:
        cfg, tensors = _weights(name, dtype)
        folder = tempfile.mkdtemp(prefix="perf_model_")
        try:
            write_model_folder(folder, cfg, tensors, DTYPES[dtype])
            del tensors
            # contexts that several inputs hold at a time, and a continuation of one of them
            lanes = 64 if dtype == "float32" or name not in ("small", "medium") else 5 * REQUESTS[name]
            _loaded[key] = load_lm(folder, dtype=dtype, max_lanes=lanes, maxpos=POSITIONS,
                                   max_batched_tokens=STEP_TOKENS, share_prefixes=False)
        finally:
            shutil.rmtree(folder, ignore_errors=True)
    return _loaded[key]


# ----------------------------------------------------------------------------------- inputs
_count = [0]


class State:
    """What a program holds for one input: the model, token ids, contexts in the cache."""


def _tokens(case, seed):
    """(contexts or prompts, given tokens [steps][request], the arriving prompt) of a seed."""
    _arch, cfg = named_size(case["model"])
    vocab = getattr(cfg, "vocab_size", None) or cfg.vocab
    g = torch.Generator()
    g.manual_seed(int(seed))
    ids = lambda n: torch.randint(vocab, (n,), generator=g).tolist()  # noqa: E731
    prompts = [ids(n) for n in lengths(case)]
    steps = case["steps"]
    arriving = []
    if case["kind"] == "portions":
        arriving = ids(case["tokens"])
        steps = -(-case["tokens"] // case["portion"])
        # a decoding request needs room for its own steps
        prompts = [p[:POSITIONS - steps] for p in prompts]
    given = [ids(case["requests"]) for _ in range(steps)]
    return vocab, prompts, given, arriving


def _cut(rids, prompts, score):
    """Whole prompts as steps of at most STEP_TOKENS tokens."""
    steps, room = [[]], STEP_TOKENS
    for rid, p in zip(rids, prompts):
        at = 0
        while at < len(p):
            if room == 0:
                steps.append([])
                room = STEP_TOKENS
            n = min(room, len(p) - at)
            want = list(range(n)) if score else [n - 1] if at + n == len(p) else []
            steps[-1].append(Entry(rid, p[at:at + n], want))
            at, room = at + n, room - n
    return steps


def _close(cache, rids):
    for rid in rids:
        cache.close(rid)


def prepare(case, seed):
    s = State()
    s.case = case
    s.lm = _model(case["model"], case["dtype"])
    vocab, s.prompts, s.given, s.arriving = _tokens(case, seed)
    _count[0] += 1
    s.contexts = [("context", _count[0], i) for i in range(case["requests"])]
    s.rids = [("request", _count[0], i) for i in range(case["requests"])]
    cache, runner = s.lm.loaded.cache, s.lm.loaded.runner
    kind, rows = case["kind"], case["requests"]
    if kind in ("decode", "portions"):
        for rid in s.contexts:
            cache.open(rid)
        weakref.finalize(s, _close, cache, list(s.contexts))
        for entries in _cut(s.contexts, s.prompts, False):
            runner.step(entries)
    if kind == "prompt":
        rows = sum(len(p) for p in s.prompts) if case["score"] else rows
        s.logits = torch.empty(rows, vocab, device="cuda")
    elif kind != "generate":
        s.logits = torch.empty(len(s.given), rows, vocab, device="cuda")
        s.first = torch.empty(rows if kind == "turn" else 1, vocab, device="cuda")
    return s


# ------------------------------------------------------------------------------------- a pass
def _run_prompts(s, out):
    runner, at = s.lm.loaded.runner, 0
    for entries in _cut(s.rids, s.prompts, s.case["score"]):
        logits = runner.step(entries)
        out[at:at + logits.shape[0]].copy_(logits)
        at += logits.shape[0]


def run(s):
    kind = s.case["kind"]
    if kind == "generate":
        out = generate_batch(s.lm, s.prompts, s.case["steps"])
        return torch.tensor(out, dtype=torch.int64)
    cache, runner = s.lm.loaded.cache, s.lm.loaded.runner
    if kind in ("decode", "portions"):
        for source, rid in zip(s.contexts, s.rids):
            cache.fork(source, rid)
    else:
        for rid in s.rids:
            cache.open(rid)
    if kind == "prompt":
        _run_prompts(s, s.logits)
        _close(cache, s.rids)
        return s.logits
    if kind == "turn":
        _run_prompts(s, s.first)
    new, at, portion = ("arriving",) + s.rids[0][1:], 0, s.case["portion"]
    if s.arriving:
        cache.open(new)
    for k, given in enumerate(s.given):
        entries = [Entry(rid, [t], [0]) for rid, t in zip(s.rids, given)]
        if s.arriving:
            part = s.arriving[at:at + portion]
            at += len(part)
            entries.append(Entry(new, part, [len(part) - 1] if at == len(s.arriving) else []))
        logits = runner.step(entries)
        s.logits[k].copy_(logits[:len(given)])
        if s.arriving and at == len(s.arriving):
            s.first.copy_(logits[len(given):])
    if s.arriving:
        cache.close(new)
    _close(cache, s.rids)
    return {"logits": s.logits} if kind == "decode" else {"logits": s.logits, "first": s.first}


# ------------------------------------------------------------------------------------- counts
def _matrices(model):
    """(numbers in the matrices and tables a step reads once, multiply-adds a token needs in
    them without the head's, the head's, cache numbers a token keeps over all layers,
    multiply-adds a token needs for each token it attends to)."""
    arch, cfg = named_size(model)
    raw = cfg.to_dict()
    if "n_layer" in raw:
        d, f, n = raw["n_embd"], raw["n_inner"], raw["n_layer"]
        body, head = n * (4 * d * d + 2 * d * f), raw["vocab_size"] * d
        return body + head, body, head, n * 2 * d, n * 2 * d
    size = lambda t: math.prod(t.shape)  # noqa: E731
    tensors = arch.expected_tensors(cfg)
    head = size(tensors["head"])
    body = run_body = kept = seen = 0
    for i, layer in enumerate(raw["layers"]):
        times = 1
        loop = raw.get("loop")
        if loop and loop["start"] <= i < loop["stop"]:
            times = loop["times"]
        n = sum(size(t) for name, t in tensors.items() if name.startswith(f"l{i}.") and len(t.shape) == 2)
        body += n
        run_body += times * n
        mx = layer["mixer"]
        if layer["type"] == "attention":
            kept += times * 2 * mx["kv_heads"] * mx["dim"]
            seen += times * 2 * mx["heads"] * mx["dim"]
        else:                                    # a state of dim x vdim a head, read and written
            run_body += times * 2 * mx["heads"] * mx["dim"] * mx["vdim"]
    if raw.get("loop"):
        n = size(tensors["loop.in"])
        body, run_body = body + n, run_body + raw["loop"]["times"] * n
    return body + head, run_body, head, kept, seen


def _prompt_work(case, longs, starts, wanted, item):
    weights, body, head, kept, seen = _matrices(case["model"])
    tokens = sum(longs)
    pairs = sum(n * s + n * (n + 1) / 2 for n, s in zip(longs, starts))
    vocab_bytes = 4 * wanted * _vocab(case)
    return (weights * item + kept * item * (tokens + sum(starts)) + vocab_bytes,
            2 * tokens * body + 2 * pairs * seen + 2 * wanted * head)


def _vocab(case):
    raw = named_size(case["model"])[1].to_dict()
    return raw.get("vocab_size") or raw["vocab"]


def work(case):
    """Weights once a step, every cached row that is attended to once a step, new rows and logits
    once; the operations of the products and of the attention."""
    item = 2 if case["dtype"] == "bfloat16" else 4
    longs, kind = lengths(case), case["kind"]
    nbytes = flops = 0
    if kind in ("prompt", "turn", "generate"):
        wanted = sum(longs) if case["score"] else len(longs)
        steps = -(-sum(longs) // STEP_TOKENS)
        nbytes, flops = _prompt_work(case, longs, [0] * len(longs), wanted, item)
        nbytes += (steps - 1) * _matrices(case["model"])[0] * item
    steps, beside = case["steps"], 0
    if kind == "portions":
        beside = case["portion"]
        steps = -(-case["tokens"] // beside)
        longs = [min(n, POSITIONS - steps) for n in longs]
    if kind == "generate":
        steps -= 1                               # the prompt's step chooses the first token
    for k in range(steps):
        ones, starts = [1] * len(longs), [n + k for n in longs]
        wanted = len(longs)
        if beside:
            ones = ones + [min(beside, case["tokens"] - k * beside)]
            starts = starts + [k * beside]
            wanted += k == steps - 1
        b, f = _prompt_work(case, ones, starts, wanted, item)
        nbytes, flops = nbytes + b, flops + f
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """Four times the distance from the 64-bit results that was measured: 0.0037 in bfloat16 (0.008
    behind the norms around every branch of the other design), 1.5e-6 in 32-bit."""
    if case["kind"] == "generate":
        return {"rel": 0.0, "differ": 0.01}      # whole tokens: two logits may tie within rounding
    if case["dtype"] == "float32":
        return {"rel": 6e-6}
    return {"rel": 1.5e-2 if case["model"] in ("small", "medium", "xl") else 3e-2}


# -------------------------------------------------------------------------- plain 64-bit torch
def _layer_norm(x, w, b, eps):
    c = x - x.mean(dim=-1, keepdim=True)
    return c / torch.sqrt(c.square().mean(dim=-1, keepdim=True) + eps) * w + b


def _gelu(u):
    return 0.5 * u * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (u + 0.044715 * u ** 3)))


def _hidden(t):
    return torch.ones(t, t, dtype=torch.bool, device="cuda").triu(1)


def _gpt2(W, raw, ids, rows):
    heads, eps = raw["n_head"], raw.get("layer_norm_epsilon", 1e-5)
    t = len(ids)
    x = W["wte.weight"][ids] + W["wpe.weight"][:t]
    d = x.shape[1]
    for i in range(raw["n_layer"]):
        p = f"h.{i}."
        h = _layer_norm(x, W[p + "ln_1.weight"], W[p + "ln_1.bias"], eps)
        q, k, v = (h @ W[p + "attn.c_attn.weight"] + W[p + "attn.c_attn.bias"]).view(
            t, 3, heads, d // heads).permute(1, 2, 0, 3)
        a = (q @ k.transpose(1, 2) / math.sqrt(d // heads)).masked_fill(_hidden(t), -math.inf)
        y = (torch.softmax(a, dim=-1) @ v).transpose(0, 1).reshape(t, d)
        x = x + y @ W[p + "attn.c_proj.weight"] + W[p + "attn.c_proj.bias"]
        h = _layer_norm(x, W[p + "ln_2.weight"], W[p + "ln_2.bias"], eps)
        u = _gelu(h @ W[p + "mlp.c_fc.weight"] + W[p + "mlp.c_fc.bias"])
        x = x + u @ W[p + "mlp.c_proj.weight"] + W[p + "mlp.c_proj.bias"]
    x = _layer_norm(x[rows], W["ln_f.weight"], W["ln_f.bias"], eps)
    return x @ W["wte.weight"].T


def _turned(v, freqs, interleaved):
    """v [heads, T, n] with its first 2 * len(freqs) coordinates turned by position x frequency."""
    n = len(freqs)
    angle = torch.arange(v.shape[1], device="cuda", dtype=torch.float64)[:, None] * torch.tensor(
        freqs, device="cuda", dtype=torch.float64)
    c, s = torch.cos(angle), torch.sin(angle)
    first, second = (slice(0, 2 * n, 2), slice(1, 2 * n, 2)) if interleaved else (slice(0, n), slice(n, 2 * n))
    out = v.clone()
    out[..., first] = v[..., first] * c - v[..., second] * s
    out[..., second] = v[..., second] * c + v[..., first] * s
    return out


def _frequencies(rot):
    out = []
    sc = rot.get("scaling")
    for i in range(rot["dims"] // 2):
        f = rot["base"] ** (-2.0 * i / rot["dims"])
        if sc:
            wave = 2.0 * math.pi / f
            s = (sc["original"] / wave - sc["low"]) / (sc["high"] - sc["low"])
            s = min(1.0, max(0.0, s))
            f = (1.0 - s) * f / sc["factor"] + s * f
        out.append(f)
    return out


def _convolved(u, taps):
    out = torch.zeros_like(u)
    n = taps.shape[1]
    for back in range(min(n, u.shape[0])):
        out[back:] += taps[:, n - 1 - back] * u[:u.shape[0] - back]
    return out


def _unit(v, eps):
    return v / torch.sqrt(v.square().mean(dim=-1, keepdim=True) + eps)


def _musilorn(W, raw, ids, rows):
    eps, mult, t = raw["norm"]["eps"], raw["residual_mult"], len(ids)
    norm = lambda v, name: _layer_norm(v, W[name], W[name + ".b"], eps)  # noqa: E731

    def attention(h, p, mx):
        H, G, D = mx["heads"], mx["kv_heads"], mx["dim"]
        q = _convolved(h @ W[p + "q"].T, W[p + "q.conv"]).view(t, H, D).transpose(0, 1)
        v = _convolved(h @ W[p + "k"].T, W[p + "k.conv"]).view(t, G, D).transpose(0, 1)
        freqs = _frequencies(mx["rot"])
        q = _turned(_unit(q, eps) * W[p + "q.norm"], freqs, True)
        k = _turned(_unit(v, eps) * W[p + "k.norm"], freqs, True).repeat_interleave(H // G, 0)
        a = q @ k.transpose(1, 2) * mx["scale"]
        if mx.get("softcap"):
            a = mx["softcap"] * torch.tanh(a / mx["softcap"])
        a = a.masked_fill(_hidden(t), -math.inf)
        # a key of score 0 that has no value
        a = torch.softmax(torch.cat([a, torch.zeros_like(a[..., :1])], dim=-1), dim=-1)[..., :-1]
        return (a @ v.repeat_interleave(H // G, 0)).transpose(0, 1).reshape(t, -1) @ W[p + "o"].T

    def retention(h, p, mx):
        H, D = mx["heads"], mx["dim"]
        split = lambda name, n: (h @ W[p + name].T).view(t, H, n).transpose(0, 1)  # noqa: E731
        freqs = _frequencies(mx["rot"])
        q = _turned(split("q", D), freqs, False)
        k = _turned(split("k", D), freqs, False) * D ** -0.5
        at = torch.arange(t, device="cuda", dtype=torch.float64)
        decay = torch.tensor(mx["decay"], device="cuda", dtype=torch.float64)[:, None, None]
        past = (at[:, None] - at[None, :]).clamp(min=0.0)
        a = (q @ k.transpose(1, 2) * decay ** past).masked_fill(_hidden(t), 0.0)
        o = _unit(a @ split("v", mx["vdim"]), eps).transpose(0, 1).reshape(t, -1)
        return (o * torch.nn.functional.silu(h @ W[p + "g"].T)) @ W[p + "o"].T

    order = [(i, False) for i in range(len(raw["layers"]))]
    loop = raw.get("loop")
    if loop:
        span = [(i, i == loop["start"]) for i in range(loop["start"], loop["stop"])]
        order = order[:loop["start"]] + span * loop["times"] + order[loop["stop"]:]
    x = start = W["embed"][ids]
    for i, joins in order:
        layer, p = raw["layers"][i], f"l{i}."
        if joins:
            x = torch.cat([x, start], dim=-1) @ W["loop.in"].T
        mixer = attention if layer["type"] == "attention" else retention
        x = x + mult * norm(mixer(norm(x, p + "norm1"), p + "mix.", layer["mixer"]), p + "norm1b")
        if layer.get("mlp"):
            h = norm(x, p + "norm2")
            u = _gelu(h @ W[p + "mlp.gate"].T) * (h @ W[p + "mlp.up"].T)
            x = x + mult * norm(u @ W[p + "mlp.down"].T, p + "norm2b")
    y = norm(x[rows], "final.norm") @ W["head"].T
    cap = raw.get("logit_softcap")
    return cap * torch.tanh(y / cap) if cap else y


@torch.no_grad()
def exact(case, seed):
    if case["kind"] == "generate":
        return None                              # whole tokens
    cfg, tensors = _weights(case["model"], case["dtype"])
    raw = cfg.to_dict()
    W = {name: t.double() for name, t in tensors.items()}
    del tensors
    forward = _gpt2 if "n_layer" in raw else _musilorn

    def logits(ids, rows):
        return forward(W, raw, torch.tensor(ids, device="cuda"), rows)

    _vocab_size, prompts, given, arriving = _tokens(case, seed)
    if case["kind"] == "prompt":
        return torch.cat([logits(p, list(range(len(p))) if case["score"] else [len(p) - 1])
                          for p in prompts])
    after, first = [], []
    for i, p in enumerate(prompts):
        y = logits(p + [g[i] for g in given], list(range(len(p) - 1, len(p) + len(given))))
        first.append(y[:1])
        after.append(y[1:])
    out = {"logits": torch.stack(after, dim=1)}
    if case["kind"] == "portions":
        out["first"] = logits(arriving, [len(arriving) - 1])
    elif case["kind"] == "turn":
        out["first"] = torch.cat(first)
    return out
