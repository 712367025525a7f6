"""What this engine's speed is measured on: the layers that its designs are made of, and steps of a whole model.

Every case is one call that a program makes of this package: the step function of an engine, or the entry points in
``prefixserve_b200.ops`` that a layer of one of the designs calls, on a paged cache or on per-request states laid out as
the cache manager lays them out.  Sizes are those of the presets: layer sizes of a 1B-class decoder (width 2,048) and of
an 8B-class one (width 4,096).  A step is either single tokens of many requests (decode) or portions of prompts; the
requests of a step have different lengths and lie at different positions.

A case's ``kind`` names the layer.  ``requests``: how many requests are in the step; ``tokens``: new tokens of the
longest of them (1: a decode step); ``context``: how many tokens the longest has behind it already.  A layer's pass may
be run again on the same state: it writes the same rows of the cache, and carries a recurrent state further.
"""

from __future__ import annotations

import tempfile
from types import SimpleNamespace

import torch

from prefixserve_b200 import LlamaConfig, ops
from prefixserve_b200.config.presets import PRESETS
from prefixserve_b200.engine import Engine, EngineConfig, StepItem
from prefixserve_b200.parts.base import ItemView, StepContext
from prefixserve_b200.weights import write_random_model

PAGE = 16
STEP_LAYERS = 4          # layers of the 1B-class decoder in the cases of a whole step, under its full vocabulary
STEP_VOCAB = 128256
FF = {2048: 8192, 4096: 14336}      # feed-forward width by model width
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}


def listed():
    return [
        # a whole decode step: eight conversations of up to 4,000 tokens, the workload the engine is quoted on
        dict(name="step_decode", kind="step", requests=8, context=4000, portion=0),
        # the gated feed-forward of the wider model on a prompt's tokens; no multiple of any tile
        dict(name="ffn_prompt", kind="ffn", width=4096, tokens=1979),
        # the smallest call: the same of the smaller model for a handful of decoded tokens, all of it reading weights
        dict(name="ffn_few", kind="ffn", width=2048, tokens=4),
        # grouped-query attention of three prompt portions that continue behind cached tokens
        dict(name="attention_prompt", kind="attention", width=2048, requests=3, tokens=900, context=2100),
        # windowed attention with capped scores and an output gate, one prompt and a shorter one beside it
        dict(name="rows_prompt", kind="rows", design="dogotar", width=2048, requests=2, tokens=1500, context=700),
        # attention with a window and kept first keys for 32 decoding requests of the wider model
        dict(name="rows_decode", kind="rows", design="zomolix", width=4096, requests=32, tokens=1, context=3000),
        # the gated delta rule over a prompt of 2,000 tokens
        dict(name="delta_prompt", kind="delta", width=2048, requests=1, tokens=2000, context=0, dtype="bfloat16"),
        # the delta rule with a decay per channel over two portions that continue earlier ones
        dict(name="channel_delta_prompt", kind="channel_delta", width=2048, requests=2, tokens=1200, context=512, dtype="bfloat16"),
        # gated linear attention over a prompt, the wider model
        dict(name="linear_attention_prompt", kind="linear", width=4096, requests=1, tokens=1811, context=0, dtype="bfloat16"),
        # routed experts on a prompt's tokens
        dict(name="experts_prompt", kind="experts", design="bumalix", width=2048, tokens=2037),
        # routed experts on the tokens of a dozen decoding requests
        dict(name="experts_decode", kind="experts", design="zomolix", width=4096, tokens=12),
        # attention through latents for sixteen decoding requests without a window
        dict(name="latent_decode", kind="latent", design="zomolix", width=4096, requests=16, tokens=1, context=3500),
    ]


def _between(rng, low, high):
    """A whole number from low to high, spread evenly over its logarithm."""
    return int(round(low * (high / low) ** rng.random()))


def draw(rng):
    kind = rng.choice(["step", "ffn", "attention", "rows", "delta", "channel_delta", "linear", "experts", "latent"])
    width = rng.choice([2048, 4096])
    if kind == "step":
        return dict(kind=kind, requests=rng.randint(1, 8), context=_between(rng, 100, 4000), portion=rng.choice([0, 0, _between(rng, 20, 600)]))
    if kind == "ffn":
        return dict(kind=kind, width=width, tokens=_between(rng, 1, 1979))
    if kind == "experts":
        return dict(kind=kind, design=rng.choice(["gekopel", "zomolix", "bumalix"]), width=width, tokens=_between(rng, 1, 2037))
    case = dict(kind=kind, width=width)
    if kind == "rows":
        case["design"] = rng.choice(["dogotar", "bumalix", "zomolix", "gekopel"])
    if kind == "latent":
        case["design"] = rng.choice(["nerenex", "zomolix"])
    if rng.random() < 0.5:  # a decode step
        case.update(requests=_between(rng, 1, 32), tokens=1, context=_between(rng, 30, 3500))
    else:
        case.update(requests=rng.randint(1, 3), context=rng.choice([0, _between(rng, 30, 2100)]))
        case["tokens"] = _between(rng, 24, 2000 // case["requests"])
    if kind in ("delta", "channel_delta", "linear"):
        case["dtype"] = rng.choice(["bfloat16"] * 4 + ["float32"])
    return case


# ---- the step's requests


def _portions(case):
    """(new tokens, tokens already held) of every request; each is shorter than the one before it."""
    r = case["requests"]
    new = [max(1, int(case["tokens"] * (1 - 0.4 * i / r))) for i in range(r)]
    held = [int(case["context"] * (1 - 0.5 * i / r)) for i in range(r)]
    return list(zip(new, held))


def _step(portions, generator, device="cuda"):
    """The step's context and the number of pages its block table names, page numbers in no order."""
    i32 = dict(dtype=torch.int32, device=device)
    starts = [0]
    views = []
    for i, (n, held) in enumerate(portions):
        views.append(ItemView(slot=i, start=held, end=held + n, first_token=starts[-1]))
        starts.append(starts[-1] + n)
    total, width = starts[-1], max(-(-(n + held) // PAGE) for n, held in portions)
    pages = len(portions) * width
    table = torch.randperm(pages, generator=generator, device=device).to(torch.int32).view(len(portions), width)
    ctx = StepContext(
        num_tokens=total, num_items=len(portions), compute_dtype=torch.bfloat16, device=torch.device(device), items=views,
        token_ids=torch.zeros(total, **i32),
        positions=torch.cat([torch.arange(held, held + n, **i32) for n, held in portions]),
        token_item=torch.cat([torch.full((n,), i, **i32) for i, (n, _) in enumerate(portions)]),
        item_start=torch.tensor(starts, **i32), kv_len=torch.tensor([n + held for n, held in portions], **i32),
        slots=torch.arange(len(portions), **i32), block_tables={0: table.contiguous()},
        max_new_tokens=max(n for n, _ in portions), max_kv_len=max(n + held for n, held in portions),
        all_decode=all(n == 1 for n, _ in portions))
    return ctx, pages


class _Random:
    """Tensors on the GPU from one seed."""

    def __init__(self, seed):
        self.generator = torch.Generator(device="cuda")
        self.generator.manual_seed(int(seed))

    def normal(self, *shape, std=1.0, mean=0.0, dtype=torch.float32):
        return (torch.randn(shape, generator=self.generator, device="cuda") * std + mean).to(dtype)

    def uniform(self, low, high, *shape):
        return torch.rand(shape, generator=self.generator, device="cuda") * (high - low) + low


def prepare(case, seed):
    return _KINDS[case["kind"]].prepare(case, _Random(seed))


def run(state):
    return state.kind.run(state)


def work(case):
    return _KINDS[case["kind"]].work(case)


def tolerance(case):
    return _KINDS[case["kind"]].tolerance(case)


def exact(case, seed):
    kind = _KINDS[case["kind"]]
    return kind.exact(kind.prepare(case, _Random(seed)))


def _keys(case, window=None):
    """Pairs of (query, visible key) of the step."""
    pairs = 0
    for n, held in _portions(case):
        for end in range(held + 1, held + n + 1):
            pairs += end if window is None else min(end, window)
    return pairs


def _rows_read(case, window=None):
    """Cached rows that a step's queries see."""
    return sum(n + held if window is None else min(n + held, window + n - 1) for n, held in _portions(case))


# ---- a whole step of the engine


class _Step:
    @staticmethod
    def prepare(case, rnd):
        seed = int(torch.randint(1 << 30, (1,), generator=rnd.generator, device="cuda"))
        config = LlamaConfig.from_dicts(dict(PRESETS["llama-3.2-1b"], num_hidden_layers=STEP_LAYERS))
        portion = case["portion"]
        longest = case["context"] + max(portion, 1)
        with tempfile.TemporaryDirectory() as folder:
            write_random_model(folder, config, seed, std=0.02, dtype=torch.bfloat16, device="cuda")
            engine = Engine(EngineConfig(model_path=folder, dtype=torch.bfloat16, max_num_seqs=case["requests"], max_prefill_tokens=2048,
                                         max_seq_len=4096 + 1024, num_blocks=case["requests"] * (longest // PAGE + 2) + 8, page_size=PAGE,
                                         enable_prefix_cache=False))
        cache, items = engine.cache, []
        ids = torch.randint(STEP_VOCAB, (case["requests"], longest), generator=rnd.generator, device="cuda").to(torch.int32).cpu().numpy()
        for i in range(case["requests"]):
            held = int(case["context"] * (1 - 0.5 * i / case["requests"]))
            n = max(1, portion) if i == 0 else 1
            slot = cache.open()
            for at in range(0, held, 2048):
                upto = min(held, at + 2048)
                cache.reserve(slot, upto)
                engine.runner.step([StepItem(slot, at, ids[i, at:upto], ())])
                cache.advance(slot, upto)
            cache.reserve(slot, held + n)
            items.append(StepItem(slot, held, ids[i, held: held + n], (n - 1,)))
        return SimpleNamespace(kind=_Step, engine=engine, items=items)

    @staticmethod
    def run(s):
        return s.engine.runner.step(s.items)

    @staticmethod
    def work(case):
        layer = 2048 * (2048 + 1024) + 2048 * 2048 + 3 * 2048 * 8192
        r, n = case["requests"], case["requests"] + max(case["portion"] - 1, 0)
        held = sum(int(case["context"] * (1 - 0.5 * i / r)) for i in range(r))
        kv = STEP_LAYERS * 2 * 8 * 64 * 2
        pairs = held + case["portion"] * case["context"]
        return {"bytes": 2 * (STEP_LAYERS * layer + STEP_VOCAB * 2048) + kv * held + 4 * r * STEP_VOCAB,
                "flops": 2 * STEP_LAYERS * layer * n + 2 * r * STEP_VOCAB * 2048 + 4 * STEP_LAYERS * 2048 * pairs}

    @staticmethod
    def tolerance(case):  # a rounding of 16 bits in one layer travels through all that follow
        return {"rel": 0.02, "max": 0.3}

    @staticmethod
    def exact(s):  # a model in 64 bits over all the cached tokens takes too long
        return None


# ---- feed-forward


class _FeedForward:
    @staticmethod
    def prepare(case, rnd):
        h, ff, t = case["width"], FF[case["width"]], case["tokens"]
        b16 = dict(dtype=torch.bfloat16)
        return SimpleNamespace(kind=_FeedForward, x=rnd.normal(t, h, **b16), w_in=rnd.normal(2 * ff, h, std=0.02, **b16),
                               w_out=rnd.normal(h, ff, std=0.02, **b16))

    @staticmethod
    def run(s):
        return ops.linear(ops.gated_linear(s.x, s.w_in, "silu"), s.w_out)

    @staticmethod
    def work(case):
        h, ff, t = case["width"], FF[case["width"]], case["tokens"]
        return {"bytes": 2 * (3 * ff * h + 2 * t * h), "flops": 6 * t * h * ff}

    @staticmethod
    def tolerance(case):  # the activation and the result are rounded to bfloat16
        return {"rel": 0.012, "max": 0.1}

    @staticmethod
    def exact(s):
        up = s.x.double() @ s.w_in.double().t()
        g, u = up.chunk(2, dim=1)
        return (torch.nn.functional.silu(g) * u) @ s.w_out.double().t()


# ---- attention over pages


def _softmax_over_keys(q, keys, values, held, *, scale, window=None, chunk=None, keep_first=0, bias=None, sink=None, softcap=None):
    """One request in 64 bits: q [n, hq, d], keys [len, hkv, d], values [len, hkv, v] -> [n, hq, v]."""
    n, hq, _ = q.shape
    per = hq // keys.shape[1]
    i = torch.arange(held, held + n, device=q.device)[:, None]
    j = torch.arange(keys.shape[0], device=q.device)[None, :]
    seen = j <= i
    if window is not None:
        seen &= (i - j < window) | (j < keep_first)
    if chunk is not None:
        seen &= j // chunk == i // chunk
    out = []
    for h in range(hq):
        s = (q[:, h].double() @ keys[:, h // per].double().t()) * scale
        if softcap is not None:
            s = softcap * torch.tanh(s / softcap)
        if bias is not None:
            s = s + bias[h].double()[(i - j).clamp(0, bias.shape[1] - 1)]
        s = s.masked_fill(~seen, float("-inf"))
        if sink is not None:
            s = torch.cat([s, sink[h].double().expand(n, 1)], dim=1)
        p = torch.softmax(s, dim=1)[:, : keys.shape[0]]
        out.append(p @ values[:, h // per].double())
    return torch.stack(out, dim=1)


class _Attention:
    """Grouped-query attention over keys and values in planes of their own: the 1B-class model's heads of 64 or the
    8B-class one's of 128."""

    @staticmethod
    def prepare(case, rnd):
        ctx, pages = _step(_portions(case), rnd.generator)
        d = 64 if case["width"] == 2048 else 128
        return SimpleNamespace(kind=_Attention, ctx=ctx, q=rnd.normal(ctx.num_tokens, 32, d, dtype=torch.bfloat16),
                               kv=rnd.normal(pages, 2, 8, PAGE, d, dtype=torch.bfloat16))

    @staticmethod
    def run(s):
        return ops.attention(s.q, s.kv, s.ctx.block_tables[0], s.ctx.positions, s.ctx.token_item, ctx=s.ctx)

    @staticmethod
    def work(case):
        d, t = (64 if case["width"] == 2048 else 128), sum(n for n, _ in _portions(case))
        return {"bytes": 2 * (2 * t * 32 * d + _rows_read(case) * 2 * 8 * d), "flops": 4 * 32 * d * _keys(case)}

    @staticmethod
    def tolerance(case):  # weights and result in bfloat16
        return {"rel": 0.015, "max": 0.1}

    @staticmethod
    def exact(s):
        out = []
        for i, it in enumerate(s.ctx.items):
            rows = s.kv[s.ctx.block_tables[0][i].long()]  # [pages, 2, heads, page, d]
            keys, values = (rows[:, p].transpose(1, 2).reshape(-1, rows.shape[2], rows.shape[4])[: it.end] for p in (0, 1))
            q = s.q[it.first_token: it.first_token + it.end - it.start]
            out.append(_softmax_over_keys(q, keys, values, it.start, scale=q.shape[-1] ** -0.5).flatten(1))
        return torch.cat(out)


class _Rows:
    """Attention over cache rows that hold a key and then its value, with each design's options."""

    @staticmethod
    def options(case):
        heads, span = (16, 1024) if case["width"] == 2048 else (32, 2048)
        return heads, heads // 4, span

    @staticmethod
    def prepare(case, rnd):
        heads, kv_heads, span = _Rows.options(case)
        ctx, pages = _step(_portions(case), rnd.generator)
        t, d, design = ctx.num_tokens, 128, case["design"]
        proj = rnd.normal(t, (2 * heads + 2 * kv_heads) * d, dtype=torch.bfloat16)  # [queries, keys, values, output gate]
        more = dict(num_heads=heads, num_kv_heads=kv_heads, dim=d, vdim=d, page_size=PAGE, scale=d ** -0.5)
        if design == "dogotar":
            more.update(window=span, softcap=50.0, gate=proj[:, (heads + 2 * kv_heads) * d:])
        elif design == "bumalix":
            more.update(window=span)
        elif design == "zomolix":
            more.update(window=span, keep_first=4, sink=rnd.normal(heads))
        else:
            more.update(chunk=span, bias=rnd.normal(heads, span, std=0.5), sink=rnd.normal(heads))
        return SimpleNamespace(kind=_Rows, ctx=ctx, q=proj[:, : heads * d].contiguous().view(t, heads, d),
                               kv=rnd.normal(pages, 1, kv_heads, PAGE, 2 * d, dtype=torch.bfloat16), more=more)

    @staticmethod
    def run(s):
        return ops.attention_over_rows(s.q, s.kv, s.ctx.block_tables[0], s.ctx, **s.more)

    @staticmethod
    def work(case):
        heads, kv_heads, span = _Rows.options(case)
        t, gate = sum(n for n, _ in _portions(case)), case["design"] == "dogotar"
        return {"bytes": 2 * ((3 if gate else 2) * t * heads * 128 + _rows_read(case, span) * kv_heads * 256),
                "flops": 4 * heads * 128 * _keys(case, span)}

    @staticmethod
    def tolerance(case):  # weights and result in bfloat16
        return {"rel": 0.015, "max": 0.1}

    @staticmethod
    def exact(s):
        out = []
        m = s.more
        for i, it in enumerate(s.ctx.items):
            rows = s.kv[s.ctx.block_tables[0][i].long()][:, 0].transpose(1, 2).reshape(-1, m["num_kv_heads"], 256)[: it.end]
            q = s.q[it.first_token: it.first_token + it.end - it.start]
            out.append(_softmax_over_keys(q, rows[:, :, :128], rows[:, :, 128:], it.start, scale=m["scale"], window=m.get("window"),
                                          chunk=m.get("chunk"), keep_first=m.get("keep_first", 0), bias=m.get("bias"),
                                          sink=m.get("sink"), softcap=m.get("softcap")).flatten(1))
        out = torch.cat(out)
        return out * torch.sigmoid(m["gate"].double()) if "gate" in m else out


class _Latent:
    """Attention of latent-space queries over cached latents, a row of 512 + 64 numbers a token that all heads share."""

    RANK, ROT = 512, 64

    @staticmethod
    def options(case):
        heads, window = (16, 1024) if case["width"] == 2048 else (32, 2048)
        return heads, window if case["design"] == "nerenex" else None

    @staticmethod
    def prepare(case, rnd):
        heads, window = _Latent.options(case)
        ctx, pages = _step(_portions(case), rnd.generator)
        d = _Latent.RANK + _Latent.ROT
        gate = torch.sigmoid(rnd.normal(ctx.num_tokens, heads)) if case["design"] == "nerenex" else None
        sink = rnd.normal(heads) if case["design"] == "zomolix" else None
        return SimpleNamespace(kind=_Latent, ctx=ctx, q=rnd.normal(ctx.num_tokens, heads, d, std=0.6), gate=gate, sink=sink, window=window,
                               cache=rnd.normal(pages, 1, 1, PAGE, d, dtype=torch.bfloat16))

    @staticmethod
    def run(s):
        c = s.ctx
        return ops.latent_attention(s.q, s.cache, c.block_tables[0], c.positions, c.token_item, s.gate, rank=_Latent.RANK, page_size=PAGE,
                                    window=s.window, scale=192 ** -0.5, out_dtype=torch.bfloat16, items=c.items, key_hint=c.max_kv_len,
                                    sink=s.sink)

    @staticmethod
    def work(case):
        heads, window = _Latent.options(case)
        t, d = sum(n for n, _ in _portions(case)), _Latent.RANK + _Latent.ROT
        return {"bytes": 4 * t * heads * d + 2 * t * heads * _Latent.RANK + 2 * d * _rows_read(case, window),
                "flops": 2 * heads * (d + _Latent.RANK) * _keys(case, window)}

    @staticmethod
    def tolerance(case):  # prompt portions round the queries to bfloat16, single tokens the result only
        return {"rel": 0.02, "max": 0.15}

    @staticmethod
    def exact(s):
        out = []
        for i, it in enumerate(s.ctx.items):
            rows = s.cache[s.ctx.block_tables[0][i].long()].reshape(-1, 1, _Latent.RANK + _Latent.ROT)[: it.end]
            q = s.q[it.first_token: it.first_token + it.end - it.start]
            out.append(_softmax_over_keys(q, rows, rows[:, :, : _Latent.RANK], it.start, scale=192 ** -0.5, window=s.window, sink=s.sink))
        out = torch.cat(out)
        return out if s.gate is None else out * s.gate.double()[:, :, None]


# ---- recurrences with a matrix state per head


def _short_convolution(proj, taps, before, start):
    """[n, C] inputs behind the K-1 rows ``before`` (zeros in front of the sequence) -> silu of the causal convolution."""
    k = taps.shape[1]
    before = before.clone()
    for row in range(k - 1):
        if start - (k - 1) + row < 0:
            before[row] = 0
    x = torch.cat([before, proj])
    y = sum(x[j: j + proj.shape[0]] * taps[:, j] for j in range(k))
    return torch.nn.functional.silu(y), x[-(k - 1):]


def _unit(x):
    return x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)


class _Delta:
    """The gated delta rule behind short convolutions (``channel`` False), or the one with a decay per key channel."""

    channel = False

    @staticmethod
    def sizes(case):
        heads = 16 if case["width"] == 2048 else 32
        return dict(groups=heads // 2, heads=heads, dim=128, vdim=128), 4

    @classmethod
    def prepare(cls, case, rnd):
        sizes, k = cls.sizes(case)
        heads, dim, vdim = sizes["heads"], sizes["dim"], sizes["vdim"]
        ctx, _ = _step(_portions(case), rnd.generator)
        t, c, dtype = ctx.num_tokens, 2 * sizes["groups"] * dim + heads * vdim, DTYPES[case["dtype"]]
        # the columns behind the convolved channels: the output gate, or the decay's and gate's latents and the write strengths
        more = 256 + heads if cls.channel else heads * vdim
        state = torch.cat([rnd.normal(case["requests"], (k - 1) * c), rnd.normal(case["requests"], heads * dim * vdim, std=0.1)], dim=1)
        s = SimpleNamespace(kind=cls, ctx=ctx, proj=rnd.normal(t, c + more, dtype=dtype), taps=rnd.normal(c, k, std=0.4),
                            state=state.contiguous(), sizes=sizes)
        if cls.channel:
            rate, bias = torch.exp(rnd.uniform(-2.0, 1.0, heads, 1)), rnd.uniform(-4.0, 1.0, heads, dim)
            s.decay = torch.exp(-rate * torch.nn.functional.softplus(rnd.normal(t, heads, dim) + bias)).view(t, heads * dim)
            s.beta_at = c + 256
        else:
            s.ba, s.a_log, s.dt_bias = rnd.normal(t, 2 * heads), rnd.uniform(-2.0, 1.0, heads), rnd.uniform(-4.0, 1.0, heads)
            s.gain, s.eps = rnd.normal(vdim, std=0.1, mean=1.0), 1e-6
        return s

    @classmethod
    def run(cls, s):
        if cls.channel:
            out = ops.channel_delta_rule(s.proj, s.beta_at, s.decay, s.taps, s.state, s.ctx, **s.sizes)
        else:
            out = ops.delta_rule(s.proj, s.ba, s.taps, s.a_log, s.dt_bias, s.gain, s.state, s.ctx, eps=s.eps, **s.sizes)
        return out, s.state

    @classmethod
    def work(cls, case):
        sizes, k = cls.sizes(case)
        heads, dim, vdim = sizes["heads"], sizes["dim"], sizes["vdim"]
        t, c, size = sum(n for n, _ in _portions(case)), 2 * sizes["groups"] * dim + heads * vdim, DTYPES[case["dtype"]].itemsize
        more = 4 * heads * (dim + vdim) + size * heads if cls.channel else 2 * size * heads * vdim + 8 * heads
        return {"bytes": t * (size * c + more) + 8 * case["requests"] * ((k - 1) * c + heads * dim * vdim),
                "flops": 6 * t * heads * dim * vdim}

    @classmethod
    def tolerance(cls, case):
        # float32 throughout (the largest of 67 million sums is a long way from the typical one); the gated rule's
        # result leaves in the compute type
        if cls.channel or case["dtype"] == "float32":
            return {"rel": 1e-5, "max": 1e-3}
        return {"rel": 0.008, "max": 0.05}

    @classmethod
    def exact(cls, s):
        groups, heads, dim, vdim = (s.sizes[n] for n in ("groups", "heads", "dim", "vdim"))
        c, k = 2 * groups * dim + heads * vdim, s.taps.shape[1]
        state, out = s.state.double().clone(), []
        for i, it in enumerate(s.ctx.items):
            run = slice(it.first_token, it.first_token + it.end - it.start)
            p, n = s.proj[run].double(), it.end - it.start
            u, tail = _short_convolution(p[:, :c], s.taps.double(), state[i, : (k - 1) * c].view(k - 1, c), it.start)
            q, key = (_unit(u[:, a: a + groups * dim].view(n, groups, dim)).repeat_interleave(heads // groups, 1) for a in (0, groups * dim))
            q, v = q * dim ** -0.5, u[:, 2 * groups * dim:].view(n, heads, vdim)
            if cls.channel:
                beta = torch.sigmoid(p[:, s.beta_at: s.beta_at + heads])
                decay = s.decay[run].double().view(n, heads, dim, 1)
            else:
                beta = torch.sigmoid(s.ba[run, :heads].double())
                decay = torch.exp(-torch.exp(s.a_log.double()) * torch.nn.functional.softplus(s.ba[run, heads:].double() + s.dt_bias.double()))
                decay = decay.view(n, heads, 1, 1)
            m = state[i, (k - 1) * c:].view(heads, dim, vdim)
            o = torch.empty(n, heads, vdim, dtype=torch.float64, device=p.device)
            for t in range(n):
                m = m * decay[t]
                w = beta[t, :, None] * (v[t] - torch.bmm(key[t, :, None], m)[:, 0])
                m = m + key[t, :, :, None] * w[:, None]
                o[t] = torch.bmm(q[t, :, None], m)[:, 0]
            state[i, : (k - 1) * c] = tail.reshape(-1)
            state[i, (k - 1) * c:] = m.reshape(-1)
            if not cls.channel:
                o = o / torch.sqrt((o * o).mean(-1, keepdim=True) + s.eps) * s.gain.double()
                o = (o * torch.nn.functional.silu(p[:, c:].view(n, heads, vdim))).flatten(1)
            out.append(o)
        return torch.cat(out), state


class _ChannelDelta(_Delta):
    channel = True


class _Linear:
    """Gated linear attention: a decay per head and key channel, close to one."""

    @staticmethod
    def sizes(case):
        return dict(heads=8 if case["width"] == 2048 else 16, dim=128, vdim=128)

    @staticmethod
    def prepare(case, rnd):
        sizes = _Linear.sizes(case)
        heads, dim, vdim = sizes["heads"], sizes["dim"], sizes["vdim"]
        ctx, _ = _step(_portions(case), rnd.generator)
        t = ctx.num_tokens
        # the projection's rows carry the output gate and the decay's latent behind q, k and v
        return SimpleNamespace(kind=_Linear, ctx=ctx, sizes=sizes, proj=rnd.normal(t, heads * 2 * (dim + vdim) + 64, dtype=DTYPES[case["dtype"]]),
                               alpha=torch.sigmoid(rnd.normal(t, heads * dim)) ** (1 / 16.0),
                               state=rnd.normal(case["requests"], heads * dim * vdim))

    @staticmethod
    def run(s):
        return ops.linear_attention(s.proj, s.alpha, s.state, s.ctx, **s.sizes), s.state

    @staticmethod
    def work(case):
        z = _Linear.sizes(case)
        t, size = sum(n for n, _ in _portions(case)), DTYPES[case["dtype"]].itemsize
        return {"bytes": t * z["heads"] * (size * (2 * z["dim"] + z["vdim"]) + 4 * (z["dim"] + z["vdim"])) + 8 * case["requests"] * z["heads"] * z["dim"] * z["vdim"],
                "flops": 4 * t * z["heads"] * z["dim"] * z["vdim"]}

    @staticmethod
    def tolerance(case):  # float32 throughout
        return {"rel": 1e-5, "max": 1e-3}

    @staticmethod
    def exact(s):
        heads, dim, vdim = (s.sizes[n] for n in ("heads", "dim", "vdim"))
        state, out = s.state.double().clone(), []
        for i, it in enumerate(s.ctx.items):
            run, n = slice(it.first_token, it.first_token + it.end - it.start), it.end - it.start
            p = s.proj[run].double()
            q, k = (p[:, a: a + heads * dim].view(n, heads, dim) for a in (0, heads * dim))
            v, g = p[:, 2 * heads * dim: 2 * heads * dim + heads * vdim].view(n, heads, vdim), s.alpha[run].double().view(n, heads, dim, 1)
            m, o = state[i].view(heads, dim, vdim), torch.empty(n, heads, vdim, dtype=torch.float64, device=p.device)
            for t in range(n):
                m = g[t] * m + k[t, :, :, None] * v[t, :, None]
                o[t] = torch.bmm(q[t, :, None], m)[:, 0]
            state[i] = m.reshape(-1)
            out.append(o * dim ** -0.5)
        return torch.cat(out), state


# ---- routed experts


class _Experts:
    """The router's choice and the chosen experts, as each design has them; the shared expert's result is given."""

    ROUTER = {
        "gekopel": dict(groups=8, keep=4, scale=2.5),
        "zomolix": dict(groups=8, keep=4, scale=1.0, scores="softmax", group_score="max", normalize=False),
        "bumalix": dict(groups=1, keep=1, scale=1.0, normalize=False),
    }
    GLU = {"gekopel": None, "zomolix": (7.0, 1.702, 1.0), "bumalix": "silu"}
    EXPERTS, TOP = 32, 4

    @classmethod
    def prepare(cls, case, rnd):
        h, t, design = case["width"], case["tokens"], case["design"]
        ff, b16 = h // 2, dict(dtype=torch.bfloat16)
        glu = cls.GLU[design]
        z = rnd.normal(t, cls.EXPERTS + (1 if design == "gekopel" else 0))
        return SimpleNamespace(
            kind=_Experts, x=rnd.normal(t, h, **b16), z=z, correction=rnd.normal(cls.EXPERTS, std=0.05) if design == "gekopel" else None,
            up=rnd.normal(cls.EXPERTS, ff if glu is None else 2 * ff, h, std=0.02, **b16), down=rnd.normal(cls.EXPERTS, h, ff, std=0.02, **b16),
            shared=rnd.normal(t, h, **b16), design=design, glu=glu)

    @classmethod
    def run(cls, s):
        chosen, weight = ops.moe_route(s.z, s.correction, experts=cls.EXPERTS, top=cls.TOP, **cls.ROUTER[s.design])
        out = ops.moe_experts(s.x, chosen, weight, s.up, s.down, activation="relu2" if s.glu is None else None, shared=s.shared,
                              shared_gate=s.z[:, cls.EXPERTS:] if s.design == "gekopel" else None, glu=s.glu,
                              weight_on_input=s.design == "bumalix")
        return out, chosen, weight

    @classmethod
    def work(cls, case):
        h, t = case["width"], case["tokens"]
        matrices = (2 if cls.GLU[case["design"]] is None else 3) * h * (h // 2)
        used = cls.EXPERTS * (1 - (1 - cls.TOP / cls.EXPERTS) ** t)
        return {"bytes": 2 * used * matrices + 6 * t * h, "flops": 2 * t * cls.TOP * matrices}

    @staticmethod
    def tolerance(case):  # the activations, the experts' results and their sum are rounded to bfloat16
        return {"rel": 0.015, "max": 0.1, "differ": 0.001}

    @classmethod
    def exact(cls, s):
        r, e = cls.ROUTER[s.design], cls.EXPERTS
        z = s.z[:, :e].double()
        score = torch.softmax(z, 1) if r.get("scores") == "softmax" else torch.sigmoid(z)
        choice = score if s.correction is None else score + s.correction.double()
        if r["groups"] > 1:
            grouped = choice.view(-1, r["groups"], e // r["groups"])
            best = grouped.amax(2) if r.get("group_score") == "max" else grouped.topk(2, dim=2).values.sum(2)
            kept = torch.zeros_like(best).scatter_(1, best.topk(r["keep"], dim=1).indices, 1.0)
            choice = choice.masked_fill(kept.repeat_interleave(e // r["groups"], 1) == 0, float("-inf"))
        chosen = choice.topk(cls.TOP, dim=1).indices
        weight = score.gather(1, chosen)
        if r.get("normalize", True):
            weight = weight / (weight.sum(1, keepdim=True) + 1e-20)
        weight = weight * r["scale"]
        out = s.shared.double() * (torch.sigmoid(s.z[:, e:].double()) if s.design == "gekopel" else 1.0)
        for i in range(e):
            row, which = (chosen == i).nonzero(as_tuple=True)
            if not len(row):
                continue
            w = weight[row, which, None]
            x = s.x[row].double()
            if s.design == "bumalix":
                x = x * w
            y = x @ s.up[i].double().t()
            if s.glu is None:
                y = torch.relu(y) ** 2
            else:
                g, u = y.chunk(2, dim=1)
                if s.glu == "silu":
                    y = torch.nn.functional.silu(g) * u
                else:
                    limit, alpha, offset = s.glu
                    g, u = g.clamp(max=limit), u.clamp(-limit, limit)
                    y = g * torch.sigmoid(alpha * g) * (u + offset)
            y = y @ s.down[i].double().t()
            out.index_add_(0, row, y if s.design == "bumalix" else y * w)
        return out, None, None


_KINDS = {"step": _Step, "ffn": _FeedForward, "attention": _Attention, "rows": _Rows, "latent": _Latent, "delta": _Delta,
          "channel_delta": _ChannelDelta, "linear": _Linear, "experts": _Experts}
