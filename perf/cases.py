"""What a user of this framework has it do, as cases that can be timed: decode attention over a prefix tree of cached keys
and values (`Attention.forward`, the reference's own benchmark), a serving step around it, the cache layers of the other
decoders (grouped heads, windowed latent rows) on prompts and on decoded tokens, and a whole decoder.

Every kind of case has a class below: what it is in real use, its inputs, one pass through the public entry points, the
work that the pass cannot do without, and the same results in 64 bits.
"""
import math
import os
import sys

import torch

sys.path.insert(1, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "chunk-attention_b200"))
import chunk_attn  # noqa: E402
from chunk_attn import SpanBatch  # noqa: E402

DEVICE = "cuda:0"
DTYPES = {"float16": torch.float16, "bfloat16": torch.bfloat16, "float32": torch.float32}
EPS = 1e-5
BASE = 10000.0


class Draws:
    """Seeded tensors on the GPU, always drawn in the same order."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEVICE).manual_seed(seed)

    def normal(self, *shape, scale=1.0, mean=0.0, dtype=torch.float32):
        return torch.randn(shape, generator=self.g, device=DEVICE).mul_(scale).add_(mean).to(dtype)

    def tokens(self, n, vocab):
        return torch.randint(0, vocab, (n,), generator=self.g, device=DEVICE).tolist()


def item(case):
    return 4 if case["dtype"] == "float32" else 2


def megabytes(n_tokens, token_bytes):
    """A pool for so many tokens and a part-filled chunk or two for each sequence."""
    return int(n_tokens * token_bytes / 2 ** 20) + 64


def lengths(n, longest, ragged):
    """All alike, or spread between half of the longest and the longest."""
    return [max(1, longest - (i * 7919) % (longest // 2 + 1)) if ragged else longest for i in range(n)]


def attend(q, k, v, scale, sink=None):
    """q [T, H, d]; k, v [S, G, .]; every query sees every key.  `sink`: [H] scores of an entry that is dropped again."""
    T, H, _ = q.shape
    G = k.shape[1]
    qg = q.view(T, G, H // G, -1).permute(1, 2, 0, 3).reshape(G, H // G * T, -1)
    s = torch.bmm(qg, k.permute(1, 2, 0)) * scale
    return soften(s.view(G, H // G, T, -1), v, sink)


def soften(s, v, sink):
    """s [G, H / G, T, S] scores, -inf where nothing is seen; [T, H, dv]."""
    G, per, T, S = s.shape
    m = s.amax(-1, keepdim=True)
    if sink is not None:
        z = sink.view(G, per, 1, 1)
        m = torch.maximum(m, z)
    e = torch.exp(s - m)
    total = e.sum(-1, keepdim=True) + (torch.exp(z - m) if sink is not None else 0.0)
    o = torch.bmm(e.view(G, per * T, S), v.transpose(0, 1)).view(G, per, T, -1) / total
    return o.permute(2, 0, 1, 3).reshape(T, G * per, -1)


def causal(q, k, v, scale, sink, window=0, block=512):
    """Attention of a prompt's tokens to themselves and to those before them, at most `window` in all (0: any number)."""
    T, H, _ = q.shape
    G = k.shape[1]
    out = []
    for a in range(0, T, block):
        b = min(T, a + block)
        lo = max(0, a - window + 1) if window else 0
        kk, vv = k[lo:b], v[lo:b]
        qg = q[a:b].view(b - a, G, H // G, -1).permute(1, 2, 0, 3).reshape(G, H // G * (b - a), -1)
        s = (torch.bmm(qg, kk.permute(1, 2, 0)) * scale).view(G, H // G, b - a, b - lo)
        i, j = torch.arange(a, b, device=q.device)[:, None], torch.arange(lo, b, device=q.device)[None]
        hidden = (j > i) | ((j <= i - window) if window else torch.zeros_like(j, dtype=torch.bool))
        out.append(soften(s.masked_fill(hidden, float("-inf")), vv, sink))
    return torch.cat(out)


def pair_frequencies(dims):
    return (BASE ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64) / dims)).to(DEVICE)


def turn_pairs(x, positions, dims, sign=1.0):
    """x [T, heads, d]: the pairs (2 i, 2 i + 1) of the leading dims turned by position times frequency i."""
    a = sign * positions.double()[:, None, None] * pair_frequencies(dims)
    u, w, c, s = x[..., 0:dims:2], x[..., 1:dims:2], torch.cos(a), torch.sin(a)
    turned = torch.stack([u * c - w * s, w * c + u * s], -1).flatten(-2)
    return torch.cat([turned, x[..., dims:]], -1)


def turn_halves(x, positions):
    """x [T, ..., r]: element i and element i + r / 2 turned by position times frequency i."""
    half = x.shape[-1] // 2
    a = positions.double().view((-1,) + (1,) * (x.dim() - 1)) * pair_frequencies(2 * half)
    u, w, c, s = x[..., :half], x[..., half:], torch.cos(a), torch.sin(a)
    return torch.cat([u * c - w * s, w * c + u * s], -1)


def rms(x, w=1.0):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS) * w


def groups_of(heads):
    """Key/value heads of a layer: a quarter of the query heads, or the next number below that divides them."""
    return next(g for g in range(max(1, heads // 4), 0, -1) if heads % g == 0)


def log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


class Decode:
    """One decode step's attention on an up-to-date tree: every sequence has one query, `shared` leading tokens are common
    to all, the rest is each sequence's own.  The reference's benchmark protocol."""

    @staticmethod
    def contexts(case, seed):
        """The shared keys and values (or None), then those of each sequence's own tokens, then the queries."""
        g, dt, H, d = Draws(seed), DTYPES[case["dtype"]], case["heads"], case["dim"]

        def rows(n):
            return g.normal(n, H, d, scale=0.5, dtype=dt), g.normal(n, H, d, scale=0.5, dtype=dt)

        yield rows(case["shared"]) if case["shared"] else None
        for n in lengths(case["seqs"], case["own"], case["ragged"]):
            yield rows(n)
        yield g.normal(case["seqs"], H, d, scale=0.5, dtype=dt)

    @staticmethod
    def tokens(case, i, n):
        return list(range(case["shared"])) + [1_000_000 * (i + 1) + j for j in range(n)]

    @classmethod
    def unique(cls, case):
        return case["shared"] + sum(lengths(case["seqs"], case["own"], case["ragged"]))

    @classmethod
    def prepare(cls, case, seed):
        parts = cls.contexts(case, seed)
        shared = next(parts)
        n_tokens = cls.unique(case) + 2 * case["chunk"] * (case["seqs"] + 2)
        attn = chunk_attn.Attention(n_heads=case["heads"], d_head=case["dim"], chunk_size=case["chunk"], dtype=DTYPES[case["dtype"]],
                                    memory_mb=megabytes(n_tokens, 2 * case["heads"] * case["dim"] * item(case)), device=DEVICE)
        for i in range(case["seqs"]):
            k, v = next(parts)
            tokens = cls.tokens(case, i, k.shape[0])
            if shared is not None:
                k, v = torch.cat([shared[0], k]), torch.cat([shared[1], v])
            attn.add_seq(tokens=tokens, k=k, v=v)
        q = next(parts)
        state = {"attn": attn, "q": q, "host": case["host"]}
        if case["host"]:
            state["q"] = q.cpu().pin_memory()
            state["out"] = torch.empty_like(state["q"]).pin_memory()
        return state

    @staticmethod
    def run(state):
        if state["host"]:
            return state["attn"].forward_host(q=state["q"], out=state["out"])
        return state["attn"].forward(q=state["q"])

    @classmethod
    def work(cls, case):
        per = case["heads"] * case["dim"]
        pairs = case["seqs"] * case["shared"] + sum(lengths(case["seqs"], case["own"], case["ragged"]))
        return {"bytes": item(case) * per * (2 * cls.unique(case) + 2 * case["seqs"]), "flops": 4.0 * per * pairs}

    @classmethod
    def exact(cls, case, seed):
        parts = list(cls.contexts(case, seed))
        shared, q, out = parts[0], parts[-1].double(), []
        if shared is not None:
            shared = shared[0].double(), shared[1].double()
        for i, (k, v) in enumerate(parts[1:-1]):
            k, v = k.double(), v.double()
            if shared is not None:
                k, v = torch.cat([shared[0], k]), torch.cat([shared[1], v])
            out.append(attend(q[i:i + 1], k, v, case["dim"] ** -0.5))
        return torch.cat(out).cpu() if case["host"] else torch.cat(out)

    tolerances = {"float16": {"rel": 1.2e-3, "max": 6e-3}, "float32": {"rel": 1.2e-6, "max": 8e-6}}

    @staticmethod
    def draw(rng):
        pick = rng.random()
        case = {"kind": "decode", "dtype": "float16", "dim": 128, "chunk": 64, "ragged": rng.random() < 0.6, "host": rng.random() < 0.15}
        if pick < 0.45:  # the sizes of 7B to 70B models
            case.update(heads=rng.choice([8, 16, 32, 40]), seqs=log_int(rng, 1, 256), shared=rng.choice([0, log_int(rng, 16, 4096)]))
            most = min(4096, 24_000_000 // (case["heads"] * 128 * case["seqs"]))
            case["own"] = log_int(rng, 4, max(8, most))
        elif pick < 0.8:  # small models and odd heads, half of them in fp32
            case.update(dtype=rng.choice(["float16", "float32"]), dim=rng.choice([32, 64, 64, 80, 96, 128]), chunk=rng.choice([16, 32, 64]),
                        heads=rng.choice([4, 8, 12, 16]), seqs=log_int(rng, 1, 64), shared=rng.choice([0, log_int(rng, 16, 1024)]), own=log_int(rng, 4, 1024))
        else:  # many requests over one long prompt
            case.update(heads=rng.choice([16, 32]), seqs=rng.randint(128, 1024), shared=log_int(rng, 512, 2048), own=rng.randint(1, 32))
        return case


class Serve:
    """One step of continuous batching on a two-level tree (a system prompt, group prompts, own tokens): the oldest
    sequence has finished, a new one takes its place, every sequence appends a token and attends."""

    @staticmethod
    def data(case, seed):
        g, H, dt = Draws(seed), case["heads"], DTYPES[case["dtype"]]

        def rows(n):
            return g.normal(n, H, 128, scale=0.5, dtype=dt), g.normal(n, H, 128, scale=0.5, dtype=dt)

        n = case["seqs"]
        d = {"root": rows(case["root"]), "group": [rows(case["group"]) for _ in range(case["groups"])], "own": [rows(case["own"] + n) for _ in range(n)]}
        d["q"] = g.normal(n, H, 128, scale=0.5, dtype=dt)
        d["new"] = rows(n)
        return d

    @staticmethod
    def sequence(case, data, i, length):
        g = i % case["groups"]
        tokens = list(range(case["root"])) + [10_000 * (g + 1) + j for j in range(case["group"])] + [1_000_000 * (i + 1) + j for j in range(length)]
        parts = data["root"], data["group"][g], [x[:length] for x in data["own"][i]]
        return tokens, torch.cat([p[0] for p in parts]), torch.cat([p[1] for p in parts])

    @classmethod
    def prepare(cls, case, seed):
        data, n = cls.data(case, seed), case["seqs"]
        n_tokens = case["root"] + case["group"] * case["groups"] + n * (case["own"] + n + 4 * 64)
        attn = chunk_attn.Attention(n_heads=case["heads"], d_head=128, chunk_size=64, memory_mb=megabytes(n_tokens, 512 * case["heads"]),
                                    dtype=DTYPES[case["dtype"]], device=DEVICE)
        rows = []
        for i in range(n):  # sequence i has been running for n - 1 - i steps
            tokens, k, v = cls.sequence(case, data, i, case["own"] + n - 1 - i)
            rows.insert(attn.add_seq(tokens=tokens, k=k, v=v), i)
        arrivals = [cls.sequence(case, data, i, case["own"]) for i in range(n)]
        return {"attn": attn, "rows": rows, "arrivals": arrivals, "next": 0, "q": data["q"], "new": data["new"], "ids": list(range(n))}

    @staticmethod
    def run(state):
        attn, rows, oldest = state["attn"], state["rows"], state["next"]
        state["next"] = (oldest + 1) % len(rows)
        row = rows.index(oldest)
        attn.remove_seq(row)
        del rows[row]
        tokens, k, v = state["arrivals"][oldest]
        rows.insert(attn.add_seq(tokens=tokens, k=k, v=v), oldest)
        attn.append_token(tokens=state["ids"], k=state["new"][0], v=state["new"][1])
        return attn.forward(q=state["q"])

    @staticmethod
    def work(case):
        n, per = case["seqs"], 128 * case["heads"]
        own = n * (case["own"] + n / 2.0 + 0.5)
        unique = case["root"] + case["group"] * case["groups"] + own
        # the arrival's own rows and the appended ones are also stored
        return {"bytes": 2.0 * per * (2 * unique + 4 * case["own"] + 4 * n + 2 * n), "flops": 4.0 * per * (n * (case["root"] + case["group"]) + own)}

    @classmethod
    def exact(cls, case, seed):
        data, n, groups = cls.data(case, seed), case["seqs"], case["groups"]
        # rows follow the tree: where a group has whole chunks of its own its sequences stand together, and the newcomer is
        # the last of them; else all stand in the order in which they came
        apart = (case["root"] + case["group"]) // 64 > case["root"] // 64
        order = [i for g in range(groups) for i in range(g, n, groups)] if apart else list(range(n))
        order.remove(0)
        order.insert(len(range(0, n, groups)) - 1 if apart else n - 1, 0)
        out = []
        for row, i in enumerate(order):
            length = case["own"] if i == 0 else case["own"] + n - 1 - i
            _, k, v = cls.sequence(case, data, i, length)
            k, v = (torch.cat([x, y[row:row + 1]]).double() for x, y in zip((k, v), data["new"]))
            out.append(attend(data["q"][row:row + 1].double(), k, v, 128 ** -0.5))
        return torch.cat(out)

    tolerances = {"float16": {"rel": 1.2e-3, "max": 6e-3}}

    @staticmethod
    def draw(rng):
        groups = rng.randint(1, 6)
        return {"kind": "serve", "dtype": "float16", "heads": rng.choice([8, 16, 32]), "groups": groups, "seqs": log_int(rng, max(8, 2 * groups), 128),
                "root": log_int(rng, 32, 1024), "group": log_int(rng, 16, 1024), "own": log_int(rng, 8, 300)}


class Grouped:
    """What the grouped-head layers share: projections [q | k | v], head norms, keys and values turned by their position,
    results turned back, one more entry of score zero in the softmax."""

    @staticmethod
    def cache(case, n_tokens):
        wide = case["kv_heads"] * (case["dim"] + case["vdim"] + 14) * item(case)
        return chunk_attn.Attention.shaped(n_heads=case["heads"], n_kv_heads=case["kv_heads"], d_key=case["dim"], d_value=case["vdim"],
                                           scale=case["dim"] ** -0.5, sink=True, chunk_size=64, memory_mb=megabytes(n_tokens, wide),
                                           dtype=DTYPES[case["dtype"]], device=DEVICE)

    @staticmethod
    def columns(case):
        return case["heads"] * case["dim"] + case["kv_heads"] * (case["dim"] + case["vdim"])

    @staticmethod
    def norms(case, g):
        return g.normal(case["dim"], scale=0.1, mean=1.0), g.normal(case["dim"], scale=0.1, mean=1.0)

    @staticmethod
    def store_args(case, norms):
        return norms + (EPS, case["rot"], pair_frequencies(case["rot"]).float(), pair_frequencies(case["vdim"]).float())

    @classmethod
    def heads(cls, case, qkv, positions, norms):
        """64-bit q, k, v of a sequence's tokens as attention sees them."""
        H, G, d, dv = case["heads"], case["kv_heads"], case["dim"], case["vdim"]
        q, k, v = qkv.double().split([H * d, G * d, G * dv], -1)
        q, k = rms(q.view(-1, H, d), norms[0].double()), rms(k.view(-1, G, d), norms[1].double())
        return turn_pairs(q, positions, case["rot"]), turn_pairs(k, positions, case["rot"]), turn_pairs(v.view(-1, G, dv), positions, dv)

    @staticmethod
    def geometry(rng):
        heads = rng.choice([8, 16, 32])
        case = {"dtype": "bfloat16", "heads": heads, "kv_heads": heads // rng.choice([1, 2, 4, 8])}
        if rng.random() < 0.75:
            case["dim"] = case["vdim"] = rng.choice([64, 128, 128])
        else:
            case["dim"], case["vdim"] = rng.choice([40, 80, 96]), rng.choice([48, 64, 80])
        case["rot"] = rng.choice([case["dim"], case["dim"] // 4 * 2])
        return case

    tolerances = {"bfloat16": {"rel": 1.4e-2, "max": 0.2}, "float32": {"rel": 2e-5, "max": 6e-4}}


class GroupedPrompts(Grouped):
    """One layer's cache and attention for whole prompts: rows in the tree, keys and values stored, causal attention, and
    the sequences leave again."""

    @classmethod
    def data(cls, case, seed):
        g = Draws(seed)
        lens = lengths(case["seqs"], case["tokens"], case["ragged"])
        return lens, cls.norms(case, g), g.normal(sum(lens), cls.columns(case), dtype=DTYPES[case["dtype"]])

    @classmethod
    def prepare(cls, case, seed):
        lens, norms, qkv = cls.data(case, seed)
        tokens = [[1_000_000 * (i + 1) + j for j in range(n)] for i, n in enumerate(lens)]
        return {"cache": cls.cache(case, sum(lens) + 128 * len(lens)), "tokens": tokens, "qkv": qkv, "args": cls.store_args(case, norms)}

    @staticmethod
    def run(state):
        cache, tokens = state["cache"], state["tokens"]
        n = len(tokens)
        cache.extend([-1] * n, tokens)
        spans = SpanBatch(tokens, [0] * n, list(range(n)), torch.device(DEVICE))
        q = cache.store_qkv(state["qkv"], spans.positions, *state["args"])
        o = cache.forward_rows(q, spans.positions, state["args"][-1], spans.entry_of)
        for row in reversed(range(n)):
            cache.remove_seq(row)
        return o

    @classmethod
    def work(cls, case):
        lens = lengths(case["seqs"], case["tokens"], case["ragged"])
        per = case["heads"] * (case["dim"] + case["vdim"])
        return {"bytes": float(item(case) * sum(lens) * (cls.columns(case) + case["kv_heads"] * (case["dim"] + case["vdim"]) + case["heads"] * case["vdim"])),
                "flops": sum(n * (n + 1.0) for n in lens) * per}

    @classmethod
    def exact(cls, case, seed):
        lens, norms, qkv = cls.data(case, seed)
        out, zero = [], torch.zeros(case["heads"], dtype=torch.float64, device=DEVICE)
        for part in qkv.split(lens):
            pos = torch.arange(part.shape[0], device=DEVICE)
            q, k, v = cls.heads(case, part, pos, norms)
            out.append(turn_pairs(causal(q, k, v, case["dim"] ** -0.5, zero), pos, case["vdim"], -1.0))
        return torch.cat(out)

    @classmethod
    def draw(cls, rng):
        case = dict(kind="grouped prompts", **cls.geometry(rng))
        n = log_int(rng, 1, 24)
        case.update(seqs=n, tokens=log_int(rng, 16, min(4096, 8192 // n)), ragged=rng.random() < 0.6)
        if rng.random() < 0.15:
            case.update(dtype="float32", tokens=min(case["tokens"], 1024 // n + 8))
        return case


class GroupedDecode(Grouped):
    """One layer's decode attention with grouped heads, on an up-to-date tree."""

    @classmethod
    def data(cls, case, seed):
        g, dt = Draws(seed), DTYPES[case["dtype"]]
        norms = cls.norms(case, g)
        prompts = [g.normal(n, cls.columns(case), dtype=dt) for n in lengths(case["seqs"], case["tokens"], case["ragged"])]
        return norms, prompts, g.normal(case["seqs"], cls.columns(case), dtype=dt)

    @classmethod
    def prepare(cls, case, seed):
        norms, prompts, last = cls.data(case, seed)
        args, dev = cls.store_args(case, norms), torch.device(DEVICE)
        cache = cls.cache(case, sum(p.shape[0] + 192 for p in prompts))
        for i, p in enumerate(prompts):
            tokens = [1_000_000 * (i + 1) + j for j in range(p.shape[0])]
            cache.extend([-1], [tokens])
            cache.store_qkv(p, SpanBatch([tokens], [0], [i], dev).positions, *args)
        n = len(prompts)
        spans = SpanBatch([[0]] * n, [p.shape[0] for p in prompts], list(range(n)), dev)
        q = cache.store_qkv(last, spans.positions, *args, append_tokens=[0] * n)
        return {"cache": cache, "q": q, "spans": spans, "freq": args[-1]}

    @staticmethod
    def run(state):
        return state["cache"].forward_rows(state["q"], state["spans"].positions, state["freq"])

    @staticmethod
    def work(case):
        seen = sum(lengths(case["seqs"], case["tokens"], case["ragged"])) + case["seqs"]
        per = case["dim"] + case["vdim"]
        return {"bytes": float(item(case) * per * (case["kv_heads"] * seen + case["heads"] * case["seqs"])), "flops": 2.0 * case["heads"] * per * seen}

    @classmethod
    def exact(cls, case, seed):
        norms, prompts, last = cls.data(case, seed)
        out, zero = [], torch.zeros(case["heads"], dtype=torch.float64, device=DEVICE)
        for i, p in enumerate(prompts):
            pos = torch.arange(p.shape[0] + 1, device=DEVICE)
            q, k, v = cls.heads(case, torch.cat([p, last[i:i + 1]]), pos, norms)
            out.append(turn_pairs(attend(q[-1:].contiguous(), k, v, case["dim"] ** -0.5, zero), pos[-1:], case["vdim"], -1.0))
        return torch.cat(out)

    @classmethod
    def draw(cls, rng):
        case = dict(kind="grouped decode", **cls.geometry(rng))
        n = log_int(rng, 1, 256)
        case.update(seqs=n, tokens=log_int(rng, 16, min(8192, max(32, 131072 // n))), ragged=rng.random() < 0.6)
        if rng.random() < 0.15:
            case.update(dtype="float32", tokens=max(16, min(case["tokens"], 8192 // n)))
        return case


class Latent:
    """What the latent-attention layers share: one cached row per token for all heads, a latent and a turned key part."""

    @staticmethod
    def cache(case, n_tokens):
        wide = (case["latent"] + case["rot"] + 63) * item(case)
        return chunk_attn.Attention.latent(n_heads=case["heads"], latent=case["latent"], rotated=case["rot"], scale=(case["dim"] + case["rot"]) ** -0.5,
                                           window=case["window"], chunk_size=64, memory_mb=megabytes(n_tokens, wide), dtype=DTYPES[case["dtype"]], device=DEVICE)

    @staticmethod
    def weights(case, g):
        """Norms of the query latent and of the cached one, and a sink for every head."""
        return g.normal(case["q_rank"], scale=0.1, mean=1.0), g.normal(case["latent"], scale=0.1, mean=1.0), g.normal(case["heads"])

    @staticmethod
    def columns(case):
        return case["q_rank"] + case["latent"] + case["rot"]

    @staticmethod
    def frequencies(case):
        f = pair_frequencies(case["rot"])
        return torch.stack([f.float(), (f - f.float().double()).float()])

    @staticmethod
    def entries(case, x, positions, kv_norm):
        """64-bit latents and turned key parts of a sequence's tokens."""
        x = x[:, case["q_rank"]:].double()
        return rms(x[:, :case["latent"]], kv_norm.double()), turn_halves(x[:, case["latent"]:], positions)

    @staticmethod
    def seen(case, start, n):
        """How many tokens the positions start .. start + n - 1 see in all."""
        w = case["window"] or start + n
        return sum(min(p + 1, w) for p in range(start, start + n))

    @staticmethod
    def geometry(rng):
        case = {"dtype": "bfloat16", "heads": rng.choice([8, 16, 32, 64]), "dim": 128, "rot": 64, "vdim": 128, "q_rank": rng.choice([384, 768, 1536]),
                "latent": rng.choice([256, 512, 512]), "window": rng.choice([0, log_int(rng, 100, 4096)])}
        if rng.random() < 0.25:
            case.update(dim=64, rot=rng.choice([32, 64]), vdim=64)
        return case

    tolerances = {"bfloat16": {"rel": 1.4e-2, "max": 0.2}, "float32": {"rel": 2e-5, "max": 6e-4}}


class LatentPrompts(Latent):
    """One layer's cache and attention for whole prompts: rows stored, the rows of the windows gathered, one GEMM expands
    them into every head's keys and values, windowed attention; the sequences leave again."""

    @classmethod
    def data(cls, case, seed):
        g, dt, H = Draws(seed), DTYPES[case["dtype"]], case["heads"]
        lens = lengths(case["seqs"], case["tokens"], case["ragged"])
        expand = g.normal(H * (case["dim"] + case["vdim"]), case["latent"], scale=case["latent"] ** -0.5, dtype=dt)
        return lens, cls.weights(case, g), expand, g.normal(sum(lens), cls.columns(case), dtype=dt), g.normal(sum(lens), H, case["dim"] + case["rot"], dtype=dt)

    @classmethod
    def prepare(cls, case, seed):
        lens, weights, expand, x, q = cls.data(case, seed)
        tokens = [[1_000_000 * (i + 1) + j for j in range(n)] for i, n in enumerate(lens)]
        return {"cache": cls.cache(case, sum(lens) + 128 * len(lens)), "tokens": tokens, "weights": weights, "expand": expand, "x": x, "q": q,
                "freq": cls.frequencies(case), "vdim": case["vdim"]}

    @staticmethod
    def run(state):
        cache, tokens, freq = state["cache"], state["tokens"], state["freq"]
        q_norm, kv_norm, sink = state["weights"]
        n = len(tokens)
        cache.extend([-1] * n, tokens)
        spans = SpanBatch(tokens, [0] * n, list(range(n)), torch.device(DEVICE))
        c = cache.store_latent(state["x"], spans.positions, q_norm, kv_norm, EPS, freq)
        lat, rot = cache.gather_latents()
        kv = torch.nn.functional.linear(lat, state["expand"])
        o = cache.forward_expanded(state["q"], kv, rot, spans.positions, freq, sink, state["vdim"])
        for row in reversed(range(n)):
            cache.remove_seq(row)
        return c, o

    @classmethod
    def work(cls, case):
        lens = lengths(case["seqs"], case["tokens"], case["ragged"])
        T, H, d, r, dv, R = sum(lens), case["heads"], case["dim"], case["rot"], case["vdim"], case["latent"]
        pairs = sum(cls.seen(case, 0, n) for n in lens)
        return {"bytes": float(item(case) * (T * (cls.columns(case) + case["q_rank"] + R + r + H * (d + r + dv)) + H * (d + dv) * R)),
                "flops": 2.0 * T * H * (d + dv) * R + 2.0 * pairs * H * (d + r + dv)}

    @classmethod
    def exact(cls, case, seed):
        lens, (q_norm, kv_norm, sink), expand, x, q = cls.data(case, seed)
        H, d, dv, scale = case["heads"], case["dim"], case["vdim"], (case["dim"] + case["rot"]) ** -0.5
        cs, out = [], []
        for xs, qs in zip(x.split(lens), q.split(lens)):
            pos = torch.arange(xs.shape[0], device=DEVICE)
            cs.append(rms(xs[:, :case["q_rank"]].double(), q_norm.double()))
            lat, rot = cls.entries(case, xs, pos, kv_norm)
            kv = lat @ expand.double().t()
            k = torch.cat([kv[:, :H * d].view(-1, H, d), rot[:, None].expand(-1, H, -1)], -1)
            qs = qs.double()
            qs = torch.cat([qs[..., :d], turn_halves(qs[..., d:], pos)], -1)
            out.append(causal(qs, k, kv[:, H * d:].view(-1, H, dv), scale, sink.double(), case["window"]))
        return torch.cat(cs), torch.cat(out)

    @classmethod
    def draw(cls, rng):
        case = dict(kind="latent prompts", **cls.geometry(rng))
        n = log_int(rng, 1, 16)
        case.update(heads=min(case["heads"], 32), seqs=n, tokens=log_int(rng, 32, min(4096, 8192 // n)), ragged=rng.random() < 0.6)
        return case


class LatentDecode(Latent):
    """One layer's decode attention in the latent space, on an up-to-date tree."""

    @classmethod
    def data(cls, case, seed):
        g, dt, n, H = Draws(seed), DTYPES[case["dtype"]], case["seqs"], case["heads"]
        weights = cls.weights(case, g)
        prompts = [g.normal(t, cls.columns(case), dtype=dt) for t in lengths(n, case["tokens"], case["ragged"])]
        return (weights, prompts, g.normal(n, cls.columns(case), dtype=dt), g.normal(n, H, case["latent"], scale=(case["dim"] / case["latent"]) ** 0.5, dtype=dt),
                g.normal(n, H, case["dim"] + case["rot"], dtype=dt))

    @classmethod
    def prepare(cls, case, seed):
        (q_norm, kv_norm, sink), prompts, last, q_lat, q = cls.data(case, seed)
        freq, dev, n = cls.frequencies(case), torch.device(DEVICE), case["seqs"]
        cache = cls.cache(case, sum(p.shape[0] + 192 for p in prompts))
        for i, p in enumerate(prompts):
            tokens = [1_000_000 * (i + 1) + j for j in range(p.shape[0])]
            cache.extend([-1], [tokens])
            cache.store_latent(p, SpanBatch([tokens], [0], [i], dev).positions, q_norm, kv_norm, EPS, freq)
        spans = SpanBatch([[0]] * n, [p.shape[0] for p in prompts], list(range(n)), dev)
        cache.store_latent(last, spans.positions, q_norm, kv_norm, EPS, freq, append_tokens=[0] * n)
        return {"cache": cache, "q_lat": q_lat, "q": q, "spans": spans, "freq": freq, "sink": sink}

    @staticmethod
    def run(state):
        return state["cache"].forward_latent(state["q_lat"], state["q"], state["spans"].positions, state["freq"], state["sink"])

    @classmethod
    def work(cls, case):
        n, H, R, r = case["seqs"], case["heads"], case["latent"], case["rot"]
        seen = sum(cls.seen(case, t, 1) for t in lengths(n, case["tokens"], case["ragged"]))
        return {"bytes": float(item(case) * (seen * (R + r) + n * H * (2 * R + r))), "flops": 2.0 * seen * H * (2 * R + r)}

    @classmethod
    def exact(cls, case, seed):
        (_, kv_norm, sink), prompts, last, q_lat, q = cls.data(case, seed)
        out = []
        for i, p in enumerate(prompts):
            pos = torch.arange(p.shape[0] + 1, device=DEVICE)
            lat, rot = cls.entries(case, torch.cat([p, last[i:i + 1]]), pos, kv_norm)
            lo = max(0, p.shape[0] + 1 - case["window"]) if case["window"] else 0
            turned = turn_halves(q[i:i + 1, :, case["dim"]:].double(), pos[-1:])
            qq = torch.cat([q_lat[i:i + 1].double(), turned], -1)
            k = torch.cat([lat, rot], -1)[lo:, None]
            out.append(attend(qq, k, lat[lo:, None], (case["dim"] + case["rot"]) ** -0.5, sink.double()))
        return torch.cat(out)

    @classmethod
    def draw(cls, rng):
        case = dict(kind="latent decode", **cls.geometry(rng))
        n = log_int(rng, 1, 256)
        case.update(seqs=n, tokens=log_int(rng, 16, min(8192, max(32, 131072 // n))), ragged=rng.random() < 0.6)
        return case


class Decoder:
    """A whole decoder of scan, attention and linear-attention layers: prompts in, then given tokens decoded one by one (a
    scored continuation), the logits of every step out, and the sequences leave again."""

    @staticmethod
    def config(case):
        W, ff = case["width"], {"kind": "dense", "ff": case["ff"]}
        H = W // 128
        kinds = {
            "m": {"type": "mamba1", "mlp": None, "mixer": {"inner": 2 * W, "state": 16, "dt_rank": W // 16, "conv": 4}},
            "a": {"type": "attention", "mlp": ff, "mixer": {"heads": H, "kv_heads": groups_of(H), "dim": 128, "vdim": 128, "rot": {"base": BASE, "dims": 128},
                                                             "scale": 128 ** -0.5}},
            "l": {"type": "lightning", "mlp": None, "mixer": {"heads": H, "dim": 128, "vdim": 128, "decay": [1.0 - 2.0 ** (-5 - i / 4) for i in range(H)]}},
        }
        return {"architecture": "Gagorax", "vocab": case["vocab"], "width": W, "layers": [kinds[c] for c in case["layers"]], "norm": {"eps": EPS}}

    @classmethod
    def weights(cls, case, g):
        """Named tensors: matrices N(0, 1 / fan-in), step sizes and decays in their usual ranges, norms near one."""
        W, w = case["width"], {}

        def matrix(name, rows, cols):
            w[name] = g.normal(rows, cols, scale=cols ** -0.5, dtype=torch.bfloat16)

        def vector(name, mean, spread, *shape):
            w[name] = g.normal(*shape, scale=spread, mean=mean, dtype=torch.bfloat16)

        w["embed"] = g.normal(case["vocab"], W, dtype=torch.bfloat16)
        for i, spec in enumerate(cls.config(case)["layers"]):
            p, m, x = "l%d." % i, spec["mixer"], "l%d.mix." % i
            vector(p + "norm1", 1.0, 0.1, W)
            vector(p + "shift", 0.3, 0.2, W)
            matrix(p + "rg1", W, W)
            vector(p + "rg1.b", 0.0, 0.5, W)
            if spec["type"] == "mamba1":
                C, N, R = m["inner"], m["state"], m["dt_rank"]
                matrix(x + "in", 2 * C, W)
                vector(x + "conv", 0.0, 0.5, C, m["conv"])
                vector(x + "conv.b", 0.0, 0.1, C)
                matrix(x + "x", R + 2 * N, C)
                matrix(x + "dt", C, R)
                vector(x + "dt.b", -3.0, 1.0, C)
                w[x + "A_log"] = torch.log(torch.arange(1, N + 1, device=DEVICE).float()).repeat(C, 1).to(torch.bfloat16)
                vector(x + "D", 1.0, 0.1, C)
                matrix(x + "o", W, C)
                continue
            G = m.get("kv_heads", m["heads"])
            matrix(x + "q", m["heads"] * m["dim"], W)
            matrix(x + "k", G * m["dim"], W)
            matrix(x + "v", G * m["vdim"], W)
            matrix(x + "o", W, m["heads"] * m["vdim"])
            if spec["type"] == "lightning":
                matrix(x + "g", m["heads"] * m["vdim"], W)
                vector(x + "norm", 1.0, 0.1, m["heads"] * m["vdim"])
                continue
            vector(x + "q.norm", 1.0, 0.1, m["dim"])
            vector(x + "k.norm", 1.0, 0.1, m["dim"])
            vector(p + "norm2", 1.0, 0.1, W)
            matrix(p + "rg2", W, W)
            vector(p + "rg2.b", 0.0, 0.5, W)
            matrix(p + "mlp.up", spec["mlp"]["ff"], W)
            matrix(p + "mlp.down", W, spec["mlp"]["ff"])
        vector("final.norm", 1.0, 0.1, W)
        matrix("head", case["vocab"], W)
        return w

    @classmethod
    def data(cls, case, seed):
        g = Draws(seed)
        w = cls.weights(case, g)
        return w, [g.tokens(n + case["steps"], case["vocab"]) for n in lengths(case["seqs"], case["tokens"], case["ragged"])]

    @classmethod
    def prepare(cls, case, seed):
        from chunk_attn.models.gagorax import GagoraxConfig, GagoraxForCausalLM
        w, tokens = cls.data(case, seed)
        config = GagoraxConfig.from_dict(cls.config(case), torch_dtype=DTYPES[case["dtype"]], torch_device=DEVICE, state_slots=case["seqs"])
        model = GagoraxForCausalLM(config, w)
        return {"model": model, "caches": model.create_kv_caches(max_tokens=sum(len(t) + 128 for t in tokens)), "tokens": tokens, "steps": case["steps"]}

    @staticmethod
    def run(state):
        from chunk_attn.models.sequence import Sequence
        model, caches, steps = state["model"], state["caches"], state["steps"]
        seqs = [Sequence(t[:len(t) - steps]) for t in state["tokens"]]
        out = [model.logits(seqs, caches, True)]
        for k in range(steps):
            for s, t in zip(seqs, state["tokens"]):
                s.append(t[len(t) - steps + k])
            out.append(model.logits(seqs, caches, False))
        for row in reversed(range(len(seqs))):
            for c in caches:
                c.remove_seq(row)
        return out

    @classmethod
    def work(cls, case):
        W, ff, V = case["width"], case["ff"], case["vocab"]
        H, C = W // 128, 2 * W
        G = groups_of(H)
        per = {"m": W * 2 * C + C * (W // 16 + 32) + C * (W // 16) + C * W + W * W, "a": W * (H + 2 * G) * 128 + 2 * W * W + W * W + 2 * W * ff, "l": 6 * W * W}
        params = sum(per[c] for c in case["layers"])
        lens, steps, n = lengths(case["seqs"], case["tokens"], case["ragged"]), case["steps"], case["seqs"]
        T, layers = sum(lens) + n * steps, case["layers"]
        flops = 2.0 * T * params + 2.0 * n * (1 + steps) * V * W
        flops += layers.count("a") * sum(512.0 * H * t * (t + 1) / 2 for t in (x + steps for x in lens))
        flops += layers.count("l") * T * H * 4.0 * 128 * 128 + layers.count("m") * T * C * 16 * 7.0
        # per step the weights, the rows that attention sees and the states; the prompts' tokens only have to come in
        seen = sum(x + k + 1 for x in lens for k in range(steps))
        nbytes = item(case) * (1 + steps) * (params + V * W) + item(case) * (layers.count("a") * 256 * G * (seen + T)) + 4.0 * n * (1 + steps) * V
        nbytes += 8.0 * n * steps * (layers.count("m") * C * 19 + layers.count("l") * H * 128 * 128)
        return {"bytes": nbytes, "flops": flops}

    @classmethod
    def exact(cls, case, seed):
        w, tokens = cls.data(case, seed)
        w = {k: v.double() for k, v in w.items()}
        T, n = max(len(t) for t in tokens), len(tokens)
        ids = torch.tensor([t + [0] * (T - len(t)) for t in tokens], device=DEVICE)  # what follows a sequence's end changes nothing before it
        x = w["embed"][ids]
        silu = torch.nn.functional.silu
        for i, spec in enumerate(cls.config(case)["layers"]):
            p, m, mix = "l%d." % i, spec["mixer"], "l%d.mix." % i
            h = x + (torch.cat([torch.zeros_like(x[:, :1]), x[:, :-1]], 1) - x) * w[p + "shift"]

            def project(name, y=h):
                return y @ w[mix + name].t()

            if spec["type"] == "mamba1":
                C, N, R, K = m["inner"], m["state"], m["dt_rank"], m["conv"]
                u, z = project("in").split(C, -1)
                padded = torch.cat([u.new_zeros(n, K - 1, C), u], 1)
                u = silu(sum(padded[:, j:j + T] * w[mix + "conv"][:, j] for j in range(K)) + w[mix + "conv.b"])
                del padded
                proj = project("x", u)
                dt = torch.nn.functional.softplus(project("dt", proj[..., :R]) + w[mix + "dt.b"], threshold=50.0)
                A, S, y = -torch.exp(w[mix + "A_log"]), u.new_zeros(n, C, N), torch.empty_like(u)
                for t in range(T):
                    S = torch.exp(dt[:, t, :, None] * A) * S + (dt[:, t] * u[:, t])[..., None] * proj[:, t, None, R:R + N]
                    y[:, t] = (S * proj[:, t, None, R + N:]).sum(-1)
                r = project("o", (y + w[mix + "D"] * u) * silu(z))
                del u, z, y, dt, S
            elif spec["type"] == "attention":
                pos, zero = torch.arange(T, device=DEVICE), torch.zeros(m["heads"], dtype=torch.float64, device=DEVICE)
                o = []
                for b in range(n):
                    q, k, v = (project(name, h[b]).view(T, -1, 128) for name in ("q", "k", "v"))
                    q, k = turn_pairs(rms(q, w[mix + "q.norm"]), pos, 128), turn_pairs(rms(k, w[mix + "k.norm"]), pos, 128)
                    o.append(turn_pairs(causal(q, k, turn_pairs(v, pos, 128), m["scale"], zero), pos, 128, -1.0).reshape(T, -1))
                r = project("o", torch.stack(o))
            else:
                q, k, v = (silu(project(name)).view(n, T, m["heads"], 128) for name in ("q", "k", "v"))
                decay = torch.tensor(m["decay"], dtype=torch.float64, device=DEVICE)[:, None, None]
                S, o = q.new_zeros(n, m["heads"], 128, 128), torch.empty_like(q)
                for t in range(T):
                    S = decay * S + k[:, t, :, :, None] * v[:, t, :, None, :]
                    o[:, t] = (q[:, t, :, None, :] @ S)[:, :, 0]
                r = project("o", rms(o.reshape(n, T, -1), w[mix + "norm"]) * torch.sigmoid(project("g")))
                del q, k, v, o, S
            x = x + rms(r * torch.sigmoid(x @ w[p + "rg1"].t() + w[p + "rg1.b"]), w[p + "norm1"])
            if spec["mlp"] is not None:
                r = torch.nn.functional.gelu(x @ w[p + "mlp.up"].t(), approximate="tanh") @ w[p + "mlp.down"].t()
                x = x + rms(r * torch.sigmoid(x @ w[p + "rg2"].t() + w[p + "rg2.b"]), w[p + "norm2"])
        x = rms(x, w["final.norm"])
        at = torch.arange(n, device=DEVICE)
        first = torch.tensor([len(t) - case["steps"] - 1 for t in tokens], device=DEVICE)
        return [x[at, first + k] @ w["head"].t() for k in range(case["steps"] + 1)]

    tolerances = {"bfloat16": {"rel": 2.5e-2, "max": 0.15}, "float32": {"rel": 1e-5, "max": 6e-5}}

    @staticmethod
    def draw(rng):
        n = log_int(rng, 1, 16)
        width = 128 * rng.randint(4, 16)
        case = {"kind": "decoder", "dtype": "bfloat16", "width": width, "ff": 64 * rng.randint(width // 32, width // 20), "vocab": rng.choice([4000, 8192, 32000]),
                "layers": "".join(rng.choice("mal") for _ in range(rng.randint(1, 4))), "seqs": n, "tokens": log_int(rng, 16, min(2048, 8192 // n)),
                "steps": rng.randint(0, 4), "ragged": rng.random() < 0.6}
        if rng.random() < 0.15:
            case.update(dtype="float32", tokens=min(case["tokens"], 256))
        return case


KINDS = {"decode": Decode, "serve": Serve, "grouped prompts": GroupedPrompts, "grouped decode": GroupedDecode, "latent prompts": LatentPrompts,
         "latent decode": LatentDecode, "decoder": Decoder}


def listed():
    decode = {"kind": "decode", "dtype": "float16", "heads": 32, "dim": 128, "chunk": 64, "ragged": False, "host": False}
    grouped = {"dtype": "bfloat16", "heads": 32, "kv_heads": 8, "dim": 128, "vdim": 128, "rot": 128}
    latent = {"dtype": "bfloat16", "heads": 32, "dim": 128, "rot": 64, "vdim": 128, "q_rank": 1536, "latent": 512}
    return [
        # the smallest call: four short sequences of a small fp32 model
        dict(decode, name="decode fp32 4x288", dtype="float32", heads=8, dim=64, chunk=32, seqs=4, shared=256, own=32),
        # one user's conversation on a 7B model, queries and results in host memory
        dict(decode, name="decode one request", seqs=1, shared=0, own=1500, host=True),
        # the heads that `Attention` takes by default, a small chat batch of odd lengths
        dict(decode, name="decode heads of 64", heads=12, dim=64, seqs=16, shared=500, own=333, ragged=True),
        # the headline: a batch over one long prompt
        dict(decode, name="decode 32x(2048+512)", seqs=32, shared=2048, own=512),
        # long conversations that share nothing: as much K/V as a layer reads in earnest
        dict(decode, name="decode 64x4096", seqs=64, shared=0, own=4096, ragged=True),
        # a thousand requests that have just begun, over one system prompt
        dict(decode, name="decode 1024x(2048+8)", seqs=1024, shared=2048, own=8),
        # continuous batching over a two-level tree
        {"name": "serve 128", "kind": "serve", "dtype": "float16", "heads": 32, "groups": 4, "seqs": 128, "root": 1024, "group": 1024, "own": 192},
        # a layer with grouped heads: a batch of prompts, and the decode after it
        dict(grouped, name="grouped prompts 8x1024", kind="grouped prompts", seqs=8, tokens=1024, ragged=False),
        dict(grouped, name="grouped decode 64x1024", kind="grouped decode", seqs=64, tokens=1024, ragged=True),
        # a layer of windowed latent attention: one long prompt, and the decode of a batch
        dict(latent, name="latent prompts 1x4096", kind="latent prompts", window=1024, seqs=1, tokens=4096, ragged=False),
        dict(latent, name="latent decode 64x1024", kind="latent decode", window=4096, seqs=64, tokens=1024, ragged=True),
        # a decoder with one layer of each kind: prompts, then two tokens
        {"name": "decoder 8x1000", "kind": "decoder", "dtype": "bfloat16", "width": 4096, "ff": 11008, "vocab": 32000, "layers": "mal", "seqs": 8,
         "tokens": 1000, "steps": 2, "ragged": True},
    ]


def draw(rng):
    kind = rng.choice(["decode"] * 5 + ["serve", "grouped prompts", "grouped decode", "grouped decode", "latent prompts", "latent decode", "decoder"])
    return KINDS[kind].draw(rng)


def prepare(case, seed):
    state = KINDS[case["kind"]].prepare(case, seed)
    state["kind"] = case["kind"]
    return state


def run(state):
    return KINDS[state["kind"]].run(state)


def work(case):
    return KINDS[case["kind"]].work(case)


def tolerance(case):
    return KINDS[case["kind"]].tolerances[case["dtype"]]


def exact(case, seed):
    return KINDS[case["kind"]].exact(case, seed)
