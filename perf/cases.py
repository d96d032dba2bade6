"""Timed cases: what a program that serves models with this framework has it do, through its public entry points.

Kinds of case and where their sizes come from:

  linear            one linear layer, y = x W^T in bf16: one token, a batch of decoding sequences, a prompt
  paged_decode      one new token per sequence over a paged cache (bf16 and f16, head sizes 64 and 128)
  prefill           prompts packed one after the other, with the write of their keys and values into the paged cache
  paged_attention   the tensor surface's attention for one step of a running batch: chunks of prompts behind earlier
                    context beside sequences that decode one token
  sdpa              dense attention in f32
  llama             decode and prompt steps of six layers of the Llama-3-8B shape
  kavalorn,         decode and prompt steps of the two layer-list decoders, six layers of width 2048
  vatolorn

Sizes are those of the benchmark's workloads and of what lies around them; ``draw`` spreads them.  Lengths of ragged batches
belong to the case, values belong to the seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from singe_b200 import hybrid, llama, ops
from singe_b200.parallel_mixer import ChunkedAttentionConfig, GatedDeltaConfig, ParallelConfig, Rotation, YarnScaling

PAGE = 16
HEADS, KV_HEADS = 32, 8
TYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}

# (columns, rows) of the weight matrices of the decoders below: 4096 and 2048 wide
LINEAR_SHAPES = ((4096, 4096), (6144, 4096), (28672, 4096), (14336, 4096), (4096, 14336), (2048, 2048), (8192, 2048),
                 (2048, 8192), (32000, 2048))


def listed():
    return [
        # a single chat: the linear layer of one token, latency and weight streaming
        {"name": "linear one token", "kind": "linear", "m": 1, "n": 4096, "k": 4096},
        # the down projection of a well filled decode batch
        {"name": "linear decode batch", "kind": "linear", "m": 128, "n": 4096, "k": 14336},
        # the up projection of a long prompt
        {"name": "linear prompt", "kind": "linear", "m": 4096, "n": 14336, "k": 4096},
        # the smallest attention call: a few chats, half precision, heads of 64
        {"name": "paged decode few", "kind": "paged_decode", "batch": 4, "least": 200, "most": 1100, "dim": 64, "type": "f16"},
        # an ordinary decode batch with contexts of all lengths
        {"name": "paged decode batch", "kind": "paged_decode", "batch": 32, "least": 128, "most": 4096, "dim": 128, "type": "bf16"},
        # four prompts read at once
        {"name": "prefill four prompts", "kind": "prefill", "prompts": 4, "least": 1024, "most": 8192, "spread": "halves", "dim": 128},
        # one step of continuous batching
        {"name": "paged attention mixed step", "kind": "paged_attention", "chunks": 4, "chunk": 512, "decoding": 28, "most": 3000,
         "window": 0, "type": "bf16"},
        # an f32 encoder-sized attention
        {"name": "sdpa f32", "kind": "sdpa", "batch": 1, "heads": 8, "kv_heads": 8, "length": 512, "dim": 64, "causal": True},
        # decode at full load, and many prompts in one step
        {"name": "llama decode", "kind": "llama", "step": "decode", "sequences": 64, "least": 2048, "most": 2048},
        {"name": "llama prompts", "kind": "llama", "step": "prompt", "sequences": 64, "least": 60, "most": 480},
        {"name": "kavalorn prompts", "kind": "kavalorn", "step": "prompt", "sequences": 4, "least": 2048, "most": 2048},
        {"name": "vatolorn decode", "kind": "vatolorn", "step": "decode", "sequences": 64, "least": 2048, "most": 2048},
    ]


def draw(rng):
    log = lambda low, high: int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))
    kind = rng.choice(["linear"] * 3 + ["paged_decode"] * 2 + ["prefill", "paged_attention", "sdpa"] + ["llama"] * 2
                      + ["kavalorn", "vatolorn"])
    if kind == "linear":
        n, k = rng.choice(LINEAR_SHAPES)
        return {"kind": kind, "m": log(1, 6000), "n": n, "k": k}
    if kind == "paged_decode":
        most = log(64, 8192)
        return {"kind": kind, "batch": log(1, 96), "least": max(1, most // rng.choice((1, 4, 32))), "most": most,
                "dim": rng.choice((64, 128, 128)), "type": rng.choice(("bf16", "bf16", "bf16", "f16"))}
    if kind == "prefill":
        most = log(48, 8192)
        return {"kind": kind, "prompts": rng.randint(1, 8), "least": max(1, most // rng.choice((1, 4, 16))), "most": most,
                "spread": "uniform", "dim": rng.choice((64, 128, 128))}
    if kind == "paged_attention":
        return {"kind": kind, "chunks": rng.randint(1, 4), "chunk": log(16, 520), "decoding": rng.randint(0, 48),
                "most": log(100, 3000), "window": rng.choice((0, 0, 0, 1024)), "type": "bf16"}
    if kind == "sdpa":
        heads = rng.choice((4, 6, 8, 12))
        return {"kind": kind, "batch": rng.randint(1, 2), "heads": heads, "kv_heads": rng.choice((heads, heads // 2)),
                "length": log(32, 1500), "dim": rng.choice((64, 64, 128)), "causal": rng.random() < 0.6}
    if rng.random() < 0.5:
        most = log(100, 3500)
        return {"kind": kind, "step": "decode", "sequences": log(1, 64), "least": max(1, most // rng.choice((1, 4))), "most": most}
    sequences = log(1, 48)
    most = min(log(16, 4096), 6000 // sequences)
    return {"kind": kind, "step": "prompt", "sequences": sequences, "least": max(1, most // rng.choice((1, 4))), "most": most}


# ------------------------------------------------------------------------------------------------
# shared
# ------------------------------------------------------------------------------------------------

def _lengths(count, least, most, salt):
    """The lengths of a ragged batch: drawn once for the sizes of the case."""
    return np.random.default_rng([count, least, most, salt]).integers(least, most + 1, size=count).astype(np.int32)


class _Source:
    """Seeded values on the GPU."""

    def __init__(self, seed):
        self.generator = torch.Generator(device="cuda").manual_seed(int(seed))

    def normal(self, *shape, kind=torch.bfloat16, scale=1.0):
        return torch.randn(shape, generator=self.generator, device="cuda").mul_(scale).to(kind)

    def permutation(self, count):
        return torch.randperm(count, generator=self.generator, device="cuda")

    def integers(self, high, count):
        return torch.randint(0, high, (count,), generator=self.generator, device="cuda").tolist()


def _int32(values):
    return torch.tensor(np.asarray(values), dtype=torch.int32, device="cuda")


def _int64(values):
    return torch.tensor(np.asarray(values), dtype=torch.int64, device="cuda")


def _starts(lengths):
    return np.concatenate([[0], np.cumsum(lengths)]).astype(np.int64)


def _attend(query, key, value, scale, visible, gate=None):
    """One sequence in 64 bits: query [L, H, D], key and value [S, G, D]; ``visible`` maps (positions of the queries,
    positions of the keys) to what is seen, queries being the sequence's last.  Outputs [L, H, V], natural log sums [L, H]."""
    length, heads, keys, groups = query.shape[0], query.shape[1], key.shape[0], key.shape[1]
    per = heads // groups
    out = torch.empty((length, heads, value.shape[2]), dtype=torch.float64, device=query.device)
    lse = torch.empty((length, heads), dtype=torch.float64, device=query.device)
    at = torch.arange(keys, device=query.device)
    rows = max(1, (1 << 27) // (keys * per))
    for first in range(0, length, rows):
        part = slice(first, min(first + rows, length))
        hidden = ~visible(at[keys - length:][part][:, None], at[None, :])
        for group in range(groups):
            own = slice(group * per, (group + 1) * per)
            scores = torch.einsum("lhd,sd->hls", query[part, own].double(), key[:, group].double()) * scale
            scores.masked_fill_(hidden, -math.inf)
            lse[part, own] = torch.logsumexp(scores, 2).T
            out[part, own] = torch.einsum("hls,sv->lhv", torch.softmax(scores, 2), value[:, group].double())
    return out, lse


def _causal(query, key):
    return key <= query


def _seen(new, keys, window=0):
    """How many (query, key) pairs ``new`` causal queries at the end of ``keys`` keys make."""
    position = np.arange(keys - new, keys, dtype=np.int64)
    return int(np.minimum(position + 1, window if window else keys).sum())


# ------------------------------------------------------------------------------------------------
# linear
# ------------------------------------------------------------------------------------------------

class Linear:
    @staticmethod
    def prepare(case, seed):
        source = _Source(seed)
        return {"x": source.normal(case["m"], case["k"]), "weight": source.normal(case["n"], case["k"], scale=0.02)}

    @staticmethod
    def run(state):
        return ops.linear(state["x"], state["weight"])

    @staticmethod
    def exact(case, seed):
        state = Linear.prepare(case, seed)
        return state["x"].double() @ state["weight"].double().T

    @staticmethod
    def work(case):
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 2 * (m * k + n * k + m * n), "flops": 2 * m * n * k}

    @staticmethod
    def tolerance(case):
        return {"rel": 7e-3, "max": 0.02}     # the rounding of the result to bf16 is 1.7e-3


# ------------------------------------------------------------------------------------------------
# attention
# ------------------------------------------------------------------------------------------------

class _Paged:
    """Sequences in a cache of 16-token pages that lie in random order, a tenth of them free."""

    def __init__(self, source, lengths, dim, kind):
        self.counts = (lengths.astype(np.int64) + PAGE - 1) // PAGE
        pool = int(math.ceil(self.counts.sum() * 1.1))
        self.order = source.permutation(pool).cpu().numpy()
        self.starts = _starts(self.counts)
        self.keys = source.normal(pool, PAGE, KV_HEADS, dim, kind=kind)
        self.values = source.normal(pool, PAGE, KV_HEADS, dim, kind=kind)

    def of(self, sequence):
        return self.order[self.starts[sequence]: self.starts[sequence + 1]]

    def rows(self, sequence, length):
        """Keys and values of one sequence, [length, kv heads, dim]."""
        pages = _int64(self.of(sequence))
        return [cache[pages].flatten(0, 1)[:length] for cache in (self.keys, self.values)]

    def table(self):
        out = np.zeros((len(self.counts), int(self.counts.max())), dtype=np.int32)
        for sequence, count in enumerate(self.counts):
            out[sequence, :count] = self.of(sequence)
        return out


class PagedDecode:
    @staticmethod
    def _lengths(case):
        return _lengths(case["batch"], case["least"], case["most"], 1)

    @staticmethod
    def _inputs(case, seed):
        source, kind = _Source(seed), TYPES[case["type"]]
        paged = _Paged(source, PagedDecode._lengths(case), case["dim"], kind)
        return paged, source.normal(case["batch"], HEADS, case["dim"], kind=kind)

    @staticmethod
    def prepare(case, seed):
        lengths = PagedDecode._lengths(case)
        paged, query = PagedDecode._inputs(case, seed)
        # the table is as wide as the longest context a sequence may reach
        stride = -(-max(case["most"], int(lengths.max())) // PAGE)
        table = np.zeros((case["batch"], stride), dtype=np.int32)
        table[:, : paged.counts.max()] = paged.table()
        config = ops.PagedKvDecodeAttentionConfig.contiguous(case["batch"], HEADS, KV_HEADS, case["dim"], PAGE, paged.keys.shape[0],
                                                             stride, case["dim"] ** -0.5)
        return {"out": torch.empty_like(query), "query": query, "keys": paged.keys, "values": paged.values,
                "lengths": _int32(lengths), "table": _int32(table), "config": config}

    @staticmethod
    def run(s):
        ops.paged_kv_decode_attention(s["out"], s["query"], s["keys"], s["values"], s["lengths"], s["table"], s["config"])
        return s["out"]

    @staticmethod
    def exact(case, seed):
        paged, query = PagedDecode._inputs(case, seed)
        rows = [_attend(query[b: b + 1], *paged.rows(b, int(n)), case["dim"] ** -0.5, _causal)[0]
                for b, n in enumerate(PagedDecode._lengths(case))]
        return torch.cat(rows)

    @staticmethod
    def work(case):
        total, dim = int(PagedDecode._lengths(case).sum()), case["dim"]
        return {"bytes": 4 * (total * KV_HEADS * dim + case["batch"] * HEADS * dim) + total // 4, "flops": 4 * total * HEADS * dim}

    @staticmethod
    def tolerance(case):
        return {"rel": 1e-2, "max": 0.05}


class Prefill:
    @staticmethod
    def _lengths(case):
        if case["spread"] == "halves":
            return np.asarray([case["most"] >> i for i in range(case["prompts"])], dtype=np.int32)
        return _lengths(case["prompts"], case["least"], case["most"], 2)

    @staticmethod
    def _inputs(case, seed):
        source, dim, total = _Source(seed), case["dim"], int(Prefill._lengths(case).sum())
        q, k, v = (source.normal(total, heads, dim) for heads in (HEADS, KV_HEADS, KV_HEADS))
        return q, k, v, source.permutation(total // PAGE * 11 // 10 + case["prompts"])   # and the order of the cache's pages

    @staticmethod
    def _places(case, order):
        """Cache page and slot of every token."""
        lengths = Prefill._lengths(case)
        counts = -(-lengths.astype(np.int64) // PAGE)
        first = _starts(counts)
        inside = np.concatenate([np.arange(n) for n in lengths])
        page = np.concatenate([first[b] + np.arange(n) // PAGE for b, n in enumerate(lengths)])
        return order[_int64(page)], _int64(inside % PAGE)

    @staticmethod
    def prepare(case, seed):
        q, k, v, order = Prefill._inputs(case, seed)
        lengths, dim = Prefill._lengths(case), case["dim"]
        pages, slots = Prefill._places(case, order)
        total = q.shape[0]
        cache = lambda: torch.zeros((order.numel(), PAGE, KV_HEADS, dim), dtype=torch.bfloat16, device="cuda")
        config = ops.RaggedKvPrefillAttentionConfig(len(lengths), total, total, HEADS, KV_HEADS, dim, True, dim ** -0.5)
        return {"out": torch.empty_like(q), "lse": torch.empty((total, HEADS), device="cuda"), "q": q, "k": k, "v": v,
                "lengths": _int32(lengths), "offsets": _int32(_starts(lengths)[:-1]), "config": config, "keys": cache(),
                "values": cache(), "pages": pages, "slots": slots, "status": torch.zeros(1, dtype=torch.int32, device="cuda")}

    @staticmethod
    def run(s):
        ops.ragged_kv_prefill_attention(s["out"], s["lse"], s["q"], s["k"], s["v"], s["lengths"], s["lengths"], s["offsets"],
                                        s["config"], cache_write=(s["keys"], s["values"], s["pages"], s["slots"], s["status"]))
        return {"out": s["out"], "lse": s["lse"], "keys": s["keys"], "values": s["values"]}

    @staticmethod
    def exact(case, seed):
        q, k, v, order = Prefill._inputs(case, seed)
        out, lse, at = [], [], 0
        for n in Prefill._lengths(case):
            part = slice(at, at + int(n))
            o, l = _attend(q[part], k[part], v[part], case["dim"] ** -0.5, _causal)
            out.append(o)
            lse.append(l)
            at += int(n)
        caches = []
        for rows in (k, v):
            cache = torch.zeros((order.numel(), PAGE, KV_HEADS, case["dim"]), dtype=torch.float64, device="cuda")
            cache[Prefill._places(case, order)] = rows.double()
            caches.append(cache)
        return {"out": torch.cat(out), "lse": torch.cat(lse), "keys": caches[0], "values": caches[1]}

    @staticmethod
    def work(case):
        lengths, dim = Prefill._lengths(case), case["dim"]
        total = int(lengths.sum())
        return {"bytes": total * (2 * 2 * HEADS * dim + 4 * 2 * KV_HEADS * dim + 4 * HEADS),
                "flops": 4 * HEADS * dim * sum(_seen(int(n), int(n)) for n in lengths)}

    @staticmethod
    def tolerance(case):
        return {"rel": 1e-2, "max": 0.05}


class PagedAttention:
    DIM = 128

    @staticmethod
    def _lengths(case):
        """New tokens and all tokens of each sequence; the chunks of prompts come first."""
        new = np.asarray([case["chunk"] - (i % 3) for i in range(case["chunks"])] + [1] * case["decoding"], dtype=np.int32)
        return new, new + _lengths(len(new), 0, case["most"], 3)

    @staticmethod
    def _inputs(case, seed):
        source, kind = _Source(seed), TYPES[case["type"]]
        new, every = PagedAttention._lengths(case)
        paged = _Paged(source, every, PagedAttention.DIM, kind)
        return paged, source.normal(int(new.sum()), HEADS, PagedAttention.DIM, kind=kind)

    @staticmethod
    def prepare(case, seed):
        new, every = PagedAttention._lengths(case)
        paged, query = PagedAttention._inputs(case, seed)
        return {"query": query, "keys": paged.keys, "values": paged.values, "query_offsets": _int64(_starts(new)),
                "page_offsets": _int64(paged.starts), "pages": _int64(paged.order[: paged.starts[-1]]),
                "last": _int64((every - 1) % PAGE + 1), "window": case["window"],
                "status": torch.zeros(1, dtype=torch.int32, device="cuda")}

    @staticmethod
    def run(s):
        return ops.paged_attention(s["query"], s["keys"], s["values"], s["query_offsets"], s["page_offsets"], s["pages"], s["last"],
                                   window=s["window"], status=s["status"])

    @staticmethod
    def exact(case, seed):
        new, every = PagedAttention._lengths(case)
        paged, query = PagedAttention._inputs(case, seed)
        window, starts = case["window"] or 1 << 30, _starts(new)
        visible = lambda q, k: (k <= q) & (k > q - window)
        parts = [_attend(query[starts[b]: starts[b + 1]], *paged.rows(b, int(n)), PagedAttention.DIM ** -0.5, visible)
                 for b, n in enumerate(every)]
        return torch.cat([out for out, _ in parts]), torch.cat([lse for _, lse in parts]) / math.log(2.0)

    @staticmethod
    def work(case):
        new, every = PagedAttention._lengths(case)
        window, dim = case["window"], PagedAttention.DIM
        read = sum(min(int(n), int(t) + window - 1) if window else int(n) for t, n in zip(new, every))
        return {"bytes": 4 * read * KV_HEADS * dim + int(new.sum()) * HEADS * (4 * dim + 4),
                "flops": 4 * HEADS * dim * sum(_seen(int(t), int(n), window) for t, n in zip(new, every))}

    @staticmethod
    def tolerance(case):
        return {"rel": 1e-2, "max": 0.05}


class Sdpa:
    @staticmethod
    def prepare(case, seed):
        source = _Source(seed)
        shape = lambda heads: (case["batch"], heads, case["length"], case["dim"])
        q, k, v = (source.normal(*shape(heads), kind=torch.float32) for heads in (case["heads"], case["kv_heads"], case["kv_heads"]))
        return {"q": q, "k": k, "v": v, "causal": case["causal"]}

    @staticmethod
    def run(s):
        return ops.scaled_dot_product_attention(s["q"], s["k"], s["v"], causal=s["causal"])

    @staticmethod
    def exact(case, seed):
        s = Sdpa.prepare(case, seed)
        seen = _causal if case["causal"] else lambda q, k: (k >= 0) & (q >= 0)
        swap = lambda t: t.transpose(0, 1)
        return torch.stack([swap(_attend(swap(q), swap(k), swap(v), case["dim"] ** -0.5, seen)[0])
                            for q, k, v in zip(s["q"], s["k"], s["v"])])

    @staticmethod
    def work(case):
        heads, length, dim = case["batch"] * case["heads"], case["length"], case["dim"]
        pairs = _seen(length, length) if case["causal"] else length * length
        return {"bytes": 8 * length * dim * (heads + case["batch"] * case["kv_heads"]), "flops": 4 * heads * dim * pairs}

    @staticmethod
    def tolerance(case):
        return {"rel": 4e-6, "max": 4e-5}


# ------------------------------------------------------------------------------------------------
# decoders
# ------------------------------------------------------------------------------------------------

def _decoder_lengths(case):
    return _lengths(case["sequences"], case["least"], case["most"], 4)


def _capacity(case):
    """Room for the longest sequence and some new tokens."""
    return int(_decoder_lengths(case).max()) + 64


def _page_rows(lengths, page_size):
    """Cache row of every cached token of each sequence: pages are handed out in order."""
    first = _starts(-(-lengths.astype(np.int64) // page_size)) * page_size
    return [slice(int(first[b]), int(first[b]) + int(n)) for b, n in enumerate(lengths)]


def _prompts(case, source, vocab):
    return [source.integers(vocab, int(n)) for n in _decoder_lengths(case)]


def _rms(x, weight, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * weight


def _silu(x):
    return x * torch.sigmoid(x)


class _Decoder:
    """A prompt step reads every sequence's prompt from an empty cache; a decode step is one new token for every sequence behind
    its context, replayed from the captured graph."""

    @classmethod
    def prepare(cls, case, seed):
        source = _Source(seed)
        weights = cls.weights(source)
        lengths = _decoder_lengths(case)
        decoder = cls.build(case["sequences"], _capacity(case), weights)
        if case["step"] == "prompt":
            return {"decoder": decoder, "prompts": _prompts(case, source, cls.VOCAB), "parts": cls.caches(decoder)}
        decoder.table.place_prompts([int(n) for n in lengths])
        for part in cls.caches(decoder):
            part.copy_(source.normal(*part.shape, kind=part.dtype))
        decoder.capture()
        decoder.plan(source.integers(cls.VOCAB, case["sequences"]))
        return {"decoder": decoder, "prompts": None, "parts": cls.caches(decoder)}

    @staticmethod
    def run(s):
        decoder = s["decoder"]
        if s["prompts"] is None:
            decoder.run()
            return {"logits": decoder.logits, "caches": s["parts"]}
        decoder.reset()
        return {"logits": decoder.step_tokens(s["prompts"]), "caches": s["parts"]}

    @classmethod
    def exact(cls, case, seed):
        source = _Source(seed)
        weights = {name: value.double() for name, value in cls.weights(source).items()}
        lengths = _decoder_lengths(case)
        if case["step"] == "prompt":
            tokens, past = _prompts(case, source, cls.VOCAB), [None] * len(lengths)
        else:
            parts = [source.normal(*shape, kind=kind).double() for shape, kind in cls.cache_shapes(case)]
            tokens = [[t] for t in source.integers(cls.VOCAB, case["sequences"])]
            past = cls.pasts(parts, lengths)
        logits = [cls.forward(weights, torch.tensor(t, device="cuda"), p) for t, p in zip(tokens, past)]
        return {"logits": torch.stack(logits), "caches": [None] * len(cls.cache_shapes(case))}

    @classmethod
    def work(cls, case):
        lengths = _decoder_lengths(case).astype(np.int64)
        decode = case["step"] == "decode"
        rows = case["sequences"] if decode else int(lengths.sum())
        per_token = sum(math.prod(shape) for name, shape in cls.shapes().items()
                        if len(shape) == 2 and name not in ("embed", "head") and not name.endswith(".conv") and ".hc" not in name)
        head = cls.VOCAB * cls.WIDTH
        flops = 2 * rows * per_token + 2 * case["sequences"] * head
        moved = 2 * (per_token + head) + 8 * rows * cls.WIDTH
        more_bytes, more_flops = cls.mixing(lengths, decode)
        return {"bytes": moved + more_bytes, "flops": flops + more_flops}

    @classmethod
    def tolerance(cls, case):
        return cls.TOLERANCE


class Llama(_Decoder):
    CONFIG = llama.LlamaConfig(layers=6)
    VOCAB, WIDTH = CONFIG.vocab, CONFIG.hidden
    TOLERANCE = {"rel": 0.1, "max": 0.6}     # logits after six layers with the residual stream and activations in bf16

    @classmethod
    def shapes(cls):
        c = cls.CONFIG
        queries, keys = c.heads * c.head_dim, c.kv_heads * c.head_dim
        shapes = {"embed": (c.vocab, c.hidden), "head": (c.vocab, c.hidden), "final_norm": (c.hidden,)}
        for i in range(c.layers):
            shapes.update({f"{i}.wq": (queries, c.hidden), f"{i}.wk": (keys, c.hidden), f"{i}.wv": (keys, c.hidden),
                           f"{i}.wo": (c.hidden, queries), f"{i}.gate": (c.ffn, c.hidden), f"{i}.up": (c.ffn, c.hidden),
                           f"{i}.down": (c.hidden, c.ffn), f"{i}.attn_norm": (c.hidden,), f"{i}.mlp_norm": (c.hidden,)})
        return shapes

    @classmethod
    def weights(cls, source):
        return {name: source.normal(*shape, scale=0.02) if len(shape) == 2 else 1.0 + source.normal(*shape, scale=0.1)
                for name, shape in cls.shapes().items()}

    @classmethod
    def build(cls, sequences, capacity, weights):
        names = ("wq", "wk", "wv", "wo", "gate", "up", "down", "attn_norm", "mlp_norm")
        layers = [{name: weights[f"{i}.{name}"] for name in names} for i in range(cls.CONFIG.layers)]
        return llama.LlamaDecoder(cls.CONFIG, sequences, capacity, weights={
            "layers": layers, "embed": weights["embed"], "lm_head": weights["head"], "final_norm": weights["final_norm"]})

    @staticmethod
    def caches(decoder):
        return [part for pair in zip(decoder.key_caches, decoder.value_caches) for part in pair]

    @classmethod
    def cache_shapes(cls, case):
        c = cls.CONFIG
        pages = case["sequences"] * -(-_capacity(case) // c.page_size) + 1
        return [((pages, c.page_size, c.kv_heads, c.head_dim), torch.bfloat16)] * (2 * c.layers)

    @classmethod
    def pasts(cls, parts, lengths):
        flat = [part.flatten(0, 1) for part in parts]
        return [[(flat[2 * i][rows], flat[2 * i + 1][rows]) for i in range(cls.CONFIG.layers)]
                for rows in _page_rows(lengths, cls.CONFIG.page_size)]

    @classmethod
    def forward(cls, w, tokens, past):
        """Logits of the last token in 64 bits."""
        c = cls.CONFIG
        x = w["embed"][tokens]
        earlier = 0 if past is None else past[0][0].shape[0]
        # cosines and sines are rounded to the model's type in f32, as the reference has them
        inverse = np.float32(1.0) / np.power(np.float32(c.theta), np.arange(0, c.head_dim, 2).astype(np.float32) / np.float32(c.head_dim))
        angle = np.arange(earlier, earlier + len(tokens), dtype=np.float32)[:, None] * inverse.astype(np.float32)[None]
        cosine, sine = (torch.from_numpy(f(angle)).cuda().bfloat16().double()[:, None] for f in (np.cos, np.sin))

        def turn(t):
            low, high = t.chunk(2, -1)
            return torch.cat([low * cosine - high * sine, high * cosine + low * sine], -1)

        for i in range(c.layers):
            h = _rms(x, w[f"{i}.attn_norm"], c.eps)
            q, k, v = ((h @ w[f"{i}.{name}"].T).unflatten(1, (-1, c.head_dim)) for name in ("wq", "wk", "wv"))
            q, k = turn(q), turn(k)
            if past is not None:
                k, v = torch.cat([past[i][0], k]), torch.cat([past[i][1], v])
            attended, _ = _attend(q, k, v, c.head_dim ** -0.5, _causal)
            x = x + attended.flatten(1) @ w[f"{i}.wo"].T
            h = _rms(x, w[f"{i}.mlp_norm"], c.eps)
            x = x + (_silu(h @ w[f"{i}.gate"].T) * (h @ w[f"{i}.up"].T)) @ w[f"{i}.down"].T
        return w["head"] @ _rms(x[-1], w["final_norm"], c.eps)

    @classmethod
    def mixing(cls, lengths, decode):
        c = cls.CONFIG
        token = 4 * c.kv_heads * c.head_dim
        new = [1 if decode else int(n) for n in lengths]
        every = [int(n) + 1 if decode else int(n) for n in lengths]
        return c.layers * token * sum(every), c.layers * 4 * c.heads * c.head_dim * sum(_seen(t, n) for t, n in zip(new, every))


class _LayerList(_Decoder):
    TOLERANCE = {"rel": 0.03, "max": 0.2}    # the residual stream is f32, activations are bf16

    @classmethod
    def weights(cls, source):
        constants = {"a2.b": 2.0, "A_log": -3.0, "dt_bias": 0.0}
        out = {}
        for name, shape in cls.shapes().items():
            if len(shape) == 1:
                base = next((value for ending, value in constants.items() if name.endswith(ending)), 1.0)
                if name.endswith((".in", ".out")) and ".hc" in name:
                    base = 1.0 / shape[0]
                if name.endswith(("q.b", "k.b", "v.b")):
                    base = 0.0
                out[name] = base + source.normal(*shape, scale=0.05)
            else:
                values = source.normal(*shape, kind=torch.float32, scale=1.0 if name == "embed" else shape[1] ** -0.5)
                if ".hc" in name:
                    values = 0.1 * values + torch.eye(shape[0], device="cuda")
                out[name] = values.bfloat16()
        return out

    @classmethod
    def build(cls, sequences, capacity, weights):
        return hybrid.HybridDecoder(cls.CONFIG, sequences, capacity, weights)

    @staticmethod
    def caches(decoder):
        return [part for cache in decoder.caches for part in (cache if isinstance(cache, tuple) else (cache,))]


class Kavalorn(_LayerList):
    """Latent attention with a window and gated linear attention, one residual stream."""

    ATTENTION = hybrid.LatentAttentionConfig(heads=16, dim=128, vdim=128, q_rank=768, kv_rank=256, scale=128 ** -0.5, window=1024)
    RECURRENT = hybrid.GatedLinearConfig(heads=16, dim=64, vdim=128, rank=16, tau=16.0)
    PATTERN, FFN, VOCAB, WIDTH = "aagaag", 8192, 32000, 2048
    CONFIG = hybrid.HybridConfig(layers=list(map({"a": hybrid.LayerConfig(ATTENTION, FFN), "g": hybrid.LayerConfig(RECURRENT, FFN)}.get,
                                                 PATTERN)), width=WIDTH, vocab=VOCAB)

    @classmethod
    def shapes(cls):
        w, a, r = cls.WIDTH, cls.ATTENTION, cls.RECURRENT
        shapes = {"embed": (cls.VOCAB, w), "embed.norm": (w,), "final.norm": (w,), "head": (cls.VOCAB, w)}
        for i, kind in enumerate(cls.PATTERN):
            if kind == "a":
                mix = {"dq": (a.q_rank, w), "dq.norm": (a.q_rank,), "uq": (a.heads * a.dim, a.q_rank), "dkv": (a.kv_rank, w),
                       "dkv.norm": (a.kv_rank,), "uk": (a.heads * a.dim, a.kv_rank), "uv": (a.heads * a.vdim, a.kv_rank),
                       "g": (a.heads, w), "o": (w, a.heads * a.vdim)}
            else:
                keys, values = r.heads * r.dim, r.heads * r.vdim
                mix = {"q": (keys, w), "k": (keys, w), "v": (values, w), "g": (values, w), "o": (w, values), "norm": (r.vdim,),
                       "a1": (r.rank, w), "a2": (keys, r.rank), "a2.b": (keys,)}
            shapes.update({f"l{i}.mix.{name}": shape for name, shape in mix.items()})
            shapes.update({f"l{i}.norm1": (w,), f"l{i}.norm2": (w,), f"l{i}.mlp.up": (cls.FFN, w), f"l{i}.mlp.down": (w, cls.FFN)})
        return shapes

    @classmethod
    def cache_shapes(cls, case):
        page, a, r = cls.CONFIG.page_size, cls.ATTENTION, cls.RECURRENT
        pages = case["sequences"] * -(-_capacity(case) // page) + 1
        return [((pages, page, 1, a.kv_rank), torch.bfloat16) if kind == "a"
                else ((case["sequences"], r.heads, r.dim, r.vdim), torch.float32) for kind in cls.PATTERN]

    @classmethod
    def pasts(cls, parts, lengths):
        return [[part.flatten(0, 1)[rows, 0] if kind == "a" else part[b] for kind, part in zip(cls.PATTERN, parts)]
                for b, rows in enumerate(_page_rows(lengths, cls.CONFIG.page_size))]

    @classmethod
    def forward(cls, w, tokens, past):
        eps, a, r = cls.CONFIG.eps, cls.ATTENTION, cls.RECURRENT

        def norm(x, weight):
            x = x - x.mean(-1, keepdim=True)
            return _rms(x, weight, eps)

        def latent_attention(h, m, earlier):
            latent = _rms(h @ m["dkv"].T, m["dkv.norm"], eps)
            if earlier is not None:
                latent = torch.cat([earlier, latent])
            q = (_rms(h @ m["dq"].T, m["dq.norm"], eps) @ m["uq"].T).unflatten(1, (a.heads, -1))
            k, v = ((latent @ m[name].T).unflatten(1, (a.heads, -1)) for name in ("uk", "uv"))
            out, _ = _attend(q, k, v, a.scale, lambda i, j: (j <= i) & (j > i - a.window))
            return (out * torch.sigmoid(h @ m["g"].T)[:, :, None]).flatten(1) @ m["o"].T

        def recurrence(h, m, earlier):
            q, k, v = ((h @ m[name].T).unflatten(1, (r.heads, -1)) for name in ("q", "k", "v"))
            decay = torch.sigmoid((h @ m["a1"].T) @ m["a2"].T + m["a2.b"]).pow(1.0 / r.tau).unflatten(1, (r.heads, -1))
            state = h.new_zeros(r.heads, r.dim, r.vdim) if earlier is None else earlier.clone()
            out = torch.empty_like(v)
            for t in range(len(h)):
                state.mul_(decay[t][:, :, None]).addcmul_(k[t][:, :, None], v[t][:, None])
                out[t] = torch.matmul(q[t][:, None], state)[:, 0]
            out = _rms(out * r.dim ** -0.5, m["norm"], eps).flatten(1)
            return (out * _silu(h @ m["g"].T)) @ m["o"].T

        x = norm(w["embed"][tokens], w["embed.norm"])
        for i, kind in enumerate(cls.PATTERN):
            m = {name[len(f"l{i}.mix."):]: value for name, value in w.items() if name.startswith(f"l{i}.mix.")}
            mixer = latent_attention if kind == "a" else recurrence
            x = x + mixer(norm(x, w[f"l{i}.norm1"]), m, None if past is None else past[i])
            x = x + torch.relu(norm(x, w[f"l{i}.norm2"]) @ w[f"l{i}.mlp.up"].T).square() @ w[f"l{i}.mlp.down"].T
        return w["head"] @ norm(x[-1], w["final.norm"])

    @classmethod
    def mixing(cls, lengths, decode):
        a, r = cls.ATTENTION, cls.RECURRENT
        latent, recurrent = cls.PATTERN.count("a"), cls.PATTERN.count("g")
        new = [1 if decode else int(n) for n in lengths]
        every = [int(n) + 1 if decode else int(n) for n in lengths]
        states = len(lengths) * r.heads * r.dim * r.vdim
        moved = latent * 2 * a.kv_rank * sum(min(n, a.window + t - 1) for t, n in zip(new, every)) + recurrent * (8 if decode else 4) * states
        pairs = sum(_seen(t, n, a.window) for t, n in zip(new, every))
        return moved, latent * 4 * a.heads * a.dim * pairs + recurrent * 4 * r.heads * r.dim * r.vdim * sum(new)


class Vatolorn(_LayerList):
    """Chunked attention and the gated delta rule side by side, four residual streams."""

    ROTATION = Rotation(128, 10000.0, YarnScaling(8.0, 4096.0, 32.0, 1.0))
    LEFT = ChunkedAttentionConfig(heads=16, kv_heads=4, dim=128, vdim=128, scale=128 ** -0.5, chunk=4096, taps=4, rotation=ROTATION)
    RIGHT = GatedDeltaConfig(heads=16, kv_heads=16, dim=64, vdim=128, taps=4, rank=64, gate_rank=64)
    LAYERS, STREAMS, FFN, VOCAB, WIDTH, LOGIT_SCALE = 6, 4, 8192, 32000, 2048, 0.5
    CONFIG = hybrid.HybridConfig(layers=[hybrid.LayerConfig(ParallelConfig(LEFT, RIGHT), FFN, None, True)] * LAYERS, width=WIDTH,
                                 vocab=VOCAB, page_size=PAGE, streams=STREAMS, logit_scale=LOGIT_SCALE)
    PROJECTIONS = {"left": {"q": LEFT.heads * LEFT.dim, "k": LEFT.kv_heads * LEFT.dim, "v": LEFT.kv_heads * LEFT.vdim},
                   "right": {"q": RIGHT.kv_heads * RIGHT.dim, "k": RIGHT.kv_heads * RIGHT.dim, "v": RIGHT.heads * RIGHT.vdim}}

    @classmethod
    def shapes(cls):
        w, a, r, s = cls.WIDTH, cls.LEFT, cls.RIGHT, cls.STREAMS
        shapes = {"embed": (cls.VOCAB, w), "final.norm": (w,), "head": (cls.VOCAB, w)}
        keys, values = r.heads * r.dim, r.heads * r.vdim
        mix = {"left.out": (w,), "right.out": (w,), "left.o": (w, a.heads * a.vdim), "right.o": (w, values),
               "left.q.norm": (a.heads * a.dim,), "left.k.norm": (a.kv_heads * a.dim,), "right.norm": (r.vdim,), "right.b": (r.heads, w),
               "right.A_log": (r.heads,), "right.dt_bias": (keys,), "right.a1": (r.rank, w), "right.a2": (keys, r.rank),
               "right.g1": (r.gate_rank, w), "right.g2": (values, r.gate_rank)}
        for side, taps in (("left", a.taps), ("right", r.taps)):
            for name, rows in cls.PROJECTIONS[side].items():
                mix.update({f"{side}.{name}": (rows, w), f"{side}.{name}.conv": (rows, taps)})
                if side == "left":
                    mix[f"left.{name}.b"] = (rows,)
        for i in range(cls.LAYERS):
            shapes.update({f"l{i}.mix.{name}": shape for name, shape in mix.items()})
            shapes.update({f"l{i}.norm1": (w,), f"l{i}.norm2": (w,), f"l{i}.mlp.gate": (cls.FFN, w), f"l{i}.mlp.up": (cls.FFN, w),
                           f"l{i}.mlp.down": (w, cls.FFN)})
            for n in (1, 2):
                shapes.update({f"l{i}.hc{n}.in": (s,), f"l{i}.hc{n}.out": (s,), f"l{i}.hc{n}.mix": (s, s)})
        return shapes

    @classmethod
    def cache_shapes(cls, case):
        a, r, n = cls.LEFT, cls.RIGHT, case["sequences"]
        pages = (n * -(-_capacity(case) // PAGE) + 1, PAGE, a.kv_heads, a.dim)
        rows = {side: (n, 3, sum(widths.values())) for side, widths in cls.PROJECTIONS.items()}
        half = torch.bfloat16
        return [(pages, half), (pages, half), (rows["left"], half), ((n, r.heads, r.dim, r.vdim), torch.float32),
                (rows["right"], half)] * cls.LAYERS

    @classmethod
    def pasts(cls, parts, lengths):
        out = []
        for b, rows in enumerate(_page_rows(lengths, PAGE)):
            layers = [parts[5 * i: 5 * i + 5] for i in range(cls.LAYERS)]
            out.append([(k.flatten(0, 1)[rows], v.flatten(0, 1)[rows], left[b], state[b], right[b])
                        for k, v, left, state, right in layers])
        return out

    @classmethod
    def forward(cls, w, tokens, past):
        eps, a, r = cls.CONFIG.eps, cls.LEFT, cls.RIGHT
        earlier = 0 if past is None else past[0][0].shape[0]
        positions = torch.arange(earlier, earlier + len(tokens), dtype=torch.float64, device="cuda")
        index = np.arange(64, dtype=np.float64)
        scaling = cls.ROTATION.scaling
        plain = cls.ROTATION.base ** (-2.0 * index / 128)
        pair = lambda turns: 128 * math.log(scaling.original / (2 * math.pi * turns)) / (2 * math.log(cls.ROTATION.base))
        low, high = max(math.floor(pair(scaling.fast)), 0), min(math.ceil(pair(scaling.slow)), 127)
        ramp = np.clip((index - low) / max(high - low, 0.001), 0.0, 1.0)
        frequency = torch.from_numpy(plain / scaling.factor * ramp + plain * (1 - ramp)).cuda()
        size = 0.1 * math.log(scaling.factor) + 1.0
        cosine, sine = ((f(positions[:, None] * frequency) * size)[:, None] for f in (torch.cos, torch.sin))

        def turn(t):
            even, odd = t[..., 0::2], t[..., 1::2]
            return torch.stack([even * cosine - odd * sine, odd * cosine + even * sine], -1).flatten(-2)

        def convolve(h, m, side, name, last):
            rows = h @ m[f"{side}.{name}"].T
            widths = cls.PROJECTIONS[side]
            at = sum(widths[other] for other in "qkv"[: "qkv".index(name)])
            before = rows.new_zeros(3, rows.shape[1])
            bias = m.get(f"{side}.{name}.b")
            if bias is not None:
                rows = rows + bias
            if last is not None:
                before = last[:, at: at + widths[name]]
                before = before if bias is None else before + bias
            rows, taps = torch.cat([before, rows]), m[f"{side}.{name}.conv"]
            return sum(taps[:, j] * rows[j: j + len(h)] for j in range(4))

        def attention(h, m, now):
            q, k, v = (convolve(h, m, "left", name, None if now is None else now[2]) for name in "qkv")
            q = turn(_rms(q, m["left.q.norm"], eps).unflatten(1, (a.heads, -1)))
            k = turn(_rms(k, m["left.k.norm"], eps).unflatten(1, (a.kv_heads, -1)))
            v = v.unflatten(1, (a.kv_heads, -1))
            if now is not None:
                k, v = torch.cat([now[0], k]), torch.cat([now[1], v])
            seen = lambda i, j: (j <= i) & (j >= i // a.chunk * a.chunk)
            return _attend(q, k, v, a.scale, seen)[0].flatten(1) @ m["left.o"].T

        def delta(h, m, now):
            q, k, v = (_silu(convolve(h, m, "right", name, None if now is None else now[4])) for name in "qkv")
            unit = lambda t: t * torch.rsqrt(t.square().sum(-1, keepdim=True) + 1e-6)
            q, k = (unit(t.unflatten(1, (r.kv_heads, -1))) for t in (q, k))
            v = v.unflatten(1, (r.heads, -1))
            step = torch.nn.functional.softplus((h @ m["right.a1"].T) @ m["right.a2"].T + m["right.dt_bias"]).unflatten(1, (r.heads, -1))
            decay = torch.exp(-m["right.A_log"].exp()[:, None] * step)
            strength = torch.sigmoid(h @ m["right.b"].T)
            state = h.new_zeros(r.heads, r.dim, r.vdim) if now is None else now[3].clone()
            out = torch.empty_like(v)
            for t in range(len(h)):
                state.mul_(decay[t][:, :, None])
                written = strength[t][:, None] * (v[t] - torch.matmul(k[t][:, None], state)[:, 0])
                state.addcmul_(k[t][:, :, None], written[:, None])
                out[t] = torch.matmul(q[t][:, None], state)[:, 0]
            out = _rms(out * r.dim ** -0.5, m["right.norm"], eps).flatten(1)
            return (out * torch.sigmoid((h @ m["right.g1"].T) @ m["right.g2"].T)) @ m["right.o"].T

        streams = torch.stack([w["embed"][tokens]] * cls.STREAMS)
        for i in range(cls.LAYERS):
            m = {name[len(f"l{i}.mix."):]: value for name, value in w.items() if name.startswith(f"l{i}.mix.")}
            now = None if past is None else past[i]
            for n in (1, 2):
                h = _rms(torch.einsum("s,stw->tw", w[f"l{i}.hc{n}.in"], streams), w[f"l{i}.norm{n}"], eps)
                if n == 1:
                    y = 0.5 * (_rms(attention(h, m, now), m["left.out"], eps) + _rms(delta(h, m, now), m["right.out"], eps))
                else:
                    y = (_silu(h @ w[f"l{i}.mlp.gate"].T) * (h @ w[f"l{i}.mlp.up"].T)) @ w[f"l{i}.mlp.down"].T
                streams = torch.einsum("sn,stw->ntw", w[f"l{i}.hc{n}.mix"], streams) + w[f"l{i}.hc{n}.out"][:, None, None] * y
        return w["head"] @ _rms(streams.sum(0)[-1], w["final.norm"], eps) * cls.LOGIT_SCALE

    @classmethod
    def mixing(cls, lengths, decode):
        a, r = cls.LEFT, cls.RIGHT
        cached = sum((int(n) % a.chunk) + 1 if decode else int(n) for n in lengths)
        pairs = cached if decode else sum(_seen(min(a.chunk, int(n) - at), min(a.chunk, int(n) - at))
                                          for n in lengths for at in range(0, int(n), a.chunk))
        rows = len(lengths) if decode else int(lengths.sum())
        state = r.heads * r.dim * r.vdim
        moved = cached * 4 * a.kv_heads * a.dim + len(lengths) * state * (8 if decode else 4) + 8 * rows * (cls.STREAMS - 1) * cls.WIDTH
        return cls.LAYERS * moved, cls.LAYERS * (4 * a.heads * a.dim * pairs + 6 * state * rows)


# ------------------------------------------------------------------------------------------------

KINDS = {"linear": Linear, "paged_decode": PagedDecode, "prefill": Prefill, "paged_attention": PagedAttention, "sdpa": Sdpa,
         "llama": Llama, "kavalorn": Kavalorn, "vatolorn": Vatolorn}


def prepare(case, seed):
    return KINDS[case["kind"]], KINDS[case["kind"]].prepare(case, seed)


def run(state):
    kind, held = state
    return kind.run(held)


def exact(case, seed):
    return KINDS[case["kind"]].exact(case, seed)


def work(case):
    return KINDS[case["kind"]].work(case)


def tolerance(case):
    return KINDS[case["kind"]].tolerance(case)
