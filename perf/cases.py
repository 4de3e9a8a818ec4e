"""Work that users of this package have it do, as cases that can be timed and checked.

A case is a dict of plain values.  ``listed()`` gives the cases, ``draw(rng)`` one more of the same ranges, ``prepare`` what a
user's program holds before the call (model, pool, prompts, device buffers), ``run`` one pass through the public entry points,
``work`` what the pass cannot do without, ``tolerance`` how far a correct implementation may be off, ``exact`` the outputs in
64-bit torch arithmetic.

Kinds of case
  decode   steps of the GPT model (the 35M configuration) for sequences of ragged lengths.  A pass takes the sequences back to
           their first length and replays given tokens (what a caller of the reference's forwardDecode does); the last step
           returns the logits.  ``pick``: ids by argmax, or drawn on the device with temperature and top-k
  prefill  prompts of ragged lengths through the same model, filling the paged cache; last logits and first ids
  attend   append + attention of one decode step on device buffers, for hosts that run their own projections: one call for
           all layers, or one per layer as a model with dependent layers issues them
  store    tokens of one layer appended to the paged cache and read back as the contiguous planes of getK / getV
  matmul   the projection primitive on device buffers
  layered  a model described layer by layer (the Lipelix design: attention with sinks, windowed attention, generalised delta
           rule): a batch of prompts in one step, then decode steps, the last one with logits
"""
from __future__ import annotations

import collections
import math

import numpy as np
import torch

from jgpt_b200 import decoder as D
from jgpt_b200 import registry
from jgpt_b200.kv_cache import KvPool
from jgpt_b200.model import GPTModel
from jgpt_b200.runtime import Context

# the 35M configuration: 24 heads of 16
VOCAB, POSITIONS, WIDTH, HEADS, LAYERS, FF, EPS = 8000, 1024, 384, 24, 12, 768, 1e-5
DHEAD = WIDTH // HEADS
PREFILL_ROWS = 32 * 1024
STATES = 4  # sets of sequences that a server's pool has room for
LAYERED_VOCAB, LAYERED_RANK = 32000, 64


# ---- the cases ------------------------------------------------------------------------------------------
def listed():
    return [
        # interactive chat: one row, the logits go to the host's sampler
        {"name": "chat", "kind": "decode", "rows": 1, "context": 150, "steps": 1, "pick": "argmax"},
        # a few chats served together, ids drawn on the device
        {"name": "decode-8-sampled", "kind": "decode", "rows": 8, "context": 400, "steps": 16, "pick": "sample"},
        # the batch size of the serving benchmark
        {"name": "decode-64", "kind": "decode", "rows": 64, "context": 512, "steps": 16, "pick": "argmax"},
        # a full server near the end of the context
        {"name": "decode-250", "kind": "decode", "rows": 250, "context": 1000, "steps": 8, "pick": "argmax"},
        # the prompt of one chat
        {"name": "prompt", "kind": "prefill", "rows": 1, "context": 201},
        # a full batch of prompts: 32 x 1024
        {"name": "prompts-32x1024", "kind": "prefill", "rows": 32, "context": 1024},
        # the headline benchmark: 64 sequences of 1024, 12 layers in one call
        {"name": "attend-64x1024", "kind": "attend", "rows": 64, "shortest": 1024, "longest": 1024, "layers_per_call": 12},
        # long contexts of mixed lengths, a call per layer
        {"name": "attend-long", "kind": "attend", "rows": 48, "shortest": 1024, "longest": 8192, "layers_per_call": 1},
        # a host that fills the cache itself and inspects it
        {"name": "store-24", "kind": "store", "rows": 24, "longest": 1000},
        # the projections of a host's own forward pass
        {"name": "matmul", "kind": "matmul", "m": 3000, "k": 384, "n": 768},
        # serving a layered model: prompts, then tokens
        {"name": "layered-serve", "kind": "layered", "width": 1024, "rows": 16, "context": 200, "steps": 24},
        # a large batch of prompts through a wider one
        {"name": "layered-8x1024", "kind": "layered", "width": 2048, "rows": 8, "context": 1024, "steps": 1},
    ]


def _between(rng, low, high):
    """A whole number, spread over the logarithm."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "prefill", "prefill", "attend", "store", "matmul", "layered"])
    if kind == "decode":
        rows = _between(rng, 1, 250)
        return {"kind": kind, "rows": rows, "context": _between(rng, 24, 1000), "steps": 1 if rows == 1 else rng.randint(4, 16) if rows <= 100 else 8,
                "pick": rng.choice(["argmax", "argmax", "sample"])}
    if kind == "prefill":
        rows = _between(rng, 1, 32)
        return {"kind": kind, "rows": rows, "context": _between(rng, 16, 1024)}
    if kind == "attend":
        shortest = _between(rng, 64, 4096)
        longest = min(8192, shortest + rng.choice([0, rng.randint(1, 4096)]))
        return {"kind": kind, "rows": _between(rng, 1, 64 if longest <= 1024 else 48), "shortest": shortest, "longest": longest,
                "layers_per_call": rng.choice([1, 12])}
    if kind == "store":
        return {"kind": kind, "rows": _between(rng, 1, 64), "longest": _between(rng, 20, 1024)}
    if kind == "matmul":
        return {"kind": kind, "m": _between(rng, 1, 32768), "k": 4 * _between(rng, 16, 512), "n": 4 * _between(rng, 16, 512)}
    rows = _between(rng, 1, 32)
    return {"kind": kind, "width": rng.choice([1024, 2048]), "rows": rows, "context": _between(rng, 16, 8192 // rows if rows > 8 else 1024),
            "steps": rng.randint(1, 24)}


# ---- inputs, from the seed alone ------------------------------------------------------------------------
def _lengths(case, seed):
    """Ragged lengths: the longest is the case's context, the others lie above half of it."""
    rng = np.random.default_rng([seed, 1])
    longest = case["context"]
    n = rng.integers(max(1, longest // 2), longest + 1, case["rows"])
    if case["kind"] == "prefill" and case["context"] == POSITIONS:
        n[:] = longest  # full prompts
    n[0] = longest
    return n.astype(np.int32)


def _tokens(case, seed, vocab):
    """Per row: prompt and the tokens of the steps behind it."""
    rng = np.random.default_rng([seed, 2])
    return [rng.integers(1, vocab, int(n) + case.get("steps", 0)).astype(np.int32) for n in _lengths(case, seed)]


def _draws(case, seed):
    return np.random.default_rng([seed, 3]).random((case["steps"], case["rows"]), np.float32)


def _normal(shape, *key):
    g = torch.Generator("cuda").manual_seed(int(np.random.default_rng(key).integers(1 << 62)))
    return torch.randn(shape, generator=g, device="cuda")


def _gpt_weights():
    """Matrices N(0, 0.02), norm weights near 1, in the order of getParameters()."""
    shapes = [(VOCAB, WIDTH), (POSITIONS, WIDTH)]
    for _ in range(LAYERS):
        shapes += [(WIDTH, WIDTH)] * 4 + [(WIDTH, FF), (FF, WIDTH), (WIDTH, FF), (WIDTH,), (WIDTH,)]
    shapes += [(WIDTH,), (WIDTH, VOCAB)]
    return [_normal(s, 0, i) * 0.02 if len(s) == 2 else 1 + 0.1 * _normal(s, 0, i) for i, s in enumerate(shapes)]


def _layered_config(width):
    h, mlp = width // 128, {"kind": "dense", "ff": width * 25 // 8}
    att = {"heads": h, "kv_heads": max(h // 4, 1), "dim": 128, "vdim": 128, "rot": {"base": 10000.0, "dims": 128}, "scale": 128 ** -0.5, "v_mix": True}
    block = [("attention", att), ("attention_2", {**att, "mask": {"size": 512, "keep_first": 16}}), ("general_delta", {"heads": h, "dim": 128})]
    return {"architecture": "Lipelix", "width": width, "vocab": LAYERED_VOCAB, "norm": {"eps": 1e-6}, "residual_mult": 0.5,
            "embedding": {"scale": 8.0}, "layers": [{"type": t, "mixer": m, "mlp": mlp} for t, m in block * 2]}


def _layered_shapes(cfg):
    width = cfg["width"]
    shapes = {"embed": (LAYERED_VOCAB, width), "head": (LAYERED_VOCAB, width), "final.norm": (width,)}
    for i, e in enumerate(cfg["layers"]):
        p, m, ff = f"l{i}.", e["mixer"], e["mlp"]["ff"]
        new = {n: (width,) for n in ("norm1", "norm1b", "norm2", "norm2b", "shift", "rg1.b", "rg2.b")}
        new.update({"rg1": (width, width), "rg2": (width, width), "mlp.up": (ff, width), "mlp.down": (width, ff)})
        H, d = m["heads"], m["dim"]
        if e["type"] == "general_delta":
            new.update({f"mix.{s}": (H * d, width) for s in "rkvga"})
            new.update({"mix.a.b": (H * d,), "mix.w0": (H * d,), "mix.norm": (H * d,), "mix.w1": (LAYERED_RANK, width),
                        "mix.w2": (H * d, LAYERED_RANK), "mix.o": (width, H * d)})
        else:
            G, v = m["kv_heads"], m["vdim"]
            new.update({"mix.q": (H * d, width), "mix.k": (G * d, width), "mix.v": (G * v, width), "mix.o": (width, H * v), "mix.vmix": (1,)})
            if e["type"] == "attention":
                new.update({"mix.q.norm": (H * d,), "mix.k.norm": (G * d,), "mix.sink": (H,)})
        shapes.update({p + n: s for n, s in new.items()})
    return shapes


def _layered_weight(name, shape, index):
    """Values that bf16 holds: matrices of unit gain, norm weights near 1, moderate biases, shares between 0 and 1."""
    x = _normal(shape, 0, index)
    if len(shape) == 2:
        x = x / math.sqrt(shape[1])
    elif name.endswith((".shift", ".vmix")):
        x = 0.3 + 0.1 * torch.tanh(x)
    elif name.endswith(".w0"):
        x = x - 4
    elif name.endswith((".a.b", ".rg1.b", ".rg2.b")):
        x = 0.1 * x
    else:
        x = 1 + 0.1 * x
    return x.bfloat16().float()


# ---- what a user's program holds ------------------------------------------------------------------------
class _Server:
    """A model with its pool, made once and kept while prompts come and go."""

    def __init__(self, case):
        self.ctx = Context(0)
        if case["kind"] == "layered":
            cfg = _layered_config(case["width"])
            shapes = _layered_shapes(cfg)
            where = {n: i for i, n in enumerate(shapes)}
            self.model = D.DecoderModel(self.ctx, registry.describe(cfg, shapes.__getitem__), "bfloat16", 8192)
            self.model.loadTensors(lambda n: _layered_weight(n, shapes[n], where[n]).cpu().numpy())
            rows, tokens = 32, 8192 + 32 * 40
        else:
            prompts = case["kind"] == "prefill"
            self.model = GPTModel(self.ctx, VOCAB, POSITIONS, WIDTH, HEADS, LAYERS, FF, rmsNormEps=EPS, maxRows=PREFILL_ROWS if prompts else 8192)
            self.model.setParameters([w.cpu().numpy() for w in _gpt_weights()])
            rows = 32 if prompts else 250
            tokens = rows * POSITIONS
        self.pool = self.model.newPool(STATES * (tokens // 16 + rows), STATES * rows, POSITIONS // 16 + 4)

    def close(self):
        self.pool.close(), self.model.close(), self.ctx.close()


_servers = collections.OrderedDict()


def _server(case):
    key = (case["kind"], case.get("width"))
    if key not in _servers:
        while len(_servers) >= 3:
            _servers.popitem(last=False)[1].close()
        _servers[key] = _Server(case)
    return _servers[key]


class _State:
    def __init__(self, case, seed):
        self.case, self.server, self.own, self.seqs = case, None, None, []
        getattr(self, "_" + case["kind"])(case, seed)
        torch.cuda.synchronize()

    def __del__(self):
        if self.server is not None and self.server.pool.handle:
            for s in self.seqs:
                self.server.pool.seq_free(s)
        if self.own is not None:
            self.own[0].close() if self.own[0] is not None else None
            self.own[1].close()

    def _sequences(self, case, seed, vocab):
        self.server = _server(case)
        self.lens, self.tokens = _lengths(case, seed), _tokens(case, seed, vocab)
        for _ in range(case["rows"]):
            self.seqs.append(self.server.pool.seq_alloc())
        self.ids = np.asarray(self.seqs, np.int32)
        self.prompts = [t[:n] for t, n in zip(self.tokens, self.lens)]

    def _forced(self, case):
        """Token and cache length of every row at every step."""
        self.steps = [(np.asarray([t[n + j] for t, n in zip(self.tokens, self.lens)], np.int32), self.lens + np.int32(j)) for j in range(case["steps"])]

    def _decode(self, case, seed):
        self._sequences(case, seed, VOCAB)
        self._forced(case)
        self.u = _draws(case, seed)
        model, pool, at = self.server.model, self.server.pool, 0
        while at < len(self.seqs):  # prompts in calls of at most the model's rows
            end, rows = at, 0
            while end < len(self.seqs) and rows + self.lens[end] <= model.maxRows:
                rows += int(self.lens[end])
                end += 1
            model.forwardPrefillBatch(pool, self.seqs[at:end], self.prompts[at:end])
            at = end
        for s, n in zip(self.seqs, self.lens):
            pool.reserve(s, min(int(n) + case["steps"], POSITIONS))

    def _prefill(self, case, seed):
        self._sequences(case, seed, VOCAB)

    def _layered(self, case, seed):
        self._sequences(case, seed, LAYERED_VOCAB)
        self._forced(case)
        self.ends = np.cumsum(self.lens).astype(np.int32) - 1

    def _attend(self, case, seed):
        ctx = Context(0)
        self.own = [None, ctx]
        lens = _attend_lengths(case, seed)
        n, longest = case["rows"], case["longest"]
        blocks = [-(-int(x) // 16) for x in lens]
        pool = self.own[0] = KvPool(ctx, LAYERS, HEADS, DHEAD, sum(blocks), n, -(-longest // 16), max_positions=longest)
        seqs = [pool.seq_alloc() for _ in range(n)]
        for s, x in zip(seqs, lens):
            pool.reserve(s, int(x))
        sid = torch.from_numpy(np.repeat(np.asarray(seqs, np.int32), lens)).cuda()
        pos = torch.from_numpy(np.concatenate([np.arange(x, dtype=np.int32) for x in lens])).cuda()
        for layer in range(LAYERS):
            k, v = _normal((pos.numel(), WIDTH), seed, 10, layer), _normal((pos.numel(), WIDTH), seed, 11, layer)
            torch.cuda.synchronize()
            pool.append(layer, k.data_ptr(), v.data_ptr(), sid.data_ptr(), pos.data_ptr(), pos.data_ptr(), pos.numel())
            torch.cuda.synchronize()
        self.q, self.k, self.v = (_normal((LAYERS, n, WIDTH), seed, 12 + i) for i in range(3))
        self.out = torch.empty_like(self.q)
        self.ids = torch.tensor(seqs, dtype=torch.int32, device="cuda")
        self.lens = torch.from_numpy(lens).cuda()
        self.pos = self.lens - 1
        self.ctx, self.pool = ctx, pool

    def _store(self, case, seed):
        ctx = Context(0)
        self.own = [None, ctx]
        n, longest = case["rows"], case["longest"]
        self.lens = lens = _store_lengths(case, seed)
        pool = self.own[0] = KvPool(ctx, 2, HEADS, DHEAD, n * -(-longest // 16), n, -(-longest // 16), max_positions=longest)
        self.seqs_ = [pool.seq_alloc() for _ in range(n)]
        for s, x in zip(self.seqs_, lens):
            pool.reserve(s, int(x))
            pool.set_length(s, int(x))
        self.ids = torch.from_numpy(np.repeat(np.asarray(self.seqs_, np.int32), lens)).cuda()
        self.pos = torch.from_numpy(np.concatenate([np.arange(x, dtype=np.int32) for x in lens])).cuda()
        self.k, self.v = (_normal((self.pos.numel(), WIDTH), seed, 20 + i) for i in range(2))
        self.planes = [torch.empty((n, HEADS, longest, DHEAD), device="cuda") for _ in range(2)]
        self.pool = pool

    def _matmul(self, case, seed):
        ctx = Context(0)
        self.own = [None, ctx]
        m, k, n = case["m"], case["k"], case["n"]
        self.a, self.b = ctx.alloc((m, k)), ctx.alloc((k, n))
        self.a.copy_from(_normal((m, k), seed, 30).cpu().numpy())
        self.b.copy_from((_normal((k, n), seed, 31) * 0.05).cpu().numpy())
        self.c, self.ctx = torch.empty((m, n), device="cuda"), ctx
        self.c_buffer = _Borrowed(self.c)


class _Borrowed:
    """A torch tensor where the package takes a device buffer."""

    def __init__(self, tensor):
        self.tensor, self.ptr = tensor, tensor.data_ptr()


def _attend_lengths(case, seed):
    n = np.random.default_rng([seed, 4]).integers(case["shortest"], case["longest"] + 1, case["rows"])
    n[0] = case["longest"]
    return n.astype(np.int32)


def _store_lengths(case, seed):
    n = np.random.default_rng([seed, 5]).integers(max(1, case["longest"] // 4), case["longest"] + 1, case["rows"])
    n[0] = case["longest"]
    return n.astype(np.int32)


def prepare(case, seed):
    return _State(case, seed)


# ---- one pass ---------------------------------------------------------------------------------------------
def run(state):
    return globals()["_run_" + state.case["kind"]](state, state.case)


def _run_decode(s, case):
    model, pool = s.server.model, s.server.pool
    for q, n in zip(s.seqs, s.lens):
        pool.set_length(q, n)
    picked = []
    for j, (tokens, lens) in enumerate(s.steps):
        if j + 1 == len(s.steps):
            logits, ids = model.forwardDecodeBatch(pool, s.ids, tokens, lens, lens)
        elif case["pick"] == "sample":
            ids = model.forwardDecodeSampleBatch(pool, s.ids, tokens, lens, lens, 0.8, 40, s.u[j])
        else:
            _, ids = model.forwardDecodeBatch(pool, s.ids, tokens, lens, lens, want_logits=False)
        picked.append(ids)
    return {"logits": logits, "ids": np.stack(picked)}


def _run_prefill(s, case):
    pool = s.server.pool
    for q in s.seqs:
        pool.clear(q, zero_fill=False)
    logits, ids = s.server.model.forwardPrefillBatch(pool, s.ids, s.prompts)
    return {"logits": logits, "ids": ids}


def _run_attend(s, case):
    n, per = case["rows"], case["layers_per_call"]
    slab = n * WIDTH * 4
    for layer in range(0, LAYERS, per):
        at = layer * slab
        s.pool.attn_decode_append(layer, per, s.q.data_ptr() + at, s.k.data_ptr() + at, s.v.data_ptr() + at, s.ids.data_ptr(), s.pos.data_ptr(),
                                  s.lens.data_ptr(), n, case["longest"], s.out.data_ptr() + at)
    return s.out


def _run_store(s, case):
    s.pool.append(1, s.k.data_ptr(), s.v.data_ptr(), s.ids.data_ptr(), s.pos.data_ptr(), s.pos.data_ptr(), s.pos.numel())
    s.pool.gather_batch(1, s.seqs_, s.lens, case["longest"], s.planes[0].data_ptr(), s.planes[1].data_ptr())
    return s.planes


def _run_matmul(s, case):
    s.ctx.matmul(s.a, s.b, s.c_buffer, case["m"], case["k"], case["n"])
    return s.c


def _run_layered(s, case):
    model, pool = s.server.model, s.server.pool
    for q in s.seqs:
        pool.clear(q, zero_fill=False)
    first, ids = model.step(pool, s.ids, s.prompts, s.ends, want_logits=True, want_next=True)
    picked = [ids]
    for j, (tokens, lens) in enumerate(s.steps):
        logits, ids = model.forwardDecodeBatch(pool, s.ids, tokens, lens, lens, want_logits=j + 1 == len(s.steps))
        picked.append(ids)
    return {"first": first, "logits": logits, "ids": np.stack(picked)}


# ---- what a pass cannot do without ------------------------------------------------------------------------
def work(case):
    kind, rows = case["kind"], case.get("rows", 0)
    if kind == "matmul":
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": 4 * (m * k + k * n + m * n), "flops": 2 * m * k * n}
    if kind == "store":  # rows of fp32 read, fp16 stored; fp16 read, planes of fp32 written
        tokens = rows * case["longest"] * 5 // 8
        return {"bytes": 2 * WIDTH * (tokens * (4 + 2 + 2) + rows * case["longest"] * 4), "flops": 0}
    if kind == "attend":
        tokens = rows * (case["shortest"] + case["longest"]) / 2
        return {"bytes": LAYERS * WIDTH * (tokens * 4 + rows * (4 * 4 + 4)), "flops": LAYERS * 4 * tokens * WIDTH}
    mean = case["context"] * (0.75 if rows > 1 else 1)
    if kind in ("decode", "prefill"):
        block = 4 * WIDTH * WIDTH + 3 * WIDTH * FF
        cached = LAYERS * 2 * WIDTH * 2  # bytes of a token
        if kind == "decode":
            steps = case["steps"]
            return {"bytes": steps * (4 * (LAYERS * block + WIDTH * VOCAB) + rows * mean * cached) + 4 * rows * VOCAB,
                    "flops": steps * rows * (2 * (LAYERS * block + WIDTH * VOCAB) + LAYERS * 4 * mean * WIDTH)}
        tokens = rows * (case["context"] if case["context"] == POSITIONS else mean)
        return {"bytes": 4 * (LAYERS * block + WIDTH * VOCAB) + tokens * cached + 4 * rows * VOCAB,
                "flops": 2 * tokens * LAYERS * block + LAYERS * 2 * tokens * mean * WIDTH + 2 * rows * WIDTH * VOCAB}
    w, steps = case["width"], case["steps"]
    layer = 2 * w * w * 25 // 8 + 2 * w * w  # feed-forward part and gates
    params = 6 * layer + 4 * (2 * w * w + 2 * w * max(w // 128 // 4, 1) * 128) + 2 * 6 * w * w
    tokens = rows * mean
    state = 2 * (w // 128) * 128 * 128 * 4 * 2
    cached = 4 * 2 * max(w // 128 // 4, 1) * 128 * 2
    return {"bytes": (1 + steps) * 2 * (params + w * LAYERED_VOCAB) + steps * rows * (mean * cached + state) + tokens * cached + 8 * rows * LAYERED_VOCAB,
            "flops": 2 * (tokens + steps * rows) * params + 2 * (1 + steps) * rows * w * LAYERED_VOCAB + 4 * 2 * tokens * mean * w}


def tolerance(case):
    kind = case["kind"]
    if kind == "store":
        return "exact"  # data movement, one rotation with stated roundings, one rounding to fp16
    if kind == "layered":  # bf16 operands: products by another kernel differ by 0.8 % of the logits, 0.038 at most
        return {"rel": 0.03, "max": 0.15, "differ": 0.01}
    if kind == "matmul":  # products with 22 bits of every operand against fp32 sums in order: 2.8e-6
        return {"rel": 1.2e-5}
    if kind == "attend":  # 32-bit sums over other pieces of the sequences: 2.2e-7, 1.2e-6 at most
        return {"rel": 4e-6}
    # 32-bit sums, and one more key, value or probability that rounds to the other fp16 neighbour: 9e-5, 6e-4 at most
    return {"rel": 4e-4, "differ": 0.01}


# ---- the same in 64 bits ------------------------------------------------------------------------------------
def exact(case, seed):
    return globals()["_exact_" + case["kind"]](case, seed)


def _rms(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _turn_pairs(x, positions):
    """x [..., tokens, heads, dhead]: elements (2 j, 2 j + 1) turn by position / 10000^(2 j / dhead)."""
    j = torch.arange(DHEAD // 2, device=x.device, dtype=torch.float64)
    t = positions.double()[:, None] / 10000.0 ** (2 * j / DHEAD)
    c, s = torch.cos(t)[:, None], torch.sin(t)[:, None]
    a, b = x[..., 0::2], x[..., 1::2]
    return torch.stack([a * c - b * s, a * s + b * c], -1).flatten(-2)


def _padded(tokens):
    ids = np.zeros((len(tokens), max(len(t) for t in tokens)), np.int64)
    for row, t in zip(ids, tokens):
        row[: len(t)] = t
    return torch.from_numpy(ids).cuda()


def _gpt_last(tokens, ends):
    """Logits at position ends[i] of row i."""
    P = [w.double() for w in _gpt_weights()]
    out = []
    for at in range(0, len(tokens), 8):
        part = tokens[at:at + 8]
        ids = _padded(part)
        n, T = ids.shape
        hidden = torch.ones(T, T, dtype=torch.bool, device="cuda").triu(1)
        where = torch.arange(T, device="cuda")
        x = P[0][ids] + P[1][:T]
        for i in range(LAYERS):
            wq, wk, wv, wo, w1, w2, w3, n1, n2 = P[2 + 9 * i:11 + 9 * i]
            h = _rms(x, n1, EPS)
            q, k, v = (y.view(n, T, HEADS, DHEAD) for y in (h @ wq, h @ wk, h @ wv))
            q, k = _turn_pairs(q, where), _turn_pairs(k, where)
            o = []
            for r in range(n):  # one row of the batch at a time: the scores are large
                sc = torch.einsum("qhd,khd->hqk", q[r], k[r]) / math.sqrt(DHEAD)
                o.append(torch.einsum("hqk,khd->qhd", torch.softmax(sc.masked_fill_(hidden, -math.inf), -1), v[r]))
            x = x + torch.stack(o).reshape(n, T, WIDTH) @ wo
            h = _rms(x, n2, EPS)
            g = h @ w3
            x = x + (h @ w1 * g * torch.sigmoid(g)) @ w2
        last = x[torch.arange(n), torch.as_tensor(np.asarray(ends[at:at + 8]), device="cuda").long()]
        out.append(_rms(last, P[-2], EPS) @ P[-1])
    return torch.cat(out).cpu().numpy()


def _exact_decode(case, seed):
    return {"logits": _gpt_last(_tokens(case, seed, VOCAB), _lengths(case, seed) + case["steps"] - 1), "ids": None}


def _exact_prefill(case, seed):
    return {"logits": _gpt_last(_tokens(case, seed, VOCAB), _lengths(case, seed) - 1), "ids": None}


def _exact_attend(case, seed):
    lens, n = _attend_lengths(case, seed), case["rows"]
    starts = np.concatenate([[0], np.cumsum(lens)])
    q, nk, nv = (_normal((LAYERS, n, WIDTH), seed, 12 + i).double().view(LAYERS, n, HEADS, DHEAD) for i in range(3))
    out = torch.empty((LAYERS, n, HEADS, DHEAD), dtype=torch.float64, device="cuda")
    for layer in range(LAYERS):
        k, v = (_normal((int(starts[-1]), WIDTH), seed, 10 + i, layer) for i in range(2))
        for r in range(n):
            a, b = int(starts[r]), int(starts[r + 1])
            where = torch.arange(b - a, device="cuda")
            kr, vr = (y[a:b].double().view(-1, HEADS, DHEAD) for y in (k, v))
            kr[-1], vr[-1] = nk[layer, r], nv[layer, r]
            kr = _turn_pairs(kr, where)
            qr = _turn_pairs(q[layer, r][None], where[-1:])[0]
            w = torch.softmax(torch.einsum("hd,khd->hk", qr, kr) / math.sqrt(DHEAD), -1)
            out[layer, r] = torch.einsum("hk,khd->hd", w, vr)
    return out.view(LAYERS, n, WIDTH)


def _exact_store(case, seed):
    lens, longest = _store_lengths(case, seed), case["longest"]
    starts = np.concatenate([[0], np.cumsum(lens)])
    planes = []
    for i in range(2):
        x = _normal((int(starts[-1]), WIDTH), seed, 20 + i).double().view(-1, HEADS, DHEAD)
        p = torch.zeros((case["rows"], HEADS, longest, DHEAD), dtype=torch.float64, device="cuda")
        for r, n in enumerate(lens):
            y = x[int(starts[r]):int(starts[r + 1])]
            p[r, :, :n] = (_turn_pairs(y, torch.arange(int(n), device="cuda")) if i == 0 else y).transpose(0, 1)
        planes.append(p)
    return planes


def _exact_matmul(case, seed):
    m, k, n = case["m"], case["k"], case["n"]
    return _normal((m, k), seed, 30).double() @ (_normal((k, n), seed, 31) * 0.05).double()


def _turn_halves(x, base):
    """x [rows, tokens, heads, d]: element i turns with element i + d / 2."""
    d = x.shape[-1]
    f = base ** (-2.0 * torch.arange(d // 2, device=x.device, dtype=torch.float64) / d)
    t = torch.arange(x.shape[1], device=x.device, dtype=torch.float64)[:, None] * f
    c, s = torch.cos(t)[:, None], torch.sin(t)[:, None]
    a, b = x[..., : d // 2], x[..., d // 2:]
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _with_sink(q, k, v, scale, ok, sink):
    """q [T, H, d], k, v [T, G, d] of one row; sink [H] takes its share of the weights."""
    H, G = q.shape[1], k.shape[1]
    out = []
    for h in range(H):
        s = (q[:, h] @ k[:, h * G // H].T * scale).masked_fill(~ok, -math.inf)
        p = torch.softmax(torch.cat([s, sink[h].expand(s.shape[0], 1)], 1), -1)[:, :-1]
        out.append(p @ v[:, h * G // H])
    return torch.stack(out, 1)


def _general_delta(r, k, v, w, a):
    """S <- diag(w) S - (a u)(u^T S) + k v^T, u = k / |k|, o = S^T r, token by token; [rows, T, H, d]."""
    n, T, H, d = r.shape
    S, out = torch.zeros((n, H, d, d), dtype=r.dtype, device=r.device), torch.empty_like(v)
    u = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    au = a * u
    for t in range(T):
        take = torch.matmul(u[:, t, :, None, :], S)
        S = w[:, t, :, :, None] * S - au[:, t, :, :, None] * take + k[:, t, :, :, None] * v[:, t, :, None, :]
        out[:, t] = torch.matmul(r[:, t, :, None, :], S)[:, :, 0]
    return out


def _exact_layered(case, seed):
    cfg = _layered_config(case["width"])
    shapes = _layered_shapes(cfg)
    where = {n: i for i, n in enumerate(shapes)}

    def W(name):
        return _layered_weight(name, shapes[name], where[name]).double()

    lens, eps, mult = _lengths(case, seed), cfg["norm"]["eps"], cfg["residual_mult"]
    ids = _padded(_tokens(case, seed, LAYERED_VOCAB))
    n, T = ids.shape
    x, source = W("embed")[ids] * cfg["embedding"]["scale"], None
    i, j = torch.arange(T, device="cuda")[:, None], torch.arange(T, device="cuda")[None]
    for l, e in enumerate(cfg["layers"]):
        p, m = f"l{l}.", e["mixer"]
        q = p + "mix."
        h = _rms(x, W(p + "norm1"), eps)
        before = torch.cat([torch.zeros_like(h[:, :1]), h[:, :-1]], 1)
        s = h + (before - h) * W(p + "shift")
        H = m["heads"]
        if e["type"] == "general_delta":
            r, k, v, a = (y.view(n, T, H, -1) for y in (s @ W(q + "r").T, s @ W(q + "k").T, s @ W(q + "v").T, torch.sigmoid(s @ W(q + "a").T + W(q + "a.b"))))
            w = torch.exp(-math.exp(-0.5) * torch.sigmoid(torch.tanh(s @ W(q + "w1").T) @ W(q + "w2").T + W(q + "w0"))).view(n, T, H, -1)
            o = _rms(_general_delta(r, k, v, w, a), 1.0, eps).reshape(n, T, -1) * W(q + "norm") * torch.sigmoid(s @ W(q + "g").T)
        else:
            G, full = m["kv_heads"], e["type"] == "attention"
            a, b, v = s @ W(q + "q").T, s @ W(q + "k").T, s @ W(q + "v").T
            if source is None:
                source = v
            else:
                share = W(q + "vmix")
                v = (1 - share) * v + share * source
            if full:
                a, b = _rms(a, W(q + "q.norm"), eps), _rms(b, W(q + "k.norm"), eps)
            a, b = _turn_halves(a.view(n, T, H, -1), m["rot"]["base"]), _turn_halves(b.view(n, T, G, -1), m["rot"]["base"])
            if full:
                ok, sink = j <= i, W(q + "sink")
            else:
                a, b = _rms(a, 1.0, eps), _rms(b, 1.0, eps)
                ok = (j <= i) & ((i - j < m["mask"]["size"]) | (j < m["mask"]["keep_first"]))
                sink = torch.zeros(H, dtype=torch.float64, device="cuda")
            v = v.view(n, T, G, -1)
            o = torch.stack([_with_sink(a[r], b[r], v[r], m["scale"], ok, sink) for r in range(n)]).reshape(n, T, -1)
        y = o @ W(q + "o").T
        x = x + mult * _rms(y * torch.sigmoid(h @ W(p + "rg1").T + W(p + "rg1.b")), W(p + "norm1b"), eps)
        h = _rms(x, W(p + "norm2"), eps)
        y = torch.relu(h @ W(p + "mlp.up").T) ** 2 @ W(p + "mlp.down").T
        x = x + mult * _rms(y * torch.sigmoid(h @ W(p + "rg2").T + W(p + "rg2.b")), W(p + "norm2b"), eps)
    rows, head, norm = torch.arange(n), W("head").T, W("final.norm")
    first, last = (_rms(x[rows, torch.as_tensor(at, device="cuda").long()], norm, eps) @ head for at in (lens - 1, lens + case["steps"] - 1))
    return {"first": first.cpu().numpy(), "logits": last.cpu().numpy(), "ids": None}
