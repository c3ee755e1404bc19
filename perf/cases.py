"""What a user of this library has it do, as cases that can be timed and compared.

A case is one schedule of forward passes over a paged KV arena, run through the package's public calls exactly
as a model's attention layers make them: `begin_step`, then one call per layer (`KVArena.attention`,
`attention_rope`, `KVArena.attention_host_async`, or `PagedKVCache.attention_opts` for the one-sequence
cache), then `popn` back to where the pass began, as a server does that rejects a draft or drops a finished
turn, so that the next pass finds the same cache.

Fields of a case:
  n_q, n_kv, d, layers   attention geometry
  dtype                  "f16" or "bf16" (storage and inputs; accumulation is 32-bit)
  int8                   int8 KV pages (`quantize_kv`)
  window                 0, or the sliding window of five layers in six (the sixth is global)
  api                    "arena", "cache" (one sequence, `PagedKVCache`) or "host" (pinned host tensors in and out)
  rope                   0 = inputs come rotated, 1 = rotation fused into the append, 2 = QK norm as well
  batch                  sequences; ctx_lo..ctx_hi: tokens each has cached before the pass
  prefix                 the first tokens of every context are one prompt whose pages all sequences share
  prompts                this many of the sequences are new: they start empty and prefill a prompt of
                         prompt_lo..prompt_hi tokens in chunks of `chunk`, while the others decode
  steps, new, reject     after the prompts: `steps` passes in which every sequence feeds `new` tokens
                         (1 = plain decoding, more = verifying a draft) and rolls the last `reject` back

Lengths are spread over their range (over its logarithm where it spans more than a factor of ten) by a fixed
sequence, so that they are ragged and belong to the case; values and the pages' places in the arena come from
the seed.
"""
from __future__ import annotations

import math

import torch

from combsengine_b200 import (CacheConfig, KVArena, PagedKVCache, QKNorm, RotaryEmbedding, attention_rope)

PAGE = 16
DTYPES = {"f16": torch.float16, "bf16": torch.bfloat16}
DEFAULTS = dict(dtype="f16", int8=False, window=0, api="arena", rope=0, batch=1, ctx_lo=0, ctx_hi=0, prefix=0,
                prompts=0, prompt_lo=0, prompt_hi=0, chunk=512, steps=0, new=1, reject=0)
SMOLLM2 = dict(n_q=9, n_kv=3, d=64)      # SmolLM2-135M
QWEN7B = dict(n_q=28, n_kv=4, d=128)     # Qwen2.5-7B
LLAMA8B = dict(n_q=32, n_kv=8, d=128)    # Llama-3-8B
GEMMA4B = dict(n_q=8, n_kv=4, d=256)     # Gemma-3-4B style
FULL_LAYERS = {64: 30, 128: 32, 256: 34}


def make(**fields):
    return {**DEFAULTS, **fields}


def listed():
    return [
        # One sequence, one layer, a few tokens after a 512-token prefix: the smallest call there is, made
        # through the reference's own cache interface. Launch and host latency are all it consists of.
        make(name="cache_decode_1x512", **SMOLLM2, layers=1, api="cache", ctx_lo=512, ctx_hi=512, steps=8),
        # One turn of a single-user chat: a prompt of a few hundred tokens in one chunk, then tokens one at a
        # time through every layer of an 8B model.
        make(name="chat_turn_8b", **LLAMA8B, layers=32, dtype="bf16", rope=1, prompts=1, prompt_lo=333, prompt_hi=333, steps=16),
        # The headline: batched decode, 32 sequences of one to four thousand tokens, 28 layers.
        make(name="decode_7b_b32", **QWEN7B, layers=28, batch=32, ctx_lo=1024, ctx_hi=4096, steps=2),
        # The same call from host tensors (the end-to-end form of the headline).
        make(name="decode_7b_b32_host", **QWEN7B, layers=28, batch=32, ctx_lo=1024, ctx_hi=4096, steps=2, api="host"),
        # The same with int8 pages: twice the context in the same memory.
        make(name="decode_7b_b32_int8", **QWEN7B, layers=28, batch=32, ctx_lo=1024, ctx_hi=4096, steps=2, int8=True),
        # Decode with sliding windows: five local layers per global one, head_dim 256.
        make(name="decode_gemma_b16", **GEMMA4B, layers=34, window=1024, batch=16, ctx_lo=8192, ctx_hi=8192, steps=2),
        # A serving shard: 64 sequences on one GPU that share a 1024-token system prompt, own contexts from
        # a hundred to 32 thousand tokens. The largest decode step.
        make(name="decode_7b_shard64", **QWEN7B, layers=28, batch=64, prefix=1024, ctx_lo=128, ctx_hi=32768, steps=2),
        # Speculative decoding: each sequence verifies the next token and four drafted ones, two are rejected.
        make(name="verify_7b_b8", **QWEN7B, layers=28, dtype="bf16", batch=8, ctx_lo=512, ctx_hi=6144, steps=2, new=5, reject=2),
        # Continuous batching: two prompts are prefilled in chunks in the same passes that decode 24 others.
        make(name="mixed_7b_b26", **QWEN7B, layers=28, dtype="bf16", rope=1, batch=26, ctx_lo=512, ctx_hi=4096,
             prompts=2, prompt_lo=700, prompt_hi=1500),
        # Chunked prefill of eight long prompts. The largest case: tensor throughput.
        make(name="prefill_8b_8x8192", **LLAMA8B, layers=4, rope=1, batch=8, prompts=8, prompt_lo=8192, prompt_hi=8192),
        # Prefill of ragged prompts into int8 pages.
        make(name="prefill_8b_int8_ragged", **LLAMA8B, layers=8, dtype="bf16", rope=1, int8=True, batch=6, prompts=6,
             prompt_lo=300, prompt_hi=2900),
        # Prefill with sliding windows, QK norm and head_dim 256.
        make(name="prefill_gemma_ragged", **GEMMA4B, layers=34, dtype="bf16", rope=2, window=1024, batch=4, prompts=4,
             prompt_lo=500, prompt_hi=4900),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case: any of the kinds above at any geometry, over the sizes between the smallest and the largest."""
    while True:
        geo = rng.choice([SMOLLM2, QWEN7B, LLAMA8B, GEMMA4B])
        full = FULL_LAYERS[geo["d"]]
        c = make(**geo, layers=_log_int(rng, 1, full), dtype=rng.choice(["f16", "bf16"]))
        kind = rng.choice(["cache", "chat", "decode", "decode", "host", "shared", "verify", "mixed", "prefill", "prefill"])
        ctx = sorted(_log_int(rng, 33, 32768) for _ in range(2))
        prompt = sorted(_log_int(rng, 17, 8192) for _ in range(2))
        if kind == "cache":
            c.update(api="cache", layers=min(c["layers"], 8), ctx_lo=ctx[0], ctx_hi=ctx[0], steps=rng.randint(2, 8))
        elif kind == "chat":
            c.update(rope=rng.choice([1, 2]), prompts=1, prompt_lo=prompt[0], prompt_hi=prompt[0], steps=rng.randint(4, 24))
        elif kind in ("decode", "host", "shared", "verify"):
            c.update(batch=_log_int(rng, 1, 64), ctx_lo=ctx[0], ctx_hi=ctx[1], steps=rng.randint(2, 4))
            if kind == "host":
                c.update(api="host")
            if kind == "shared":
                c.update(batch=max(2, c["batch"]), prefix=PAGE * _log_int(rng, 4, 128))
            if kind == "verify":
                c["new"] = rng.randint(2, 9)
                c["reject"] = rng.randint(0, c["new"] - 1)
        else:
            c["prompts"] = _log_int(rng, 1, 8)
            c.update(rope=rng.choice([0, 1, 1, 2]), prompt_lo=prompt[0], prompt_hi=prompt[1], chunk=rng.choice([256, 512, 512, 1024]))
            c["batch"] = c["prompts"]
            if kind == "mixed":
                c["batch"] += _log_int(rng, 2, 48)
                c.update(ctx_lo=ctx[0], ctx_hi=ctx[1])
        if kind != "shared" and rng.random() < 0.25:
            c["int8"] = True
        elif geo is GEMMA4B and kind != "cache":  # the one-sequence cache refuses to roll back past a window
            c["window"] = rng.choice([0, 1024, 1024])
        w = work(c)
        if w["bytes"] <= 40e9 and w["flops"] <= 16e12 and _state_bytes(c) <= 30e9 and sum(_contexts(c)) <= 460_000 and len(_schedule(c)) <= 40:
            return c


# ---- the schedule of a case ------------------------------------------------------------------------------


def _spread(lo, hi, n):
    u = [math.modf((i + 1) * 0.6180339887498949)[0] for i in range(n)]
    if hi > 10 * lo > 0:
        return [int(round(lo * (hi / lo) ** x)) for x in u]
    return [int(round(lo + (hi - lo) * x)) for x in u]


def _contexts(case):
    """Cached tokens per sequence before the pass, the shared prefix among them; new sequences come first, empty."""
    old = case["batch"] - case["prompts"]
    return [0] * case["prompts"] + [case["prefix"] + n for n in _spread(case["ctx_lo"], case["ctx_hi"], old)]


def _schedule(case):
    """[(sequences, new tokens of each, tokens rolled back after the pass)]"""
    left = _spread(case["prompt_lo"], case["prompt_hi"], case["prompts"])
    others = list(range(case["prompts"], case["batch"]))
    out = []
    while any(left):
        who = [i for i, n in enumerate(left) if n]
        new = [min(case["chunk"], left[i]) for i in who]
        for i, n in zip(who, new):
            left[i] -= n
        out.append((who + others, new + [1] * len(others), 0))
    out += [(list(range(case["batch"])), [case["new"]] * case["batch"], case["reject"])] * case["steps"]
    return out


def _grown(case):
    """Most tokens that each sequence gains in the pass, and how many it holds more at its end."""
    most, now = [0] * case["batch"], [0] * case["batch"]
    for who, new, reject in _schedule(case):
        for i, n in zip(who, new):
            now[i] += n
            most[i] = max(most[i], now[i])
            now[i] -= reject
    return most, now


def _windows(case):
    w = case["window"]
    return [w if w and (i + 1) % 6 else None for i in range(case["layers"])]


def _row_bytes(case):
    """Bytes of one token's K and V in the pages of one layer."""
    d = case["d"]
    return 2 * case["n_kv"] * (d + d // 16 if case["int8"] else 2 * d)


def _pages(case):
    ctx, most = _contexts(case), _grown(case)[0]
    return case["prefix"] // PAGE + sum(-(-(c + m) // PAGE) - case["prefix"] // PAGE for c, m in zip(ctx, most)) + 8


def _state_bytes(case):
    tokens = sum(sum(new) for _, new, _ in _schedule(case))
    io = tokens * case["layers"] * case["d"] * 2 * 2 * (case["n_q"] + case["n_kv"])
    # int8 layers are read by chunk steps through one layer of float pages
    return _pages(case) * PAGE * (case["layers"] * _row_bytes(case) + 4 * case["n_kv"] * case["d"]) + io


def work(case):
    """Bytes: every pass and layer reads q, k, v and the cached rows its queries see (rows shared between
    sequences once), writes the output and the new rows.  Operations: 4 per query head, dimension and visible
    (query, key) pair."""
    ctx, row, d = _contexts(case), _row_bytes(case), case["d"]
    wins = _windows(case)
    nbytes = flops = 0
    for w in sorted(set(wins), key=lambda x: x or 0):
        layers = wins.count(w)
        now = list(ctx)
        for who, new, reject in _schedule(case):
            tokens = sum(new)
            nbytes += layers * tokens * (4 * d * (case["n_q"] + case["n_kv"]) + row)
            if case["prefix"]:
                nbytes += layers * case["prefix"] * row
            for i, n in zip(who, new):
                seen = now[i] - case["prefix"] if w is None else min(now[i], w - 1)
                nbytes += layers * seen * row
                if w is None:
                    pairs = now[i] * n + n * (n + 1) // 2
                else:
                    pairs = sum(min(now[i] + j + 1, w) for j in range(n))
                flops += 4 * case["n_q"] * d * layers * pairs
                now[i] += n - reject
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """Outputs are stored in 16 bits and the probabilities meet V in 16 bits as well."""
    return {"rel": 2e-3 if case["dtype"] == "f16" else 1e-2}


# ---- what a user's program has in hand -------------------------------------------------------------------


def _normal(gen, dtype, n):
    return torch.empty(n, device="cuda", dtype=dtype).normal_(generator=gen)


def _fills(who, counts):
    """The steps in which cached rows are put in place, at most 128 Ki tokens each where a sequence allows it."""
    while who:
        n = max(1, sum(sum(counts[:i + 1]) <= 1 << 17 for i in range(len(counts))))
        yield who[:n], counts[:n]
        who, counts = who[n:], counts[n:]


class State:
    def __init__(self):
        self.arena = self.rope = None

    def __del__(self):
        if self.rope is not None:
            self.rope.close()
        if self.arena is not None:
            self.arena.close()


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    dtype = DTYPES[case["dtype"]]
    n_q, n_kv, d, layers = case["n_q"], case["n_kv"], case["d"], case["layers"]
    scale = d ** -0.5
    ctx, (most, end) = _contexts(case), _grown(case)
    longest = max(c + m for c, m in zip(ctx, most))

    def normal(n):
        return _normal(gen, dtype, n)

    st = State()
    if case["api"] == "cache":
        cache = PagedKVCache(layers, CacheConfig(_pages(case) * PAGE, PAGE, quantize_kv=case["int8"]), n_q, n_kv, d, _windows(case), dtype)
        st.arena, seqs = cache.arena, [cache.seq]
    else:
        st.arena = KVArena(layers, n_q, n_kv, d, longest, PAGE, _pages(case), _windows(case), dtype,
                           sliding_popn_refuses=False, quantize_kv=case["int8"])
    arena = st.arena
    arena.set_free_list(torch.randperm(arena.num_pages, generator=torch.Generator().manual_seed(int(seed))).numpy())

    def fill(who, counts):  # cached rows, and with them every layer's pages
        for part, rows in _fills(who, counts):
            arena.begin_step(part, rows)
            for layer in range(layers):
                arena.append(layer, normal(sum(rows) * n_kv * d), normal(sum(rows) * n_kv * d))

    if case["api"] != "cache":
        root = arena.new_seq()
        if case["prefix"]:
            fill([root], [case["prefix"]])
            seqs = [root.fork_prefix(case["prefix"]) for _ in ctx]
        else:
            seqs = [root] + [arena.new_seq() for _ in ctx[1:]]
    old = [(s, n - case["prefix"]) for s, n in zip(seqs, ctx) if n > case["prefix"]]
    if old:
        fill([s for s, _ in old], [n for _, n in old])
    else:
        fill(seqs[:1], [1])
        seqs[0].popn(1)

    if case["rope"]:
        st.rope = RotaryEmbedding(arena, 500000.0, longest)
    norms = [None] * layers
    if case["rope"] == 2:
        norms = [QKNorm(0.1 * normal(d), 0.1 * normal(d), 1e-6, True) for _ in range(layers)]

    st.passes, st.outputs = [], []
    for who, new, reject in _schedule(case):
        t = sum(new)
        q, k, v = (normal(layers * t * h * d).view(layers, -1) for h in (n_q, n_kv, n_kv))
        if case["api"] == "cache":
            q, k, v = (x.view(layers, 1, -1, t, d) for x in (q, k, v))
            out = None
        elif case["api"] == "host":
            q, k, v = (x.cpu().pin_memory() for x in (q, k, v))
            out = torch.zeros_like(q).pin_memory()
        else:
            out = torch.zeros_like(q)
        st.outputs.append(out)
        calls = [(layer, q[layer], k[layer], v[layer], out if out is None else out[layer], norms[layer]) for layer in range(layers)]
        st.passes.append(([seqs[i] for i in who], new, calls, reject))
    st.rollback = [(s, n) for s, n in zip(seqs, end) if n]
    st.api, st.scale = case["api"], scale
    if case["api"] == "cache":
        st.cache = cache
    return st


def run(st):
    arena, rope, scale = st.arena, st.rope, st.scale
    outputs = st.outputs
    if st.api == "cache":
        cache, outputs = st.cache, []
    for seqs, new, calls, reject in st.passes:
        if st.api == "cache":
            pos = cache.seq_len()
            for layer, q, k, v, _, _ in calls:
                outputs.append(cache.attention_opts(layer, q, k, v, pos, scale))
        else:
            arena.begin_step(seqs, new)
            if st.api == "host":
                for layer, q, k, v, out, _ in calls:
                    arena.attention_host_async(layer, q, k, v, out, scale)
                arena.host_sync()
            elif rope is not None:
                for layer, q, k, v, out, norm in calls:
                    attention_rope(arena, layer, rope, q, k, v, scale, norm=norm, out=out)
            else:
                for layer, q, k, v, out, _ in calls:
                    arena.attention(layer, q, k, v, scale, out=out)
        if reject:
            for s in seqs:
                s.popn(reject)
    for s, n in st.rollback:
        s.popn(n)
    return outputs


# ---- the same in 64 bits ---------------------------------------------------------------------------------


def exact(case, seed):
    """What `run` returns, in plain torch and 64 bits.  Rounded are only the values that the cache holds by
    definition: table entries, normed and rotated rows (in the case's type), and int8 pages' bytes and scales."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    dtype, f64 = DTYPES[case["dtype"]], torch.float64
    n_q, n_kv, d, layers, wins = case["n_q"], case["n_kv"], case["d"], case["layers"], _windows(case)
    ctx, most = _contexts(case), _grown(case)[0]
    longest = max(c + m for c, m in zip(ctx, most))

    def normal(n):
        return _normal(gen, dtype, n)

    def stored(x):
        return x.to(dtype).to(f64)

    def quantised(x):  # one scale for 32 values
        g = x.view(-1, 32)
        s = (g.abs().amax(1, keepdim=True) / 127).clamp(min=1e-8)
        return ((g / s).round().clamp(-127, 127) * stored(s)).view(x.shape)

    # the draws of `prepare`, in its order: cached[layer][sequence] = [k, v], each (heads, tokens, d)
    def cached_rows(who, counts, into):
        for part, rows in _fills(who, counts):
            for layer in range(layers):
                kv = [normal(sum(rows) * n_kv * d).split([n * n_kv * d for n in rows]) for _ in range(2)]
                for i, n, k, v in zip(part, rows, *kv):
                    into[layer][i] = [k.view(n_kv, n, d), v.view(n_kv, n, d)]

    shared, cached = [{} for _ in wins], [{} for _ in wins]
    if case["prefix"]:
        cached_rows([0], [case["prefix"]], shared)
    old = [(i, n - case["prefix"]) for i, n in enumerate(ctx) if n > case["prefix"]]
    if old:
        cached_rows([i for i, _ in old], [n for _, n in old], cached)
    else:
        cached_rows([0], [1], [{} for _ in wins])
    norms = [[0.1 * normal(d), 0.1 * normal(d)] for _ in wins] if case["rope"] == 2 else None
    passes = []
    for who, new, reject in _schedule(case):
        q, k, v = (normal(layers * sum(new) * h * d).view(layers, -1) for h in (n_q, n_kv, n_kv))
        passes.append((who, new, reject, q, k, v, torch.zeros(q.shape, dtype=f64, device="cuda")))

    if case["rope"]:
        angle = torch.arange(longest, device="cuda", dtype=f64)[:, None] * 500000.0 ** (-torch.arange(0, d, 2, device="cuda", dtype=f64) / d)
        cos, sin = stored(angle.cos()), stored(angle.sin())

    def normed_rotated(x, weight, pos):
        if weight is not None:
            x = stored(x * (x.square().mean(-1, keepdim=True) + 1e-6).rsqrt() * stored(weight.to(f64) + 1))
        if case["rope"]:
            c, s = cos[pos:pos + x.shape[1]], sin[pos:pos + x.shape[1]]
            a, b = x[..., :d // 2], x[..., d // 2:]
            x = stored(torch.cat([a * c - b * s, b * c + a * s], -1))
        return x

    for layer, w in enumerate(wins):
        int8 = case["int8"] and w is None

        def kept(x):
            return quantised(x).to(torch.float32) if int8 else x.to(dtype)

        held = []
        for i, n in enumerate(ctx):
            rows = torch.empty(2, n_kv, n + most[i], d, device="cuda", dtype=torch.float32 if int8 else dtype)
            at = 0
            for part in (shared[layer].get(0) if case["prefix"] else None, cached[layer].pop(i, None)):
                for j in range(2 if part else 0):
                    rows[j, :, at:at + part[j].shape[1]] = kept(part[j].to(f64).contiguous())
                at += part[0].shape[1] if part else 0
            held.append(rows)
        lengths = list(ctx)
        for who, new, reject, q, k, v, out in passes:
            off = 0
            for i, n in zip(who, new):
                pos, end = lengths[i], lengths[i] + n
                qi, ki, vi = (x[layer, off * h * d:(off + n) * h * d].view(h, n, d).to(f64) for x, h in ((q, n_q), (k, n_kv), (v, n_kv)))
                weights = norms[layer] if norms else (None, None)
                qi, ki = (normed_rotated(x, wt, pos) for x, wt in zip((qi, ki), weights))
                held[i][0, :, pos:end], held[i][1, :, pos:end] = kept(ki.contiguous()), kept(vi.contiguous())
                first = 0 if w is None else max(0, pos - w + 1)
                keys, values = held[i][:, :, first:end].to(f64)
                score = (qi.reshape(n_kv, -1, d) @ keys.transpose(1, 2) * d ** -0.5).view(n_q, n, -1)
                if n > 1:
                    p, t = torch.arange(pos, end, device="cuda")[:, None], torch.arange(first, end, device="cuda")
                    score.masked_fill_((t > p) | (t <= p - (w or end + 1)), -math.inf)
                prob = score.softmax(-1).view(n_kv, -1, end - first)
                out[layer, off * n_q * d:(off + n) * n_q * d] = (prob @ values).view(-1)
                lengths[i] = end - reject
                off += n
    outs = [p[-1] for p in passes]
    if case["api"] == "cache":
        return [x.view(1, n_q, -1, d) for o, p in zip(outs, passes) for x in o]
    return [o.cpu() for o in outs] if case["api"] == "host" else outs
