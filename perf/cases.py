"""Performance cases: what programs built on this framework have it do, through its public entry points.

The two engines (gpt-oss-20b, Qwen3-30B-A3B) are opened once per process, as a serving program does, with the
seeded synthetic weights that bench.py uses; a case's state is one request (or one batch of requests) with
token ids of its own.  Requests of the one-sequence calls start at position 0, so a state needs nothing in the
engine from before; requests of the batch calls keep their own sequences (KV caches) of the engine's pool from
prepare() on.

Kinds of cases:
  oss_generate   a chat turn, greedy: the whole prompt, then `new` tokens decoded on the device
  oss_sample     a chat turn with temperature: the prompt, then every token drawn on the host from the logits
  oss_prefill    a prompt alone (scoring, the time to the first token): next token and logits
  oss_batch      one step of continuous batching: one new token of each of `rows` sequences of different ages;
                 with logits=True the rows' logits come back as well, for sampling
  oss_mixed      one step in which `rows` sequences decode and a new request brings its prompt of `prompt` tokens
  qwen_generate  a chat turn of the second engine, greedy
  qwen_prefill   its prompt alone
"""
import ctypes as C

import numpy as np

import cpubrrr_b200 as B

OSS_VOCAB, QWEN_VOCAB = 199999, 151936      # ids drawn for prompts (below the special tokens)
OSS_POOL = 192                              # sequences of the batch engine: three sets of the largest batch
TOP_K, TEMP_MILLI = 40, 800

_engines = {}
_free = []


def _oss():
    if "oss" not in _engines:
        eng = B.Engine.synth(B.gptoss_20b_cfg(), 2)
        eng.batch_open(OSS_POOL)
        _free[:] = range(OSS_POOL)
        _engines["oss"] = eng
    return _engines["oss"]


def _qwen():
    if "qwen" not in _engines:
        _engines["qwen"] = B.QwenEngine.synth(B.qwen3_30b_a3b_cfg(), 3)
    return _engines["qwen"]


class _Request:
    """One state; gives its sequences back to the pool when it goes."""

    def __init__(self, case, engine):
        self.case, self.engine, self.seqs = case, engine, []

    def take(self, n):
        if len(_free) < n:
            raise MemoryError("out of memory: no free sequence in the pool")
        self.seqs = [_free.pop() for _ in range(n)]

    def __del__(self):
        _free.extend(self.seqs)


def listed():
    return [
        # the shortest things asked of a server: a few words, answered at once; every launch counts
        {"name": "oss prefill 7", "kind": "oss_prefill", "prompt": 7},
        # an assistant's answer drawn at temperature 0.8: host sampling after every token
        {"name": "oss sample 45+16", "kind": "oss_sample", "prompt": 45, "new": 16},
        # bench.py's own workload: 73 prompt tokens, 128 greedy ones
        {"name": "oss generate 73+128", "kind": "oss_generate", "prompt": 73, "new": 128},
        # questions about a long document: decoding over a long cache
        {"name": "oss generate 1900+200", "kind": "oss_generate", "prompt": 1900, "new": 200},
        # a system prompt with a question (ragged against every tile size)
        {"name": "oss prefill 333", "kind": "oss_prefill", "prompt": 333},
        # a long document alone, near the context limit
        {"name": "oss prefill 3001", "kind": "oss_prefill", "prompt": 3001},
        # a lightly loaded server, sampling on the host
        {"name": "oss batch 5 logits", "kind": "oss_batch", "rows": 5, "context": 600, "logits": True},
        # a loaded server
        {"name": "oss batch 64", "kind": "oss_batch", "rows": 64, "context": 60, "logits": False},
        # a server that takes a new prompt in beside running requests
        {"name": "oss mixed 21+190", "kind": "oss_mixed", "rows": 21, "context": 90, "prompt": 190},
        # the second engine: short chat turn, longer answer, prompt alone
        {"name": "qwen generate 14+24", "kind": "qwen_generate", "prompt": 14, "new": 24},
        {"name": "qwen generate 64+128", "kind": "qwen_generate", "prompt": 64, "new": 128},
        {"name": "qwen prefill 350", "kind": "qwen_prefill", "prompt": 350},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["oss_generate", "oss_sample", "oss_prefill", "oss_batch", "oss_mixed", "qwen_generate", "qwen_prefill"])
    if kind == "oss_generate":
        return {"kind": kind, "prompt": _log(rng, 4, 1900), "new": _log(rng, 8, 200)}
    if kind == "oss_sample":
        return {"kind": kind, "prompt": _log(rng, 4, 300), "new": _log(rng, 4, 32)}
    if kind == "oss_prefill":
        return {"kind": kind, "prompt": _log(rng, 2, 3000)}
    if kind == "oss_batch":
        rows = _log(rng, 1, 64)
        logits = rows <= 16 and rng.random() < 0.5
        return {"kind": kind, "rows": rows, "context": rng.randint(8, max(8, min(600, 3840 // rows))), "logits": logits}
    if kind == "oss_mixed":
        return {"kind": kind, "rows": _log(rng, 1, 32), "context": rng.randint(8, 90), "prompt": _log(rng, 8, 400)}
    if kind == "qwen_generate":
        return {"kind": kind, "prompt": _log(rng, 4, 100), "new": _log(rng, 8, 128)}
    return {"kind": kind, "prompt": _log(rng, 2, 350)}


def prepare(case, seed):
    rng = np.random.default_rng([seed, 7])
    kind = case["kind"]
    if kind.startswith("qwen"):
        s = _Request(case, _qwen())
        s.prompt = rng.integers(0, QWEN_VOCAB, case["prompt"], dtype=np.uint32)
        return s
    s = _Request(case, _oss())
    if kind in ("oss_generate", "oss_sample", "oss_prefill"):
        s.prompt = rng.integers(0, OSS_VOCAB, case["prompt"], dtype=np.uint32)
        s.rng_seed = int(rng.integers(1, 1 << 62))
        return s
    # running requests: sequences with `context` / 2 .. `context` tokens in their caches, and the token to feed next
    rows, extra = case["rows"], 1 if kind == "oss_mixed" else 0
    s.take(rows + extra)
    age = rng.integers(max(1, case["context"] // 2), case["context"] + 1, rows)
    for q, n in zip(s.seqs, age):
        s.engine.batch_prefill(q, rng.integers(0, OSS_VOCAB, int(n), dtype=np.uint32))
    toks = rng.integers(0, OSS_VOCAB, rows, dtype=np.uint32)
    pos, seq = age.astype(np.uint32), np.array(s.seqs[:rows], np.uint32)
    if extra:
        n = case["prompt"]
        toks = np.concatenate([toks, rng.integers(0, OSS_VOCAB, n, dtype=np.uint32)])
        pos = np.concatenate([pos, np.arange(n, dtype=np.uint32)])
        seq = np.concatenate([seq, np.full(n, s.seqs[-1], np.uint32)])
    s.toks, s.pos, s.seq = toks, pos, seq
    return s


def run(s):
    case, eng = s.case, s.engine
    kind = case["kind"]
    if kind in ("oss_generate", "qwen_generate"):
        first = eng.prefill(s.prompt)
        return {"first": first, "tokens": eng.decode(first, len(s.prompt), case["new"])}
    if kind in ("oss_prefill", "qwen_prefill"):
        return {"next": eng.prefill(s.prompt), "logits": eng.logits()}
    if kind == "oss_sample":
        sample, state = B.lib().brrr_sample_logits, C.c_uint64(B.lib().brrr_rng_seed(s.rng_seed))
        out = np.empty(case["new"], np.uint32)
        eng.prefill(s.prompt)
        for i in range(case["new"]):
            logits = eng.logits()
            out[i] = sample(logits.ctypes.data, logits.size, TEMP_MILLI, TOP_K, C.byref(state))
            if i + 1 < case["new"]:
                eng.run(out[i], len(s.prompt) + i)
        return {"tokens": out, "logits": logits}
    if case.get("logits"):
        toks, logits = eng.batch_step(s.toks, s.pos, s.seq, logits=True)
        return {"tokens": toks, "logits": logits}
    return {"tokens": eng.batch_step(s.toks, s.pos, s.seq)}


# ---- what a pass cannot do without
def _distinct(experts, picked, rows):
    """Experts that `rows` tokens reach, each taking `picked` of them."""
    return experts * (1.0 - (1.0 - picked / experts) ** rows)


def _oss_pass(rows, keys, heads):
    """One pass of `rows` token rows over the layers, every weight once; `keys`: (cached positions read, new positions) per
    sequence and row in all, for full and for windowed layers; `heads`: rows whose logits are wanted."""
    d, layers, q, kv, ne, k, vocab = 2880, 24, 4096, 512, 32, 4, 201088
    q8 = lambda n, m: n * m + n * (m // 32) * 4  # noqa: E731
    expert = 3 * d * (d // 32) * 17 + 3 * d * 4
    read_full, read_win, dots_full, dots_win = keys
    by = layers * (q8(q + 2 * kv, d) + q8(d, q) + ne * d * 4 + _distinct(ne, k, rows) * expert) + rows * d * 2
    by += (layers // 2) * (read_full + read_win) * kv * 8 + layers * rows * kv * 8
    fl = 2.0 * rows * layers * (d * (q + 2 * kv) + q * d + ne * d + k * 3 * d * d) + 4.0 * (layers // 2) * (dots_full + dots_win) * q
    if heads:
        by += q8(vocab, d) + heads * vocab * 4
        fl += 2.0 * heads * vocab * d
    return by, fl


def _qwen_pass(rows, keys, heads):
    d, layers, q, kv, ne, k, ff, vocab = 2048, 48, 4096, 512, 128, 8, 768, 151936
    q4, q6 = (lambda n, m: n * (m // 256) * 144), (lambda n, m: n * (m // 256) * 210)
    expert = 2 * q4(ff, d) + q6(d, ff)
    read, _, dots, _ = keys
    by = layers * (q4(q + 2 * kv, d) + q4(d, q) + ne * d * 4 + _distinct(ne, k, rows) * expert + read * kv * 8 + rows * kv * 8) + rows * q4(1, d)
    fl = 2.0 * rows * layers * (d * (q + 2 * kv) + q * d + ne * d + k * 3 * d * ff) + 4.0 * layers * dots * q
    if heads:
        by += q6(vocab, d) + heads * vocab * 4
        fl += 2.0 * heads * vocab * d
    return by, fl


def _prompt_keys(n, window=128):
    """Keys of a prompt from position 0: nothing is read from before; row i sees i + 1 keys, or the window's."""
    full = n * (n + 1) // 2
    win = sum(min(i + 1, window) for i in range(n))
    return 0, 0, full, win


def _decode_keys(positions, window=128):
    full = sum(p + 1 for p in positions)
    win = sum(min(p + 1, window) for p in positions)
    return full - len(positions), win - len(positions), full, win


def work(case):
    kind = case["kind"]
    one = _qwen_pass if kind.startswith("qwen") else _oss_pass
    if kind in ("oss_batch", "oss_mixed"):
        ages = [int(case["context"] * 0.75)] * case["rows"]
        keys, n = _decode_keys(ages), case["rows"]
        if kind == "oss_mixed":
            keys, n = tuple(a + b for a, b in zip(keys, _prompt_keys(case["prompt"]))), n + case["prompt"]
        by, fl = one(n, keys, n)
        return {"bytes": by if case.get("logits") else by - n * 201088 * 4, "flops": fl}
    n = case["prompt"]
    by, fl = one(n, _prompt_keys(n), 1)
    steps = {"oss_generate": case.get("new", 0), "qwen_generate": case.get("new", 0), "oss_sample": case.get("new", 0) - 1}.get(kind, 0)
    for i in range(steps):
        b, f = one(1, _decode_keys([n + i]), 1)
        by, fl = by + b, fl + f
    return {"bytes": by, "flops": fl}


def tolerance(case):
    # both engines fix the order of every float sum: tokens and logits are the same bits whatever the schedule
    return "exact"
