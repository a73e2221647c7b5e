"""Performance cases: what a program that uses alpacc_b200 has it do.

Every case goes through the Python entry points (``alpacc_b200.api``): single
documents lexed and parsed, token arrays parsed, batches, graph replays,
streams, and host buffers, for the three bundled grammars, from one short
message to documents of half a gibibyte.  Inputs are synthetic
(``alpacc_b200.synth``), arranged by the seed, and all outputs are integers.
"""

from __future__ import annotations

import functools
import os
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

from alpacc_b200 import api, synth, tables

DEPTH = {"json": 16, "sexp": 20, "arithmetic": 12}
DOC = {"json": synth.json_doc, "sexp": synth.sexp_doc, "arithmetic": synth.arith_doc}
# tokens and tree nodes per input byte of the generated documents (measured, for `work`)
TOKENS = {"json": 0.14, "sexp": 0.20, "arithmetic": 0.41}
NODES = {"json": 0.27, "sexp": 0.57, "arithmetic": 1.08}


def listed():
    return [
        # one short message: a request that is parsed by itself, latency only
        {"name": "parse_json_1k", "op": "parse", "grammar": "json", "bytes": 1000, "shift": 0},
        # the arithmetic configuration of the benchmark suite: 1 MiB of expressions
        {"name": "parse_arith_1m", "op": "parse", "grammar": "arithmetic", "bytes": 1 << 20, "shift": 0},
        # an ordinary file of odd size that starts inside a larger buffer, off every alignment
        {"name": "parse_json_4m_odd", "op": "parse", "grammar": "json", "bytes": 4_000_037, "shift": 3},
        # the headline document: 256 MiB of JSON to its tree
        {"name": "parse_json_256m", "op": "parse", "grammar": "json", "bytes": 256 << 20, "shift": 0},
        # tokens only, an ordinary file of odd size
        {"name": "lex_sexp_1m_odd", "op": "lex", "grammar": "sexp", "bytes": 1_048_583, "shift": 0},
        # tokens only, the largest document: the lexer benchmark
        {"name": "lex_json_512m", "op": "lex", "grammar": "json", "bytes": 512 << 20, "shift": 0},
        # the parser alone over tokens that another lexer made
        {"name": "tokens_json_32m", "op": "tokens", "grammar": "json", "bytes": 32 << 20, "shift": 0},
        # serving: many JSON documents of log-normal size in one call
        {"name": "batch_json_20000", "op": "batch", "grammar": "json", "docs": 20000, "median": 4096, "sigma": 1.5},
        # a small batch of short s-expressions
        {"name": "batch_sexp_300", "op": "batch", "grammar": "sexp", "docs": 300, "median": 600, "sigma": 1.5},
        # small batches of one shape, replayed as a CUDA graph on new documents
        {"name": "graph_json_256", "op": "graph", "grammar": "json", "docs": 256, "median": 4096, "sigma": 1.0},
        # input that arrives in pieces: the token stream, as the stdin tool reads it
        {"name": "stream_json_64m", "op": "stream", "grammar": "json", "bytes": 64 << 20, "piece": 16 << 20},
        # host memory in, the tree in host memory out
        {"name": "host_json_16m", "op": "host", "grammar": "json", "bytes": 16 << 20, "shift": 0},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    op = rng.choice(["parse", "parse", "lex", "tokens", "batch", "graph", "stream", "host"])
    if op == "batch":
        return {"op": op, "grammar": rng.choice(["json", "sexp"]), "docs": _log_int(rng, 16, 12000),
                "median": _log_int(rng, 300, 5000), "sigma": rng.choice([0.5, 1.0, 1.5])}
    if op == "graph":
        return {"op": op, "grammar": "json", "docs": _log_int(rng, 16, 2048), "median": _log_int(rng, 500, 8192),
                "sigma": 1.0}
    if op == "stream":
        size = _log_int(rng, 1 << 16, 64 << 20)
        return {"op": op, "grammar": rng.choice(["json", "sexp"]), "bytes": size,
                "piece": max(4097, size // rng.randint(1, 8))}
    top = {"parse": 200 << 20, "lex": 400 << 20, "tokens": 32 << 20, "host": 12 << 20}[op]
    grammar = rng.choice(["json", "json", "sexp", "arithmetic"])
    if grammar == "arithmetic":
        top = min(top, 16 << 20)  # expressions: a formula file, not a data dump
    if grammar == "sexp":
        top = min(top, 96 << 20)
    return {"op": op, "grammar": grammar, "bytes": _log_int(rng, 500, top),
            "shift": rng.choice([0, 0, 0, 1, 8]) if op in ("parse", "lex") else 0}


@functools.lru_cache(maxsize=None)
def _tables(grammar, mode):
    return tables.load(grammar, mode)


def _parallel(jobs):
    with ThreadPoolExecutor(min(8, os.cpu_count() or 1)) as ex:
        return list(ex.map(lambda f: f(), jobs))


def _shuffled_digits(a, rng):
    """The bytes with the digits 1 to 9 renamed: other content, the same tokens."""
    lut = np.arange(256, dtype=np.uint8)
    lut[49:58] = rng.permutation(9).astype(np.uint8) + 49
    return lut[a]


def _cut(expr, record):
    """An expression cut at the top-level '+' next after every `record` bytes."""
    step = (expr == ord("(")).astype(np.int8) - (expr == ord(")")).astype(np.int8)
    plus = np.flatnonzero((expr == ord("+")) & (np.cumsum(step, dtype=np.int32) == 0))
    at = np.unique(np.searchsorted(plus, np.arange(record, len(expr), record)))
    cuts = plus[at[at < len(plus)]]
    return [expr[a:b] for a, b in zip(np.concatenate([[0], cuts + 1]), np.concatenate([cuts, [len(expr)]]))]


@functools.lru_cache(maxsize=4)
def _records(grammar, size):
    """The records of a document of `size` bytes, the same for every seed, so that
    documents of one size have one number of tokens and nodes."""
    record = min(max(size // 64, 120), 1 << 20)
    if grammar == "arithmetic":
        # (the generator ends its expressions early and pads with spaces: ask for more, cut it off)
        return _cut(synth.arith_doc(size + 40000, DEPTH[grammar], synth.SEED_BASE)[:size - 2], record)[:-1]
    count = (size - 1) // (record + 1)
    room = size - 1 - count
    sizes = [room // count + (1 if i < room % count else 0) for i in range(count)]
    return _parallel([functools.partial(DOC[grammar], n, DEPTH[grammar] - 1, synth.SEED_BASE + i)
                      for i, n in enumerate(sizes)])


def _document(grammar, size, seed):
    """One document of exactly `size` bytes: a list (a sum) of records, their order
    and their digits by the seed."""
    rng = np.random.default_rng(seed)
    recs = _records(grammar, size)
    lead, sep, tail = {"json": (b"[", b",", b"]"), "sexp": (b"(", b" ", b")"), "arithmetic": (b" ", b"+", b" ")}[grammar]
    out = np.full(size, 32, np.uint8)
    p = 0
    for i, k in enumerate(rng.permutation(len(recs))):
        out[p] = (lead if i == 0 else sep)[0]
        out[p + 1:p + 1 + len(recs[k])] = recs[k]
        p += 1 + len(recs[k])
    out[p] = tail[0]
    return _shuffled_digits(out, rng)


@functools.lru_cache(maxsize=2)
def _documents(grammar, docs, median, sigma, cap):
    """The documents of a batch, the same for every seed."""
    sizes = synth.lognormal_sizes(docs, median=median, sigma=sigma, cap=cap, seed=synth.SEED_BASE + 4)
    depth = 8 if grammar == "json" else 20
    parts = np.array_split(sizes, max(1, min(16, len(sizes) // 64)))
    made = _parallel([functools.partial(synth.batch, grammar, s, depth, synth.SEED_BASE + i)
                      for i, s in enumerate(parts)])
    return [d[o[i]:o[i + 1]] for d, o in made for i in range(len(o) - 1)]


def _batch(case, seed):
    """Documents back to back and their offsets; their order and digits by the seed."""
    rng = np.random.default_rng(seed)
    cap = 4 << 20 if case["op"] == "batch" else 16 * case["median"]
    docs = _documents(case["grammar"], case["docs"], case["median"], case["sigma"], cap)
    docs = [docs[k] for k in rng.permutation(len(docs))]
    off = np.zeros(len(docs) + 1, np.int64)
    np.cumsum([len(d) for d in docs], out=off[1:])
    return _shuffled_digits(np.concatenate(docs), rng), off


def _on_gpu(a, shift=0):
    """The array on the GPU, `shift` elements into its buffer."""
    buf = torch.empty(len(a) + shift, dtype=torch.from_numpy(a[:1]).dtype, device="cuda:0")
    buf[shift:].copy_(torch.from_numpy(a))
    return buf[shift:]


def prepare(case, seed):
    op = case["op"]
    mode = "lexer" if op in ("lex", "stream") else "both"
    g = api.Grammar(_tables(case["grammar"], mode), device=0)
    state = {"op": op, "g": g}
    if op in ("batch", "graph"):
        data, off = _batch(case, seed)
        state["x"], state["off"] = _on_gpu(data), _on_gpu(off)
        if op == "graph":
            state["graph"] = g.parse_batch_graph(state["x"], state["off"])
        return state
    doc = _document(case["grammar"], case["bytes"], seed)
    if op == "host":
        state["x"] = doc
    elif op == "tokens":
        state["tokens"] = g.lex_int(_on_gpu(doc))
    elif op == "stream":
        x = _on_gpu(doc)
        state["pieces"] = [x[i:i + case["piece"]] for i in range(0, len(doc), case["piece"])]
        state["cap"] = len(doc) // 2 + 16
    else:
        state["x"] = _on_gpu(doc, case["shift"])
    return state


def _fields(tree):
    return (tree.parent, tree.tag, tree.kind, tree.start, tree.end)


def run(state):
    op, g = state["op"], state["g"]
    if op == "parse":
        return _fields(g.parse_int(state["x"]))
    if op == "lex":
        return g.lex_int(state["x"])
    if op == "tokens":
        return _fields(g.parse_tokens_int(*state["tokens"]))
    if op == "batch":
        tree, node_off, valid = g.parse_batch_int(state["x"], state["off"])
        return _fields(tree) + (node_off, valid)
    if op == "graph":
        pg = state["graph"]
        pg.load(state["x"], state["off"])
        pg.launch()
        tree, node_off, valid = pg.result()
        return _fields(tree) + (node_off, valid)
    if op == "stream":
        s = g.lex_stream(state["cap"])
        for p in state["pieces"]:
            s.push(p)
        tokens = s.end()
        s.close()
        return tokens
    return g.parse_host(state["x"])


def work(case):
    """Input bytes read once and output arrays written once.  The counts of
    tokens and nodes are the generators' averages; no floating-point work."""
    grammar, op = case["grammar"], case["op"]
    if op in ("batch", "graph"):
        # the documents' expected total: the mean of the size distribution
        n = int(case["docs"] * case["median"] * float(np.exp(case["sigma"] ** 2 / 2)))
        return {"bytes": n + 8 * case["docs"] + int(29 * NODES[grammar] * n) + 9 * case["docs"], "flops": 0}
    n = case["bytes"]
    if op in ("lex", "stream"):
        return {"bytes": n + int(20 * TOKENS[grammar] * n), "flops": 0}
    if op == "tokens":
        return {"bytes": int(20 * TOKENS[grammar] * n) + int(29 * NODES[grammar] * n), "flops": 0}
    return {"bytes": n + int(29 * NODES[grammar] * n), "flops": 0}


def exact(case, seed):
    """All outputs are whole numbers: they have no nearer value than themselves."""
    return None
