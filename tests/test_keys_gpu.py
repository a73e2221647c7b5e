"""parse_keys_kernel at the sizes where it can go wrong: ends and ⊢ on every place of a
lane's eight positions, of a warp's 256 and of a tile's 2048, for each lookaround it is
built for, against the oracle -- valid documents, and ones with a token taken out, put
twice or exchanged, whose pairs may have no record."""

import numpy as np
import pytest

import oracle
from alpacc_b200 import synth, tables

pytestmark = pytest.mark.gpu

_CACHE = {}


def _ctx(name, q=None, k=None):
    from alpacc_b200.api import Grammar
    key = (name, q, k)
    if key not in _CACHE:
        if q is None:
            tb = tables.load(name, "both")
        else:
            tb = tables.build_tables(LISTS % (q, k), "both")
        _CACHE[key] = (Grammar(tb), oracle.Oracle(tb.blob()))
    return _CACHE[key]


LISTS = """params {
  lookback = %d.
  lookahead = %d.
}
atom = /[a-z]+/.
ignore = /\\s/.
S [Top] -> L.
L [Cons] -> E L.
L [Nil] -> .
E [Nest] -> "(" L ")".
E [Atom] -> atom.
"""


def _batch(g, o, docs):
    off = np.concatenate([[0], np.cumsum([len(d) for d in docs])]).astype(np.int64)
    tree, node_off, valid = g.parse_batch_int(np.frombuffer(b"".join(docs), np.uint8), off)
    got = [x.cpu().numpy().astype(np.int64) for x in (tree.parent, tree.tag, tree.kind, tree.start, tree.end)]
    node_off, valid = node_off.cpu().numpy(), valid.cpu().numpy()
    for i, d in enumerate(docs):
        want = o.lex_parse(d) if d else None
        assert bool(valid[i]) == (want is not None), (i, d[:60])
        if want is not None:
            a, b = node_off[i], node_off[i + 1]
            for x, w in zip(got, want):
                np.testing.assert_array_equal(x[a:b], np.asarray(w).astype(np.int64))


def _single(g, o, d):
    want, got = o.lex_parse(d), g.parse_int(d)
    assert (got is None) == (want is None), d[:60]
    if want is not None:
        for a, b in zip((got.parent, got.tag, got.kind, got.start, got.end), want):
            np.testing.assert_array_equal(a.cpu().numpy().astype(np.int64), np.asarray(b).astype(np.int64))


CASES = [("lists", 1, 1), ("lists", 1, 2), ("lists", 1, 3), ("lists", 2, 1), ("lists", 2, 2), ("json", None, None)]


def _doc(name, tokens):
    if name == "json":
        return (b"[" + b"1," * max(tokens // 2 - 2, 0) + b"[]" * (tokens % 2) + b"1]")
    return (b"(a)" * (tokens // 3) + b"a " * (tokens % 3))[: 3 * tokens]


@pytest.mark.parametrize("name,q,k", CASES)
def test_heads_on_every_place(has_gpu, name, q, k):
    g, o = _ctx(name, q, k)
    rng = np.random.default_rng(7)
    docs = [_doc(name, t) for t in list(range(1, 40)) + [250, 251, 252, 253, 254, 255, 256, 257, 1500, 2046, 2047, 2048]]
    for d in list(docs):
        if len(d) > 2:
            i = int(rng.integers(1, len(d)))
            docs += [d[:i] + d[i + 1:], d[:i] + d[i - 1:i] + d[i:]]
    docs += [b"", b" "]
    _batch(g, o, docs)
    _batch(g, o, [docs[i] for i in rng.permutation(len(docs))])


@pytest.mark.parametrize("name,q,k", CASES)
def test_ends_on_every_place(has_gpu, name, q, k):
    g, o = _ctx(name, q, k)
    for t in [1, 2, 5, 6, 7, 8, 9, 13, 14, 15, 253, 254, 255, 256, 510, 2045, 2046, 2047, 2048, 4094, 4095, 20001]:
        d = _doc(name, t)
        _single(g, o, d)
        _single(g, o, d[:-1])
        _single(g, o, d[: len(d) // 2] + d[len(d) // 2 + 1:])


def test_random_documents(has_gpu):
    g, o = _ctx("json")
    for s in range(6):
        d = synth.json_doc(30000 + 1777 * s, 12, s).tobytes()
        _single(g, o, d)
        _batch(g, o, [d[:0], d, d[1:], d])
