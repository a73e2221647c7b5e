"""Batches that are mostly short rejected documents (no admissible pair, too many closers or
openers, empty) before, between and after valid documents that cross the parser's tiles:
every document's verdict and every valid document's tree against the oracle, through the
batch call and through the replay of a graph."""

import numpy as np
import pytest

import oracle
from alpacc_b200 import synth, tables

pytestmark = pytest.mark.gpu

BAD = {"json": [b"1 2", b"}", b"null null", b"1,2", b"]", b"[", b"[1]]", b"", b"#"],
       "sexp": [b")", b"a b", b"(", b"(a))", b"", b"((a)"],
       "arithmetic": [b"1 1", b")", b"+", b"(1", b"1)", b"", b"2 2 2"]}
_CACHE = {}


def _ctx(name):
    from alpacc_b200.api import Grammar
    if name not in _CACHE:
        tb = tables.load(name, "both")
        _CACHE[name] = (Grammar(tb), oracle.Oracle(tb.blob()), {})
    return _CACHE[name]


def _good(name):
    gen = {"json": synth.json_doc, "sexp": synth.sexp_doc, "arithmetic": synth.arith_doc}[name]
    o, c, atom, tail = {"json": (b"[", b"]", b"1", b",2"), "sexp": (b"(", b")", b"a", b" b"),
                        "arithmetic": (b"(", b")", b"1", b"+2")}[name]
    deep = o * 1200 + atom + tail + c * 1200
    flat = (o + atom + tail * 1700 + c)
    return [deep, flat, gen(25_000, 12, 41).tobytes(), o + atom + c, gen(260_000, 16, 42).tobytes()]


def _check(name, docs, result):
    _, o, known = _ctx(name)
    tree, node_off, valid = result
    node_off, valid = node_off.cpu().numpy(), valid.cpu().numpy()
    fields = [t.cpu().numpy() for t in (tree.parent, tree.tag, tree.kind, tree.start, tree.end)]
    seen = 0
    for i, d in enumerate(docs):
        if d not in known:
            known[d] = o.lex_parse(d)
        want = known[d]
        assert bool(valid[i]) == (want is not None), (i, d[:20])
        if want is None:
            continue
        seen += 1
        for got, ref in zip(fields, want):
            np.testing.assert_array_equal(got[node_off[i]:node_off[i + 1]].astype(np.int64), np.asarray(ref).astype(np.int64))
    return seen


def _run(name, docs):
    g = _ctx(name)[0]
    off = np.zeros(len(docs) + 1, np.int64)
    off[1:] = np.cumsum([len(d) for d in docs])
    data = np.frombuffer(b"".join(docs), np.uint8)
    assert _check(name, docs, g.parse_batch_int(data, off)) > 0
    pg = g.parse_batch_graph(data, off)
    try:
        for _ in range(2):
            pg.launch()
            assert _check(name, docs, pg.result()) > 0
    finally:
        pg.close()


@pytest.mark.parametrize("name,kind", [(n, k) for n in BAD for k in range(len(BAD[n]))])
def test_many_rejected_documents_of_one_kind(has_gpu, name, kind):
    bad, good = BAD[name][kind], _good(name)
    docs = []
    for i, g in enumerate(good):
        docs += [bad] * (520 + 97 * i) + [g]
    _run(name, docs + [bad] * 1100 + good[:2] + [bad] * 3)


@pytest.mark.parametrize("name", sorted(BAD))
@pytest.mark.parametrize("before", [0, 1, 2045, 2046, 2047, 2048, 2049, 4095])
def test_a_valid_document_at_a_tile_edge(has_gpu, name, before):
    """`before` positions in front of it: rejected documents of two positions and more."""
    good = _good(name)
    one = BAD[name][1]  # ⊢ token ⊣ (a sexp's: ⊢ a b ⊣)
    pos = 4 if name == "sexp" else 3
    docs = [one] * (before // pos) + [b""] * ((before % pos + 1) // 2)
    rng = np.random.default_rng(before)
    for d in good[:3] + good[:1]:
        docs += [d] + [BAD[name][k] for k in rng.integers(0, len(BAD[name]), 900)]
    _run(name, docs)
