"""tree_escape_kernel's parts of a tile: documents whose last tiles list a chosen number of
searches, below and past the first part and the rounds of the rest, with and without the
levels of minima (1024 tiles), alone and as documents of a batch, against the oracle."""

import numpy as np
import pytest

import oracle
from alpacc_b200 import tables

pytestmark = pytest.mark.gpu

_CACHE = {}


def _ctx():
    from alpacc_b200.api import Grammar
    if not _CACHE:
        tb = tables.load("sexp", "both")
        _CACHE["x"] = (Grammar(tb), oracle.Oracle(tb.blob()))
    return _CACHE["x"]


def _doc(k, fill):
    return b"(" * k + b"a " * fill + b")" * k


def _same(got, want):
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a.cpu().numpy().astype(np.int64), np.asarray(b).astype(np.int64))


def _fields(t):
    return (t.parent, t.tag, t.kind, t.start, t.end)


@pytest.mark.parametrize("k", [1, 31, 32, 33, 63, 64, 65, 96, 287, 288, 289, 320, 321, 2040, 5000, 300_000])
@pytest.mark.parametrize("fill", [4500, 2_200_000])
def test_parts_of_a_list(has_gpu, k, fill):
    g, o = _ctx()
    d = _doc(k, fill)
    want = o.lex_parse(d)
    _same(_fields(g.parse_int(d)), want)
    assert g.parse_int(d[:-1]) is None and g.parse_int(d + b")") is None


def test_parts_in_a_batch_and_a_graph(has_gpu):
    g, o = _ctx()
    docs = [_doc(k, f) for k, f in ((70, 3000), (33, 2100), (5000, 10), (1, 4100), (2500, 2500), (300, 0), (9000, 9000))] * 2
    docs[5:5] = [b")"] * 700
    off = np.zeros(len(docs) + 1, np.int64)
    off[1:] = np.cumsum([len(d) for d in docs])
    data = np.frombuffer(b"".join(docs), np.uint8)
    pg = g.parse_batch_graph(data, off)
    try:
        pg.launch()
        for tree, node_off, valid in (g.parse_batch_int(data, off), pg.result()):
            for i, d in enumerate(docs):
                want = o.lex_parse(d)
                assert bool(valid[i]) == (want is not None)
                if want is not None:
                    _same([f[node_off[i]:node_off[i + 1]] for f in _fields(tree)], want)
    finally:
        pg.close()
