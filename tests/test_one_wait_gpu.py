"""Lexer and pair sums in one run of launches, and the tile scans in one launch: the sizes
around a chunk of the scans (1024 lexer tiles of 8 KiB, 1024 position tiles), the largest
input that takes this route and the smallest that does not, a batch of one document, and
token ids of no terminal."""

import numpy as np
import pytest

import oracle
from alpacc_b200 import synth, tables

pytestmark = pytest.mark.gpu

_CACHE = {}


def _ctx(name):
    from alpacc_b200.api import Grammar
    if name not in _CACHE:
        tb = tables.load(name, "both")
        _CACHE[name] = (Grammar(tb), oracle.Oracle(tb.blob()))
    return _CACHE[name]


def _fields(t):
    return [x.cpu().numpy().astype(np.int64) for x in (t.parent, t.tag, t.kind, t.start, t.end)]


def _same(got, want):
    for a, b in zip(got, want):
        np.testing.assert_array_equal(np.asarray(a).astype(np.int64), np.asarray(b).astype(np.int64))


# positions (tokens + 2) and bytes: one, two and three chunks of either scan, and their edges
@pytest.mark.parametrize("tokens,size", [
    (1 << 20, None), ((1 << 20) - 2, None), ((1 << 20) - 1, None), (2 << 20, None),
    (500, 8 << 20), (500, (8 << 20) + 1), (3 << 20, (16 << 20) - 1),
])
def test_chunks_of_the_scans(has_gpu, tokens, size):
    g, o = _ctx("sexp")
    data = b"(" + b"(a)" * ((tokens - 2) // 3) + b"a " * ((tokens - 2) % 3) + b")"
    if size is not None:
        data = b" " * (size - len(data)) + data
    _same(_fields(g.parse_int(data)), o.lex_parse(data))
    assert g.parse_int(data[:-1]) is None


@pytest.mark.parametrize("extra", [-1, 0, 1])
def test_the_route_changes_at_its_limit(has_gpu, extra):
    g, _ = _ctx("json")
    doc = synth.json_doc(70001, 12, 5).tobytes()
    small = _fields(g.parse_int(doc))
    pad = (1 << 24) - 2 + extra - len(doc)
    _same(_fields(g.parse_int(doc + b" " * pad)), small)
    at_end = _fields(g.parse_int(b" " * pad + doc))
    at_end[3] -= pad
    at_end[4] -= pad
    root = small[3] == 0
    _same(at_end[:3], small[:3])
    _same([at_end[3][~root], at_end[4][~root]], [small[3][~root], small[4][~root]])
    off = np.array([0, len(doc), len(doc) + pad, len(doc) + pad], np.int64)  # and a rejected and an empty document
    tree, node_off, valid = g.parse_batch_int(np.frombuffer(doc + b" " * pad, np.uint8), off)
    assert valid.cpu().tolist() == [1, 0, 0]
    m = int(node_off[1])
    _same([x[:m] for x in _fields(tree)], small)


@pytest.mark.parametrize("size", [1, 2, 63, 64, 2047, 30000])
def test_a_batch_of_one_document(has_gpu, size):
    g, o = _ctx("sexp")
    for d in (b"a" * size, b"(" * size, synth.sexp_doc(size, 9, size).tobytes()):
        want = o.lex_parse(d)
        tree, node_off, valid = g.parse_batch_int(np.frombuffer(d, np.uint8), np.array([0, len(d)], np.int64))
        assert bool(valid[0]) == (want is not None)
        one = g.parse_int(d)
        assert (one is None) == (want is None)
        if want is not None:
            _same(_fields(tree), want)
            _same(_fields(one), want)


@pytest.mark.parametrize("at", [0, 1, 700, -1])
def test_ids_of_no_terminal(has_gpu, at):
    g, o = _ctx("sexp")
    data = b"(" + b"(a)" * 1000 + b")"
    term, start, end = (np.asarray(x).astype(np.int64) for x in o.lex_futhark(data))
    assert g.parse_tokens_int(term.astype(np.int32), start, end) is not None
    bad = term.copy()
    bad[at] = 0xffff
    assert g.parse_tokens_int(bad.astype(np.int32), start, end) is None
    bad[at] = 0x10000
    with pytest.raises(Exception, match="terminal id out of range"):
        g.parse_tokens_int(bad.astype(np.int32), start, end)
    assert g.parse_tokens_int(term.astype(np.int32), start, end) is not None
