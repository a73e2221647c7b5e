"""Batches of documents far shorter than a thread's 64 bytes, empty and rejected ones among
them, up to thousands a tile: the write pass follows the boundaries document by document.
Every document's tokens against the oracle, alone and behind a long document."""

import numpy as np
import pytest

import oracle
from alpacc_b200 import tables

pytestmark = pytest.mark.gpu

PIECES = {"json": [b"", b"1", b"12", b" 1", b"1 ", b"  ", b"[]", b"[1,2]", b"#", b'"a b"', b'"', b"\n{}\n", b"true,false",
                   b"[" * 9 + b"]" * 9, b"1" * 40, b"-1.5e3 ,null"],
          "sexp": [b"", b"a", b"ab", b" a", b"a ", b"  ", b"()", b"(a b)", b"#", b"(" * 20 + b"x" * 30 + b")" * 20]}
_CACHE = {}


def _ctx(name):
    from alpacc_b200.api import Grammar
    if name not in _CACHE:
        tb = tables.load(name, "lexer")
        o = oracle.Oracle(tb.blob())
        _CACHE[name] = (Grammar(tb), {d: o.lex_futhark(d) for d in PIECES[name]})
    return _CACHE[name]


@pytest.mark.parametrize("name", sorted(PIECES))
@pytest.mark.parametrize("few", [1, 2, 5, 99])
@pytest.mark.parametrize("lead", [0, 1, 31, 63, 64, 16383, 16384, 40001])
def test_tiny_documents(has_gpu, name, few, lead):
    g, known = _ctx(name)
    rng = np.random.default_rng(1000 * few + lead)
    pieces = [PIECES[name][k] for k in rng.permutation(len(PIECES[name]))[:few]]
    if not any(pieces):
        pieces.append(b"a" if name == "sexp" else b"1")
    docs = [pieces[k] for k in rng.integers(0, len(pieces), 6000)]
    front = [b" " * lead] if lead else []
    off = np.zeros(len(front) + len(docs) + 1, np.int64)
    off[1:] = np.cumsum([len(d) for d in front + docs])
    data = np.frombuffer(b"".join(front + docs), np.uint8)
    term, start, end, tok_off, valid = (t.cpu().numpy().astype(np.int64) for t in g.lex_batch_int(data, off))
    assert int(tok_off[-1]) == len(term)
    for i, d in enumerate(docs, len(front)):
        want = known[d]
        assert bool(valid[i]) == (want is not None), (i, d)
        if want is not None:
            a, b = tok_off[i], tok_off[i + 1]
            assert b - a == len(want[0]), (i, d)
            for got, ref in zip((term, start, end), want):
                np.testing.assert_array_equal(got[a:b], np.asarray(ref).astype(np.int64))
