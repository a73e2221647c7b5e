"""The lexer's walk and write passes at the sizes where they can go wrong: documents
that start and end on every offset of a chunk, dense chunks (more tokens than a
chunk's first records hold), ignored and empty last tokens, inputs off every
alignment -- batches and single documents against the oracle."""

import numpy as np
import pytest

import oracle
from alpacc_b200 import synth, tables

pytestmark = pytest.mark.gpu

_CACHE = {}

def _ctx(name):
    from alpacc_b200.api import Grammar
    if name not in _CACHE:
        tb = tables.load(name, "lexer")
        _CACHE[name] = (Grammar(tb), oracle.Oracle(tb.blob()))
    return _CACHE[name]


def _check_batch(g, o, docs):
    off = np.concatenate([[0], np.cumsum([len(d) for d in docs])]).astype(np.int64)
    data = np.frombuffer(b"".join(docs), np.uint8)
    term, start, end, tok_off, valid = (x.cpu().numpy() for x in g.lex_batch_int(data, off))
    assert tok_off[-1] == len(term)
    for i, d in enumerate(docs):
        want = o.lex_futhark(d) if d else None
        assert bool(valid[i]) == (want is not None), (i, d[:40])
        if want is not None:
            a, b = tok_off[i], tok_off[i + 1]
            for got, w in ((term, want[0]), (start, want[1]), (end, want[2])):
                np.testing.assert_array_equal(got[a:b].astype(np.int64), np.asarray(w).astype(np.int64))


@pytest.mark.parametrize("pad", [0, 1, 30, 31, 32, 33, 62, 63, 64, 65])
@pytest.mark.parametrize("name", ["json", "sexp"])
def test_documents_at_every_chunk_offset(has_gpu, name, pad):
    g, o = _ctx(name)
    atom = b"1" if name == "json" else b"a"
    open_, close = (b"[", b"]") if name == "json" else (b"(", b")")
    docs = [open_ + b" " * max(pad - 2, 0) + close] if pad >= 2 else [atom] * pad
    rng = np.random.default_rng(pad)
    docs += [atom] * 70                                     # one byte each: two boundaries a byte
    docs += [b"", atom + b" ", b" " + atom, b" ", open_ + close, b"", atom * 31, atom * 33 + b"  ", open_ * 40]
    for _ in range(60):
        k = int(rng.integers(1, 70))
        docs.append(bytes(rng.choice(np.frombuffer(atom + b" " + open_ + close, np.uint8), k)))
    docs += [open_ * 200 + close * 200, (atom + b" ") * 300]  # 32 and 16 tokens a chunk
    _check_batch(g, o, docs)
    _check_batch(g, o, docs[::-1])


@pytest.mark.parametrize("size", [1, 31, 32, 33, 63, 64, 65, 127, 2047, 2048, 2049, 16383, 16384, 16385, 40000])
def test_dense_and_shifted_documents(has_gpu, size):
    import torch
    g, o = _ctx("sexp")
    for d in (b"(" * size, (b"a " * size)[:size], (b"abc(" * size)[:size], synth.sexp_doc(max(size, 2), 20, size).tobytes()):
        want = o.lex_futhark(d)
        for shift in (0, 1, 5, 8, 15):
            buf = torch.zeros(len(d) + shift, dtype=torch.uint8, device="cuda")
            buf[shift:] = torch.from_numpy(np.frombuffer(d, np.uint8).copy())
            got = g.lex_int(buf[shift:])
            assert (got is None) == (want is None)
            if want is not None:
                for a, b in zip(got, want):
                    np.testing.assert_array_equal(a.cpu().numpy().astype(np.int64), np.asarray(b).astype(np.int64))
