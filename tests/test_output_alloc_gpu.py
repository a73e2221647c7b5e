"""The Python entry points let the native call allocate their outputs when the
counts are known (alp_set_output_alloc): exact sizes, every form of the lexer's
and the parser's passes, rejected and empty inputs, and an allocator that fails."""

import numpy as np
import pytest

import oracle
from alpacc_b200 import synth, tables

pytestmark = pytest.mark.gpu


def _np(ts):
    return [t.cpu().numpy().astype(np.int64) for t in ts]


def _fields(t):
    return (t.parent, t.tag, t.kind, t.start, t.end)


@pytest.mark.parametrize("lex_split,parse_split", [(1, 1), (0, 1), (1, 0), (0, 0)])
def test_outputs_have_their_own_exact_size(has_gpu, lex_split, parse_split):
    from alpacc_b200.api import Grammar
    tb = tables.load("json", "both")
    g, o = Grammar(tb), oracle.Oracle(tb.blob())
    g.set_tuning(g.get_tuning()[:4] + [lex_split, parse_split])
    for data in (b"[1]", synth.json_doc(8191, 8, 5).tobytes(), synth.json_doc(200_001, 16, 6).tobytes(), b"[1", b""):
        toks, want = g.lex_int(data), o.lex_futhark(data)
        assert (toks is None) == (want is None)
        tree, wtree = g.parse_int(data), o.lex_parse(data)
        assert (tree is None) == (wtree is None)
        for got, ref in ((toks, want), (tree and _fields(tree), wtree)):
            if got is None:
                continue
            for t, a, b in zip(got, _np(got), ref):
                np.testing.assert_array_equal(a, np.asarray(b).astype(np.int64))
                assert t.untyped_storage().nbytes() == t.numel() * t.element_size()
        off = np.array([0, 0, len(data)], np.int64)
        if len(data):
            bt, node_off, valid = g.parse_batch_int(data, off)
            assert valid.tolist() == [0, 0 if wtree is None else 1] and int(node_off[-1]) == len(bt)
            if wtree is not None:
                a = int(node_off[1])
                for x, b in zip(_np(_fields(bt)), wtree):
                    np.testing.assert_array_equal(x[a:], np.asarray(b).astype(np.int64))
            term, start, end, tok_off, valid = g.lex_batch_int(data, off)
            assert int(tok_off[-1]) == len(term) == len(start) == len(end)
            if want is not None:
                np.testing.assert_array_equal(start.cpu().numpy(), np.asarray(want[1]).astype(np.int64))


def test_a_failing_allocator_leaves_the_context_usable(has_gpu, monkeypatch):
    from alpacc_b200 import api
    g = api.Grammar("json")
    data = synth.json_doc(50_000, 8, 7).tobytes()
    ref_lex, ref_tree = g.lex_int(data), g.parse_int(data)
    off = np.array([0, len(data)], np.int64)

    def fail(self, n, ptrs=None):
        raise MemoryError("no room for %d" % n)

    with monkeypatch.context() as m:
        m.setattr(api._Outputs, "make", fail)
        for call in (lambda: g.lex_int(data), lambda: g.parse_int(data), lambda: g.lex_batch_int(data, off),
                     lambda: g.parse_batch_int(data, off)):
            with pytest.raises(MemoryError):
                call()
    for a, b in zip(_np(g.lex_int(data)) + _np(_fields(g.parse_int(data))), _np(ref_lex) + _np(_fields(ref_tree))):
        np.testing.assert_array_equal(a, b)
    # without an allocator the outputs are the context's own again
    host = g.parse_host(np.frombuffer(data, np.uint8))
    np.testing.assert_array_equal(host[0], ref_tree.parent.cpu().numpy())
