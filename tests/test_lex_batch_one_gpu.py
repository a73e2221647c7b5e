"""A lexer batch of one document: its offsets and validity are those of this call, whatever
the verdict, in every form of the token pass; the wire format with one rejected input."""

import numpy as np
import pytest

import oracle
from alpacc_b200 import tables, wire

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lex_split", [1, 0])
@pytest.mark.parametrize("mode", ["lexer", "both"])
def test_one_rejected_document_after_a_valid_one(has_gpu, mode, lex_split):
    from alpacc_b200.api import Grammar
    tb = tables.load("json", mode)
    g, o = Grammar(tb), oracle.Oracle(tb.blob())
    g.set_tuning(g.get_tuning()[:4] + [lex_split])
    for data in (b"[1, 2, 3]", b'"open', b"#", b"[1, 2", b'[1, "x'):
        want = o.lex_futhark(data)
        term, start, end, tok_off, valid = g.lex_batch_int(data, np.array([0, len(data)], np.int64))
        assert valid.tolist() == [0 if want is None else 1]
        assert tok_off.tolist() == [0, len(term)] and len(term) == len(start) == len(end)
        if want is not None:
            for got, ref in zip((term, start, end), want):
                np.testing.assert_array_equal(got.cpu().numpy().astype(np.int64), np.asarray(ref).astype(np.int64))
    assert g.lex_int(b"#") is None and g.lex_int(b"[1]") is not None


def test_one_rejected_input_through_the_wire_format(has_gpu):
    from alpacc_b200.api import Grammar
    g = Grammar(tables.load("json", "lexer"))
    for docs, ok in (([b"[1]"], [True]), ([b"#"], [False]), ([b""], [False])):
        res = wire.read_lexer_outputs(wire.run(g, "lexer", wire.write_inputs(docs)))
        assert [r is not None for r in res] == ok
