"""Searches that leave a tile, at the numbers of tiles where their way changes: one 32-group
of tiles, several, the last count without levels above the tiles' minima (1024) and the
first with them, each against the oracle."""

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
        _CACHE["sexp"] = (Grammar(tb), oracle.Oracle(tb.blob()))
    return _CACHE["sexp"]


@pytest.mark.parametrize("tiles", [2, 31, 32, 33, 64, 65, 1023, 1024, 1025, 1057])
@pytest.mark.parametrize("shape", ["mirror", "stairs"])
def test_matches_in_far_tiles(has_gpu, tiles, shape):
    g, o = _ctx()
    m = tiles * 2048 - 2 - 7  # tokens: the last tile not full
    if shape == "mirror":     # every closer's match as far back as it can be
        h = min(m // 2, 400000)
        data = b"(" * h + b"a " * (m - 2 * h) + b")" * h
    else:                     # a closer in each 500 tokens, its match some tiles back
        k = m // 1000
        data = (b"(" + b"a " * 499) * k + b"a " * (m % 1000 + 499 * k) + b")" * k
    for d in (data, data[:-1], b"(" + data[1:-1] + b"a"):
        want, got = o.lex_parse(d), g.parse_int(d)
        assert (got is None) == (want is None)
        if want is not None:
            for a, b in zip((got.parent, got.tag, got.kind, got.start, got.end), want):
                np.testing.assert_array_equal(a.cpu().numpy().astype(np.int64), np.asarray(b).astype(np.int64))
