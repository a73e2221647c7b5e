"""parse_tree_kernel at the sizes where it can go wrong (edges of its tiles, of a
warp's positions and of the queue), a grammar outside its compact tables (the
general kernels), and the production sequence alone, against the oracle."""

import numpy as np
import pytest

import oracle
from alpacc_b200 import synth, tables

pytestmark = pytest.mark.gpu

_CACHE = {}


def _ctx(name):
    from alpacc_b200.api import Grammar
    if name not in _CACHE:
        tb = tables.build_tables(_chain(), "both") if name == "chain" else tables.load(name, "both")
        _CACHE[name] = (Grammar(tb), oracle.Oracle(tb.blob()))
    return _CACHE[name]


def _chain(levels=40):
    """Forty unit productions above every value: more nodes a pair than the compact tables hold."""
    rules = ["A%d -> A%d." % (i, i + 1) for i in range(levels)]
    rules += ['A%d [Nest] -> "(" A0 ")".' % levels, "A%d [Atom] -> atom." % levels]
    return "params {\n  lookback = 1.\n  lookahead = 1.\n}\natom = /[a-z]+/.\nignore = /\\s/.\n" + "\n".join(rules) + "\n"


def _same(g, o, data: bytes):
    want, got = o.lex_parse(data), g.parse_int(data)
    assert (got is None) == (want is None), data[:60]
    if want is not None:
        for a, b in zip((got.parent, got.tag, got.kind, got.start, got.end), want):
            np.testing.assert_array_equal(a.cpu().numpy().astype(np.int64), np.asarray(b).astype(np.int64))


# positions of "(a a ... a)" are tokens + 2: edges of a thread's 4, a warp's 128, a tile's 2048
@pytest.mark.parametrize("positions", [5, 127, 128, 129, 132, 2047, 2048, 2049, 2176, 4096, 4097, 65535, 65536 + 3])
@pytest.mark.parametrize("shape", ["flat", "deep", "comb"])
def test_edges_of_tiles_and_warps(has_gpu, positions, shape):
    g, o = _ctx("sexp")
    m = positions - 2  # tokens
    if shape == "flat":
        data = b"(" + b"a " * (m - 2) + b")"
    elif shape == "deep":  # every closer's match lies as far back as it can
        h = (m - 1) // 2
        data = b"(" * h + b"a " * (m - 2 * h) + b")" * h
    else:  # long lists inside short ones: far and near matches side by side
        k = max((m - 2) // 3, 0)
        data = b"(" + b"(a)" * k + b"a " * (m - 2 - 3 * k) + b")"
    _same(g, o, data)
    _same(g, o, data[:-1])
    _same(g, o, data + b")")


@pytest.mark.parametrize("depth", [1, 3, 40, 700])
def test_a_grammar_outside_the_compact_tables(has_gpu, depth):
    g, o = _ctx("chain")
    _same(g, o, b"(" * depth + b"x" + b")" * depth)
    _same(g, o, b"(" * depth + b"x" + b")" * (depth - 1))


@pytest.mark.parametrize("name", ["json", "arithmetic"])
def test_production_sequence_and_batches(has_gpu, name):
    g, o = _ctx(name)
    gen = synth.json_doc if name == "json" else synth.arith_doc
    docs = [gen(s, 12, 300 + s).tobytes() for s in (60, 5000, 70001)]
    for d in docs:
        tree = g.parse_int(d)
        prods = g.pre_productions_int(g.lex_int(d)[0])
        assert len(prods) == len(tree)
        pick = tree.kind == 0
        np.testing.assert_array_equal(prods[pick].cpu().numpy(), tree.tag[pick].cpu().numpy())
    docs = docs + [b"", docs[1][:-3]] + docs
    off = np.concatenate([[0], np.cumsum([len(d) for d in docs])])
    tree, node_off, valid = g.parse_batch_int(np.frombuffer(b"".join(docs), np.uint8), off)
    for i, d in enumerate(docs):
        want = o.lex_parse(d)
        assert bool(valid[i]) == (want is not None), i
        if want is not None:
            np.testing.assert_array_equal(tree.parent[node_off[i]:node_off[i + 1]].cpu().numpy(), want[0])
