"""The general kernels (expansion and the two searches), which the bundled grammars reach only
in shards and in the fused position pass: a grammar outside the compact tables over several
tiles, in batches with many rejected documents, as a graph and through host memory, against
the oracle."""

import numpy as np
import pytest

import oracle
from alpacc_b200 import tables

pytestmark = pytest.mark.gpu

LEVELS = 34  # unit productions above every value: a pair has more nodes than the compact tables hold
_CACHE = {}


def _source():
    rules = ["A%d -> A%d." % (i, i + 1) for i in range(LEVELS)]
    rules += ['A%d [List] -> "(" L ")".' % LEVELS, "A%d [Atom] -> atom." % LEVELS, "L [More] -> A0 L.", "L [Done] -> ."]
    return "params {\n  lookback = 1.\n  lookahead = 1.\n}\natom = /[a-z]+/.\nignore = /\\s/.\n" + "\n".join(rules) + "\n"


def _ctx():
    from alpacc_b200.api import Grammar
    if not _CACHE:
        tb = tables.build_tables(_source(), "both")
        o = oracle.Oracle(tb.blob())
        known = {}

        def want(d):
            if d not in known:
                known[d] = o.lex_parse(d)
            return known[d]
        _CACHE["x"] = (Grammar(tb), want)
    return _CACHE["x"]


def _same(got, want):
    for a, b in zip(got, want):
        a = a.cpu().numpy() if hasattr(a, "cpu") else a
        np.testing.assert_array_equal(a.astype(np.int64), np.asarray(b).astype(np.int64))


def _fields(t):
    return (t.parent, t.tag, t.kind, t.start, t.end)


def _flat(m):
    return b"(" + b"a " * m + b")"


def _deep(m):
    return b"(" * m + b"b" + b")" * m


# positions are tokens + 2: around a tile of 2048, and many tiles
@pytest.mark.parametrize("doc", [_flat(m) for m in (0, 2043, 2044, 2045, 2046, 9000, 70000)] +
                         [_deep(m) for m in (1022, 1023, 1024, 9000)] + [_deep(700)[:-1] + b"(x)" * 5000 + b")"],
                         ids=lambda d: "%d" % len(d))
@pytest.mark.parametrize("split", [1, 0])
def test_single_documents_over_tiles(has_gpu, doc, split):
    g, want = _ctx()
    g.set_tuning(g.get_tuning()[:5] + [split])
    try:
        assert want(doc) is not None
        for _ in range(2):  # (the fused pass sizes itself from the parse before)
            _same(_fields(g.parse_int(doc)), want(doc))
        assert g.parse_int(doc[:-1]) is None and g.parse_int(doc + b")") is None and g.parse_int(doc + b" a") is None
        _same(g.parse_host(np.frombuffer(doc, np.uint8)), want(doc))
    finally:
        g.set_tuning(g.get_tuning()[:5] + [1])


@pytest.mark.parametrize("bad", [b"", b")", b"a b", b"(", b"(a))", b"#", None], ids=str)
def test_batches_and_graphs(has_gpu, bad):
    g, want = _ctx()
    mix = [b"", b")", b"a b", b"(", b"(a))", b"#", b"((a b) c)", b"()"]
    rng = np.random.default_rng(17)
    docs = []
    for i, good in enumerate([_deep(1500), _flat(3000), b"(a)", _flat(2044), _deep(5)]):
        docs += [mix[k] for k in rng.integers(0, len(mix), 400 + 7 * i)] if bad is None else [bad] * (400 + 7 * i)
        docs.append(good)
    off = np.zeros(len(docs) + 1, np.int64)
    off[1:] = np.cumsum([len(d) for d in docs])
    data = np.frombuffer(b"".join(docs), np.uint8)

    def check(fields, node_off, valid):
        node_off, valid = np.asarray(node_off), np.asarray(valid)
        fields = [np.asarray(f) for f in fields]
        for i, d in enumerate(docs):
            assert bool(valid[i]) == (want(d) is not None), (i, d[:20])
            if want(d) is not None:
                _same([f[node_off[i]:node_off[i + 1]] for f in fields], want(d))

    tree, node_off, valid = g.parse_batch_int(data, off)
    check([t.cpu() for t in _fields(tree)], node_off.cpu(), valid.cpu())
    host = g.parse_batch_host(data, off)
    check(host[:5], host[5], host[6])
    pg = g.parse_batch_graph(data, off)
    try:
        for _ in range(2):
            pg.launch()
            tree, node_off, valid = pg.result()
            check([t.cpu() for t in _fields(tree)], node_off.cpu(), valid.cpu())
    finally:
        pg.close()


def test_graph_capacities(has_gpu):
    from alpacc_b200.api import AlpError
    g, _ = _ctx()
    docs = [_flat(900)] * 5
    off = np.arange(6, dtype=np.int64) * len(docs[0])
    data = np.frombuffer(b"".join(docs), np.uint8)
    n = len(g.parse_batch_int(data, off)[0])
    for caps in ((n // 3, 1 << 20), (n, 7)):
        pg = g.parse_batch_graph(data, off, cap_nodes=caps[0], cap_brackets=caps[1])
        try:
            pg.launch()
            with pytest.raises(AlpError) as e:
                pg.result()
            assert e.value.code == 5  # ALP_ERR_CAPACITY
        finally:
            pg.close()
