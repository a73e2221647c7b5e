"""The rule behind parse_tree_kernel, on the CPU: a pair's rights and lefts are the
open ends of its nodes, so the left that a right matches names the node's parent.
For every bundled grammar and lookaround, the parents found this way and the
verdict are the oracle's (which searches exscan(arity - 1) and the bracket depths
apart, futhark/parser.fut:153-184, 286-298), on valid and on corrupted documents."""

import numpy as np
import pytest

import oracle
from alpacc_b200 import synth, tables

ROOT, END = -1, -2


def _open_ends(p):
    """Per pair: (symbols and nodes of its rights, of its lefts, parent inside the pair or
    None per node), or None for a pair that no key names."""
    use = [0] * len(p.pairs)
    for key, i in zip(p.keys, p.key_pair):
        use[i] |= 2 if key[p.q] == p.start else 1
    end_syms = {p.stack[p.pairs[i][0]] & 0x7fffffff for i in range(len(use)) if use[i] == 2}
    assert len(end_syms) == 1 and 3 not in use
    (end_sym,) = end_syms
    out = []
    for i, (s0, s1, a, b) in enumerate(p.pairs):
        br = p.stack[s0:s1]
        rights = [x for x in br if not x >> 31]
        lefts = [x & 0x7fffffff for x in br if x >> 31]
        assert list(br[:len(rights)]) == rights, "rights before lefts"
        stack, taken, inside = ([END, ROOT] if use[i] == 2 else []), [], []
        for k in range(b - a):
            if stack:
                inside.append(stack.pop())
                assert inside[-1] != END
            else:
                inside.append(None)
                taken.append(k)
            stack += [k] * p.arity[p.pseq[a + k]]
        if len(taken) == len(rights) - 1 and rights[-1] == end_sym:
            taken.append(END)
        if not use[i]:
            out.append(None)
            continue
        assert len(taken) == len(rights) and len(stack) == len(lefts), (i, use[i])
        out.append((list(zip(rights, taken)), list(zip(lefts, stack)), inside))
    return out


def _by_brackets(p, ends, kmap, terms):
    """(parents, accepted) of ⊢ terms ⊣."""
    arr = [p.start] + terms + [p.end]
    n, stack, parents, ok = len(arr), [], [], True
    for i in range(n):
        pid = kmap.get(tuple(arr[j] if 0 <= j < n else p.empty for j in range(i - p.q, i + p.k)))
        if pid is None:
            return None, False
        rights, lefts, inside = ends[pid]
        first = len(parents)
        parents += [0 if e in (None, ROOT) else first + e for e in inside]
        for sym, node in rights:
            if not stack:
                return None, False
            lsym, waits = stack.pop()
            ok = ok and lsym == sym
            if node != END:
                parents[first + node] = max(waits, 0)
        stack += [(sym, node if node < 0 else first + node) for sym, node in lefts]
    return parents, ok and not stack


CASES = [("json", 1, 3), ("sexp", 1, 1), ("arithmetic", 1, 1), ("arithmetic", 2, 2), ("sexp", 1, 2), ("arithmetic", 3, 1)]


@pytest.mark.parametrize("name,q,k", CASES)
def test_parents_and_verdict_follow_from_the_brackets(name, q, k):
    with open(tables.grammar_path(name)) as f:
        src = f.read()
    if name != "json":
        src = src.replace("lookback = 1.", "lookback = %d." % q).replace("lookahead = 1.", "lookahead = %d." % k)
    tb = tables.build_tables(src, "both")
    p, o = tb.parser, oracle.Oracle(tb.blob())
    assert (p.q, p.k) == (q, k)
    ends, kmap = _open_ends(p), dict(zip(p.keys, p.key_pair))
    gen = {"json": synth.json_doc, "sexp": synth.sexp_doc, "arithmetic": synth.arith_doc}[name]
    o_, c_ = (b"[", b"]") if name == "json" else (b"(", b")")
    atom = b"1" if name != "sexp" else b"a"
    docs = [gen(s, d, 70 + s).tobytes() for s, d in ((90, 4), (3000, 8), (40000, 20))] + [o_ * 300 + atom + c_ * 300]
    rng = np.random.default_rng(9)
    for d in list(docs):
        for _ in range(12):
            b = bytearray(d)
            at = int(rng.integers(0, len(b)))
            b[at:at + 1] = [b"", o_, c_, b[at:at + 1] * 2][int(rng.integers(0, 4))]
            docs.append(bytes(b))
    accepted = 0
    for d in docs:
        lexed, want = o.lex_futhark(d), o.lex_parse(d)
        if lexed is None:
            continue
        got, ok = _by_brackets(p, ends, kmap, [int(t) for t in lexed[0]])
        assert ok == (want is not None), d[:60]
        if ok:
            accepted += 1
            np.testing.assert_array_equal(np.array(got), np.asarray(want[0]))
    assert accepted >= 4
