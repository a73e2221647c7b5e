"""A tile's list of searches that it cannot answer, on the CPU: tests/tree_room_check.cu
counts them against the list's room over batches of short rejected documents, which have
next to no nodes to pay for it, with valid documents between them."""

import os
import shutil
import subprocess

import numpy as np
import pytest

import oracle
from alpacc_b200 import synth, tables

HERE = os.path.dirname(os.path.abspath(__file__))
BAD = {"json": [b"1 2", b"}", b"null null", b"1,2", b"]", b"[", b"[1]]", b""],
       "sexp": [b")", b"a b", b"()", b"(", b"(a))", b""],
       "arithmetic": [b"1 1", b")", b"+", b"(1", b"1)", b""]}
GOOD = {"json": b"[" + b"1," * 1500 + b"[]]", "sexp": b"(" * 900 + b"a" + b")" * 900, "arithmetic": b"1" + b"+(1)" * 700}


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    out = str(tmp_path_factory.mktemp("room") / "tree_room_check")
    subprocess.run([nvcc, "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", "-o", out,
                    os.path.join(HERE, "tree_room_check.cu")], check=True)
    return out


@pytest.mark.parametrize("name", ["json", "sexp", "arithmetic"])
def test_listed_searches_fit_their_tile(exe, tmp_path, name):
    tb = tables.load(name, "both")
    p, o = tb.parser, oracle.Oracle(tb.blob())
    use = [0] * len(p.pairs)
    for key, i in zip(p.keys, p.key_pair):
        use[i] |= 2 if key[p.q] == p.start else 1
    w = [len(p.pairs)]
    for (s0, s1, a, b), u in zip(p.pairs, use):
        w += [s0, s1 - s0, a, b - a, u]
    w += [len(p.stack)] + [int(x) for x in p.stack] + [len(p.pseq)] + [int(x) for x in p.pseq]
    w += [len(p.arity)] + [int(x) for x in p.arity] + [int(x) for x in p.prod_term]
    kmap = dict(zip(p.keys, p.key_pair))

    def positions(doc):
        lexed = o.lex_futhark(doc)
        arr = [p.start] + ([] if lexed is None else [int(t) for t in lexed[0]]) + [p.end]
        n = len(arr)
        return [(kmap.get(tuple(arr[j] if 0 <= j < n else p.empty for j in range(i - p.q, i + p.k)), 0xffff), i == 0)
                for i in range(n)]

    good = positions(GOOD[name])
    assert o.lex_parse(GOOD[name]) is not None
    batches = [positions(b) * 1500 for b in BAD[name]]  # one kind each, valid documents after it
    batches = [x + good + x for x in batches]
    mixed = [positions(b) for b in BAD[name]]
    rng = np.random.default_rng(3)
    batches.append(sum([mixed[k] for k in rng.integers(0, len(mixed), 3000)], []) + good)
    gen = {"json": synth.json_doc, "sexp": synth.sexp_doc, "arithmetic": synth.arith_doc}[name]
    batches.append(positions(gen(30000, 12, 8).tobytes()))
    w.append(len(batches))
    for b in batches:
        w.append(len(b))
        w += [int(x) for pos in b for x in pos]
    path = str(tmp_path / "batches")
    with open(path, "w") as f:
        f.write(" ".join(map(str, w)))
    out = subprocess.run([exe, path], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.startswith("ok "), out.stdout
