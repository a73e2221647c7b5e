"""More positions than bytes and sentinels allow for: a table blob whose lexer ends an empty
token at every document's start (the front end refuses such grammars, the loader takes them).
The capacity error comes back from every parse entry, no kernel leaves its buffers (the bound
itself on the CPU), and the context parses on."""

import copy
import os
import shutil
import struct
import subprocess

import numpy as np
import pytest

from alpacc_b200 import tables

HERE = os.path.dirname(os.path.abspath(__file__))
ERR_CAPACITY = 5


def test_count_is_cut_to_the_capacity(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    exe = str(tmp_path / "positions_check")
    subprocess.run([nvcc, "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", "-o", exe,
                    os.path.join(HERE, "positions_check.cu")], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.strip() == "ok"


class _EmptyTokens(tables.Tables):
    """Tables whose blob has the produce flag set on every transition of the initial state."""

    def blob(self):
        b = bytearray(super().blob())
        S, C = struct.unpack_from("<2I", b, 16)
        row = 16 + 24 + 256 + S * 512 + 1 * (C + 1) * 2  # the initial state is state 1
        for c in range(C + 1):
            v, = struct.unpack_from("<H", b, row + 2 * c)
            struct.pack_into("<H", b, row + 2 * c, v | 0x8000)
        return bytes(b)


def _empty_tokens(name):
    tb = copy.copy(tables.load(name, "both"))
    tb.__class__ = _EmptyTokens
    return tb


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["json", "sexp"])
@pytest.mark.parametrize("docs", [17, 3000, 700_000])
def test_a_batch_past_the_capacity(has_gpu, name, docs):
    from alpacc_b200 import api
    g = api.Grammar(_empty_tokens(name))
    data, off = np.full(docs, ord("1" if name == "json" else "a"), np.uint8), np.arange(docs + 1, dtype=np.int64)
    with pytest.raises(api.AlpError) as e:
        g.parse_batch_int(data, off)
    assert e.value.code == ERR_CAPACITY
    pg = g.parse_batch_graph(data, off, cap_nodes=4 * docs, cap_brackets=4 * docs)
    try:
        pg.launch()
        with pytest.raises(api.AlpError) as e:
            pg.result()
        assert e.value.code == ERR_CAPACITY
    finally:
        pg.close()
    # one document more than its bytes and sentinels by one position: inside the capacity, no sentence
    assert g.parse_int(data[:1]) is None
    good = api.Grammar(tables.load(name, "both"))
    _, _, valid = good.parse_batch_int(data, off)
    assert int(valid.sum()) == docs
