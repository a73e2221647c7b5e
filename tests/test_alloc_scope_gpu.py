"""An output allocator that stays set (alp_set_output_alloc, as a C program sets it once) is
asked by the entry points that take it, once a call, and by no other: state labels, host
buffers, tuning and shards give what they give without one."""

import ctypes

import numpy as np
import pytest

from alpacc_b200 import synth, tables

pytestmark = pytest.mark.gpu


def _with_allocator(g, calls):
    """Sets an allocator on g that hands out tensors and counts its calls."""
    import torch
    from alpacc_b200 import api

    keep = []

    @api._ALLOC_FN
    def alloc(user, n, ptrs):
        calls.append(n)
        for i in range(5):
            keep.append(torch.empty(n, dtype=torch.int64, device="cuda"))
            ptrs[i] = keep[-1].data_ptr()
        return 0

    api.native().alp_set_output_alloc(g.h, alloc, None)
    return alloc, keep


@pytest.mark.parametrize("name", ["json", "sexp"])
def test_only_the_calls_that_take_it(has_gpu, name):
    from alpacc_b200 import api, spec
    from alpacc_b200.shard import parse_split
    gen = {"json": synth.json_doc, "sexp": synth.sexp_doc}[name]
    data = gen(300_000, 12, 5)
    off = np.array([0, len(data)], np.int64)
    tb = tables.load(name, "both")
    plain, g, calls = api.Grammar(tb), api.Grammar(tb), []
    held = _with_allocator(g, calls)
    states = spec.exact_states(plain, data).cpu().numpy()
    np.testing.assert_array_equal(spec.exact_states(g, data).cpu().numpy(), states)
    for call in ("lex_host", "parse_host"):
        for a, b in zip(getattr(g, call)(data), getattr(plain, call)(data)):
            np.testing.assert_array_equal(a, b)
    for a, b in zip(g.parse_batch_host(data, off), plain.parse_batch_host(data, off)):
        np.testing.assert_array_equal(a, b)
    toks = plain.lex_int(data)
    host = [t.cpu().numpy() for t in toks]
    for a, b in zip(parse_split([g, plain], host, [len(host[0]) // 2]), plain.parse_host(data)):
        np.testing.assert_array_equal(a, b)
    saved = g.get_tuning()
    g.tune(data, 1)
    g.set_tuning(saved[:6])
    assert calls == []
    # and once by one that does
    L, p = api.native(), [ctypes.c_void_p() for _ in range(3)]
    n, valid = ctypes.c_int64(0), ctypes.c_int(0)
    x = g._as_device_bytes(data)
    rc = L.alp_lex(g.h, ctypes.c_void_p(x.data_ptr()), x.numel(), *[ctypes.byref(q) for q in p], ctypes.byref(n),
                   ctypes.byref(valid))
    assert rc == 0 and valid.value == 1 and calls == [n.value] and p[0].value == held[1][0].data_ptr()
    assert n.value == len(toks[0])
