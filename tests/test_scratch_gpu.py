"""Device memory that a lex call takes beside its input and outputs: 2.7 bytes a byte of input
where the walk keeps token records, 0.2 in the forms without one."""

import ctypes

import pytest

from alpacc_b200 import synth, tables

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lex_split,per_byte", [(0, 0.25), (1, 2.8)])
def test_scratch_of_a_lex_call(has_gpu, lex_split, per_byte):
    import torch
    from alpacc_b200.api import Grammar, native
    n = 96 << 20
    g = Grammar(tables.load("json", "lexer"))
    g.set_tuning(g.get_tuning()[:4] + [lex_split])
    assert g.lex_int(b"[1]") is not None  # (module loading)
    x = torch.from_numpy(synth.json_doc(n, 16, 77)).cuda()
    out = [torch.empty(n // 4, dtype=t, device="cuda") for t in (torch.int32, torch.int64, torch.int64)]
    L, count, valid = native(), ctypes.c_int64(0), ctypes.c_int(0)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    rc = L.alp_lex_into(g.h, ctypes.c_void_p(x.data_ptr()), ctypes.c_int64(n), *[ctypes.c_void_p(t.data_ptr()) for t in out],
                        ctypes.c_int64(n // 4), ctypes.byref(count), ctypes.byref(valid))
    torch.cuda.synchronize()
    assert rc == 0 and valid.value == 1 and count.value > n // 10
    assert before - torch.cuda.mem_get_info()[0] <= per_byte * n + (8 << 20)
