"""A parse whose scratch passes 1 GiB gives the device its memory back: once
the tables are freed, at most 1 GiB stays with the context's pool."""
import ctypes as C

import pytest
import torch

from gexs_b200 import Context, synth, _capi as capi
from gexs_b200._capi import check, lib

pytestmark = pytest.mark.gpu

GIB = 1 << 30
SLACK = 128 << 20          # modules loaded by the first parse, page rounding


def _kept(parse):
    torch.cuda.empty_cache()
    ctx = Context(0)
    parse(ctx, 1)                                          # loads the kernels
    before = torch.cuda.mem_get_info()[0]
    parse(ctx, None)
    return before - torch.cuda.mem_get_info()[0]


def test_hitran_scratch_is_given_back():
    part = synth.make_hitran_par(20000, 91)
    text = part * (GIB // len(part) + 1)

    def parse(ctx, small):
        t = part if small else text
        table = capi.GexsLineTable()
        check(lib().gexs_hitran_parse(ctx.h, t, len(t), 1.0, 1.0, 1.0, 1, C.byref(table)), "parse")
        assert table.count > 0
        lib().gexs_line_table_free(C.byref(table))

    assert _kept(parse) <= GIB + SLACK


def test_exomol_scratch_is_given_back():
    st = synth.make_states(5000, 40, 92)
    up, low, a = synth.make_exomol_transitions(st, 20000, 100.0, 9000.0, 93)
    states = synth.exomol_states_text(st)
    part = synth.exomol_trans_text(up, low, a)
    text = part * (GIB // 2 // len(part) + 1)

    def parse(ctx, small):
        t = part if small else text
        s, table = capi.GexsStateTable(), capi.GexsLineTable()
        check(lib().gexs_exomol_parse_states(ctx.h, states, len(states), C.byref(s)), "states")
        check(lib().gexs_exomol_parse_trans(ctx.h, C.byref(s), t, len(t), None, 0,
                                            capi.BROAD_DEFAULTS, 0.1, 0.5, 1, C.byref(table)),
              "trans")
        assert table.count > 0
        lib().gexs_line_table_free(C.byref(table))
        lib().gexs_state_table_free(C.byref(s))

    assert _kept(parse) <= GIB + SLACK
