"""The blocks of a delta-rule layer's chunks (on the host; 148 SMs): how many and how wide goes by the entries that are cut into chunks, whatever decodes beside them."""
from __future__ import annotations

import ctypes as C

import pytest

from dnet_b200 import _seqabi


def plan(counts, heads, vdim, dim=128, sms=148):
    out = (C.c_int32 * 3)()
    _seqabi.check(_seqabi.load().dn_seq_debug_delta_plan(len(counts), (C.c_int32 * len(counts))(*counts), heads, dim, vdim, sms, out))
    return tuple(out)


# 111 blocks of 64 columns of entries that are cut, 96 tokens and more with keys of 128, fill three quarters of the SMs
@pytest.mark.parametrize("counts,heads,vdim,chunks,pairs,columns", [
    ([2048], 32, 128, 64, 32, 32), ([1, 1, 1, 2048], 32, 128, 64, 32, 32), ([95, 95, 95, 96], 32, 128, 3, 32, 32), ([1] * 63 + [700], 32, 128, 22, 32, 32),
    ([700, 700], 32, 128, 44, 64, 64), ([1, 700, 1, 700], 32, 128, 44, 64, 64), ([97, 96], 28, 128, 7, 56, 64), ([97, 96], 27, 128, 7, 54, 32), ([300, 1], 111, 20, 10, 111, 64)])
def test_entries_that_are_not_cut_neither_count_nor_have_blocks(counts, heads, vdim, chunks, pairs, columns):
    assert plan(counts, heads, vdim) == (chunks, pairs, columns)


def test_no_entries_are_cut_where_chunks_are_slower():
    """Keys of 64: six entries of 32 heads and 80 or 112 tokens take 33 and 45 us token by token, 38 and 49 in chunks; three of 80 tokens with keys of 128 46 and 50."""
    assert plan([80] * 6 + [112] * 6 + [127], 32, 64, dim=64)[0] == 0 and plan([128], 32, 64, dim=64)[0] == 4
    assert plan([80] * 3 + [95], 32, 128)[0] == 0 and plan([96], 32, 128)[0] == 3


def test_bad_arguments_are_refused():
    out, run = (C.c_int32 * 3)(), _seqabi.load().dn_seq_debug_delta_plan
    assert run(0, (C.c_int32 * 1)(96), 1, 128, 1, 148, out) < 0
    assert run(1, (C.c_int32 * 1)(96), 1, 128, 1, 148, None) < 0
    assert run(1, (C.c_int32 * 1)(96), 1, 96, 1, 148, out) < 0
