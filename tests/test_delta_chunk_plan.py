"""The blocks of a delta-rule layer's chunks (on the host; 148 SMs): how many and how wide goes by the entries that are cut into chunks, whatever decodes beside them."""
from __future__ import annotations

import ctypes as C

import pytest

from dnet_b200 import _seqabi


def plan(counts, heads, vdim, sms=148):
    out = (C.c_int32 * 3)()
    _seqabi.check(_seqabi.load().dn_seq_debug_delta_plan(len(counts), (C.c_int32 * len(counts))(*counts), heads, vdim, sms, out))
    return tuple(out)


# 111 blocks of 64 columns of entries of 80 tokens and more fill three quarters of the SMs
@pytest.mark.parametrize("counts,heads,vdim,chunks,pairs,columns", [
    ([2048], 32, 128, 64, 32, 32), ([1, 1, 1, 2048], 32, 128, 64, 32, 32), ([79, 79, 79, 80], 32, 128, 3, 32, 32), ([1] * 63 + [700], 32, 128, 22, 32, 32),
    ([700, 700], 32, 128, 44, 64, 64), ([1, 700, 1, 700], 32, 128, 44, 64, 64), ([81, 80], 28, 128, 6, 56, 64), ([81, 80], 27, 128, 6, 54, 32), ([300, 1], 111, 20, 10, 111, 64)])
def test_entries_that_are_not_cut_neither_count_nor_have_blocks(counts, heads, vdim, chunks, pairs, columns):
    assert plan(counts, heads, vdim) == (chunks, pairs, columns)


def test_bad_arguments_are_refused():
    out = (C.c_int32 * 3)()
    assert _seqabi.load().dn_seq_debug_delta_plan(0, (C.c_int32 * 1)(80), 1, 1, 148, out) < 0
    assert _seqabi.load().dn_seq_debug_delta_plan(1, (C.c_int32 * 1)(80), 1, 1, 148, None) < 0
