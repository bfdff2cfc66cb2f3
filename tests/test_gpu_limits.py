"""Calls at the limits of what a context takes: buffers that cannot be had, many items, small budgets.

Bar: such a call is refused or answered exactly, and the calls after it are answered as ever.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from oracle import orc
from ps4b200 import Search, _abi, workloads

pytestmark = pytest.mark.gpu


# 2^40 records of 16 bytes are more than any device has; 2^60 of them leave 64 bits
@pytest.mark.parametrize("room", [1 << 40, 1 << 48, 1 << 60, (1 << 64) - 1])
def test_too_much_room_for_triples_fails_alone(room):
    abc = np.ascontiguousarray(workloads.triples(40, seed=3))
    want = [orc.extend_triple(*(int(v) for v in t), 10 ** 12) for t in abc]
    n = sum(map(len, want))
    with Search(2 * 10 ** 12) as s:
        out = (_abi.TriExt * (n + 1))()
        n_out = C.c_uint64()

        def call(cap):
            return s.lib.ps4_extend_triples(s.ctx, abc.ctypes.data, len(abc), 10 ** 12, None, out, cap,
                                            C.byref(n_out), None)
        assert call(n) == _abi.PS4_OK and n_out.value == n
        assert call(room) == _abi.PS4_ERR_CUDA
        for _ in range(2):
            assert call(n) == _abi.PS4_OK and n_out.value == n
            got = [[] for _ in want]
            for r in out[:n]:
                got[r.item].append(r.d)
            assert got == want
        assert s.range(10 ** 9, 10 ** 9 + 10 ** 5).stats["S_done"] == 10 ** 5
