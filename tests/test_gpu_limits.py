"""Calls at the limits of what a context takes: buffers that cannot be had, many items, small budgets.

Bar: such a call is refused or answered exactly, and the calls after it are answered as ever.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from conftest import assert_stats_equal
from oracle import orc
from ps4b200 import Search, _abi, workloads
from ps4b200.serve import Server

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


# A server's buffers besides its arena: 24 bytes for each of 2^20 queued 4-sets, 310 MB of tile lists, 6 MB of
# step buffers and 16 MB of arena at least.
@pytest.mark.parametrize("budget", [364 << 20, 512 << 20])
def test_server_on_a_small_budget(budget):
    ranges = [(10 ** 9, 10 ** 9 + 3 * 10 ** 5), (10 ** 12 - 70001, 10 ** 12), (1, 4097)]
    with Search(2 * 10 ** 12) as s:
        with Server(s, hbm_budget=budget, max_slots=4, max_step_items=64, step_S=1 << 20, max_step_triples=16) as srv:
            assert srv.info()["device_bytes"] <= budget
            for i, (lo, hi) in enumerate(ranges):
                srv.submit_range(i, lo, hi)
            done = []
            while len(done) < len(ranges):
                done += srv.progress(100000)
            got = [srv.take_range(i) for i in range(len(ranges))]
        for (lo, hi), r in zip(ranges, got):
            want = s.range(lo, hi)
            assert r.lines == want.lines
            assert_stats_equal(r.stats, want.stats)
