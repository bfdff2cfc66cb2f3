"""Calls at the limits of what a context takes: buffers that cannot be had, many items, small budgets.

Bar: such a call is refused or answered exactly, and the calls after it are answered as ever.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from conftest import COUNTERS, assert_stats_equal
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


def test_more_than_a_million_items():
    """Items on both sides of 2^20, the others empty: every counter and hit with its own item."""
    n = (1 << 20) + 8
    ranges = {3: (10 ** 9, 10 ** 9 + 400000), 7: (10 ** 6, 10 ** 6 + 5000), (1 << 20) - 1: (5, 900),
              1 << 20: (10 ** 5, 2 * 10 ** 5), (1 << 20) + 3: (15 * 10 ** 8, 15 * 10 ** 8 + 500000),
              (1 << 20) + 7: (1, 70000)}
    lo, hi = np.ones(n, dtype=np.uint64), np.ones(n, dtype=np.uint64)
    for i, (a, b) in ranges.items():
        lo[i], hi[i] = a, b
    as_u64 = C.POINTER(C.c_uint64)
    with Search(2 * 10 ** 9) as s:
        alone = {i: s.range(a, b) for i, (a, b) in ranges.items()}
        stats = (_abi.Stats * n)()
        res = s._res
        assert s.lib.ps4_search_batch(s.ctx, lo.ctypes.data_as(as_u64), hi.ctypes.data_as(as_u64), n, stats,
                                      C.byref(res)) == _abi.PS4_OK
        for i, r in alone.items():
            assert_stats_equal(stats[i].as_dict(), r.stats, label=f"item {i}")
        got = [res.hits[k].item for k in range(res.n_hits)]
        assert sorted(set(got)) == [i for i in sorted(alone) if alone[i].lines]
        other = np.frombuffer(stats, dtype=np.uint64).reshape(n, -1)
        assert sorted(np.flatnonzero(other.any(axis=1))) == sorted(ranges)


# subranges of 1 to 8 tiles, side by side: clusters of one, two and eight CTAs, with fewer subranges than clusters
# and with several rounds of them
@pytest.mark.parametrize("lo,n,w", [(10 ** 6, 20, 30), (10 ** 9, 300, 12000), (10 ** 9, 700, 8192), (10 ** 9, 4000, 8193),
                                    (10 ** 12, 20, 4096), (10 ** 12, 200, 30000), (10 ** 12, 1500, 20001),
                                    (4 * 10 ** 11, 500, 7 * 8192 + 1), (4 * 10 ** 11, 300, 65536)])
def test_batches_of_narrow_subranges_vs_one_range(lo, n, w):
    cuts = [lo + i * w for i in range(n + 1)]
    with Search(2 * 10 ** 12) as s:
        stats, r = s.batch(cuts[:-1], cuts[1:])
        one = s.range(lo, cuts[-1])
    assert r.lines == one.lines
    assert [st["S_done"] for st in stats] == [w] * n
    for k in COUNTERS:
        assert sum(st[k] for st in stats) == one.stats[k], k
    assert max(st["max_reps"] for st in stats) == one.stats["max_reps"]


# items uploaded with their zeros (16), counters landing in the context's own block (31), in one of their own
# (512) and piece by piece (256 each)
@pytest.mark.parametrize("n", [1, 16, 17, 31, 32, 512, 513, 768, 769, 5000])
def test_counters_of_every_item(n):
    los = [10 ** 6 + 997 * i % 10 ** 6 for i in range(n)]
    widths = [i * i % 389 + (i % 7 > 0) for i in range(n)]
    with Search(3 * 10 ** 6) as s:
        for _ in range(2):                               # the second call adds to nothing left from the first
            stats, _ = s.batch(los, [a + w for a, w in zip(los, widths)])
            assert [st["S_done"] for st in stats] == widths
        for i in {0, n // 2, n - 1, 255 % n, 256 % n, 511 % n, 512 % n}:
            assert_stats_equal(stats[i], s.range(los[i], los[i] + widths[i]).stats, label=f"item {i}")
