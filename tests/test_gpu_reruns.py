"""The re-runs of a search whose lists or queue were too small (ps4_check_reruns makes them so).

Bar: results bit-identical to the same search without them, after the attempts expected.
"""
from __future__ import annotations

import ctypes as C

import pytest

from conftest import assert_stats_equal
from ps4b200 import Ps4Error, Search, _abi, workloads
from ps4b200.serve import Server

pytestmark = pytest.mark.gpu

LO = 10 ** 12
NARROW, WIDE = 300 * 4096 + 7, 700 * 8192 + 7        # below and above one 2^13-S tile for each tile CTA


def attempts(s):
    n, tl = C.c_uint32(), C.c_uint32()
    s.lib.ps4_last_attempts(s.ctx, C.byref(n), C.byref(tl))
    return n.value, tl.value


def same(a, b):
    assert a.lines == b.lines
    assert_stats_equal(a.stats, b.stats)


# a queue that ends within the warps' first stretches, within their first reservations, and later
@pytest.mark.parametrize("queue", [1, 999, 5000, 40000, 200000])
@pytest.mark.parametrize("width", [NARROW, WIDE])
def test_queue_overflow(queue, width):
    with Search(2 * LO) as s:
        want = s.range(LO, LO + width)
        assert attempts(s)[0] == 1
        assert s.lib.ps4_check_reruns(s.ctx, 1, 0, queue, 0) == _abi.PS4_OK
        same(s.range(LO, LO + width), want)
        assert attempts(s)[0] == 2
        same(s.range(LO, LO + width), want)
        assert attempts(s)[0] == 1


def test_queue_overflow_in_a_batch():
    los, his = workloads.subranges(40, seed=8, wmax=2e6, omax=1e12)
    los, his = los.tolist(), his.tolist()
    with Search(2 * LO) as s:
        want = s.batch(los, his)
        s.lib.ps4_check_reruns(s.ctx, 2, 0, 30000, 0)
        got = s.batch(los, his)
        assert attempts(s)[0] == 3
    assert got[0] == want[0] and got[1].lines == want[1].lines and got[1].items == want[1].items


# lists that hold nothing, less than a part of a list, less than most tiles have, and about what they have
@pytest.mark.parametrize("list_", [1, 150, 1500, 3200])
@pytest.mark.parametrize("kernel,width", [("batched", NARROW), ("batched", WIDE), ("persist", WIDE)])
def test_tiles_whose_list_overflows_scan_for_themselves(kernel, width, list_):
    with Search(2 * LO, kernel=kernel) as s:
        want = s.range(LO, LO + width)
        s.lib.ps4_check_reruns(s.ctx, 1, list_, 0, 0)
        same(s.range(LO, LO + width), want)
        assert attempts(s)[0] == 1


TILE, EXTLIST, QUEUE = 100, 101, 102


# attempts that end with a code, and the S per tile (log2) of the attempt that is kept: a narrow call goes from
# 2^12 to the context's 2^13, and from there, as a wide one, back to 2^12
@pytest.mark.parametrize("width,code,n,tile", [
    (NARROW, 0, 1, 12), (NARROW, TILE, 1, 13), (NARROW, TILE, 2, 12), (NARROW, EXTLIST, 1, 13), (NARROW, QUEUE, 3, 12),
    (WIDE, 0, 1, 13), (WIDE, TILE, 1, 12), (WIDE, EXTLIST, 1, 13), (WIDE, QUEUE, 2, 13)])
def test_codes(width, code, n, tile):
    with Search(2 * LO) as s:
        want = s.range(LO, LO + width)
        s.lib.ps4_check_reruns(s.ctx, n, 0, 0, code)
        same(s.range(LO, LO + width), want)
        assert attempts(s) == (n + 1 if code else 1, tile)


@pytest.mark.parametrize("step_S", [1 << 20, 1 << 23])          # steps of fewer and of more tiles than tile CTAs
@pytest.mark.parametrize("list_,queue,code,reruns", [(100, 0, 0, 0), (0, 3000, 0, 2), (0, 0, TILE, 1), (0, 0, EXTLIST, 1)])
def test_server_steps(step_S, list_, queue, code, reruns):
    ranges = [(LO - 3 * 10 ** 6, LO), (10 ** 9, 10 ** 9 + 7 * 10 ** 6 + 1), (1, 50000)]
    with Search(2 * LO) as s:
        want = [s.range(a, b) for a, b in ranges]
        with Server(s, hbm_budget=1 << 30, step_S=step_S) as srv:
            s.lib.ps4_check_reruns(s.ctx, max(reruns, 1), list_, queue, code)
            for i, (a, b) in enumerate(ranges):
                srv.submit_range(i, a, b)
            done = []
            while len(done) < len(ranges):
                done += srv.progress(100000)
            got = [srv.take_range(i) for i in range(len(ranges))]
            assert srv.info()["step_reruns"] == reruns
    for a, b in zip(got, want):
        same(a, b)


@pytest.mark.parametrize("width", [4097, NARROW, WIDE])
@pytest.mark.parametrize("tile", [12, 13, 14])
def test_a_tile_size_asked_for_is_kept(width, tile):
    with Search(2 * LO) as s:
        want = s.range(LO, LO + width)
    with Search(2 * LO, log2_tile=tile) as s:
        same(s.range(LO, LO + width), want)
        assert attempts(s) == (1, tile)
        s.lib.ps4_check_reruns(s.ctx, 1, 0, 0, TILE)
        if tile > 12:
            same(s.range(LO, LO + width), want)
            assert attempts(s) == (2, tile - 1)
        else:
            with pytest.raises(Ps4Error) as e:
                s.range(LO, LO + width)
            assert "tile capacity exceeded" in e.value.message and attempts(s) == (1, 12)


def test_the_tuner_times_the_tiles_it_names():
    with Search(2 * LO) as s:
        t = s.autotune([LO], [LO + NARROW], budget_s=1e-9)       # the first candidate only
        assert (t["log2_tile"], attempts(s)) == (14, (1, 14))
        s.range(LO, LO + NARROW)
        assert attempts(s) == (1, 12)


def test_arguments():
    with Search(10 ** 6) as s:
        assert s.lib.ps4_check_reruns(s.ctx, 1, 0, 0, 99) == _abi.PS4_ERR_ARG
        assert s.lib.ps4_check_reruns(None, 1, 0, 0, 0) == _abi.PS4_ERR_ARG
        assert s.range(1, 1000).stats["S_done"] == 999 and attempts(s)[0] == 1
