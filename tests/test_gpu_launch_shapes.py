"""The launch shapes of the two-kernel pipeline: narrow calls (smaller tiles, clusters of eight
tile CTAs sharing one scan, few 4-sets per engine warp) and the sizes where the shape changes.

Bar: bit-exact against the oracle for narrow calls, and against the same range cut in two (other
tiles, other groups) where a call fills the device.
"""
from __future__ import annotations

import pytest

from conftest import COUNTERS, assert_stats_equal
from oracle import orc
from ps4b200 import Search, workloads

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def wide():
    with Search(1 << 44) as s:
        yield s


@pytest.mark.parametrize("lo", [1, 10 ** 6 + 7, 10 ** 9, 4 * 10 ** 11 + 1, 12 * 10 ** 12 + 5])
@pytest.mark.parametrize("width", [1, 4095, 4097, 8 * 4096 + 1, 70001])
def test_narrow_calls_vs_oracle(wide, lo, width):
    r = wide.range(lo, lo + width)
    rc, ost, olines, err = orc.search(lo, lo + width)
    assert rc == 0, err
    assert sorted(r.lines) == sorted(olines)
    assert_stats_equal(r.stats, ost)


# 128 tiles of 2^12 S (CTAs of 1024 threads up to there); 592 tile CTAs: one tile of 2^13 S each and a
# little less or more; several groups per cluster
@pytest.mark.parametrize("lo", [1, 10 ** 9, 10 ** 12])
@pytest.mark.parametrize("width", [128 * 4096, 128 * 4096 + 1, 592 * 8192 - 1, 592 * 8192 + 1, 592 * 3 * 8192 + 4097])
def test_shape_changes_vs_split_calls(wide, lo, width):
    one = wide.range(lo, lo + width)
    cut = lo + width // 3 + 1
    a, b = wide.range(lo, cut), wide.range(cut, lo + width)
    assert one.lines == a.lines + b.lines
    for k in COUNTERS:
        assert one.stats[k] == a.stats[k] + b.stats[k], k


# S with 3 .. 288 representations, odd, = 4 and = 0 mod 8 (among these some twice a square, whose last
# representation has p = q): the list lengths at which the tile kernel's sort changes its way, and the
# lengths of its searches
LISTS = {3: (15317, 61268), 4: (80401, 643208), 5: (33125, 132500), 7: (180625, 1445000), 8: (2331629, 18653032),
         9: (2588573, 10354292), 13: (1221025, 9768200), 16: (39637693, 317101544), 31: (763140625, 6105125000),
         32: (515290009, 4122320072), 36: (3926865241, 31414921928), 63: (40446453125, 323571625000),
         64: (87084011521, 696672092168), 96: (1480428195857, 11843425566856), 192: (8708401152100, 17416802304200),
         288: (14234886498625,)}


@pytest.mark.parametrize("k", sorted(LISTS))
def test_list_lengths_vs_oracle(wide, k):
    for S in LISTS[k]:
        r = wide.range(S, S + 1)
        rc, ost, olines, err = orc.search(S, S + 1)
        assert rc == 0, err
        assert ost["max_reps"] in (k, k + 1)          # one more for twice a square
        assert sorted(r.lines) == sorted(olines)
        assert_stats_equal(r.stats, ost)


@pytest.mark.parametrize("S0", [4205, 5785, 6205])
def test_differences_with_a_large_square_vs_oracle(wide, S0):
    """4-sets that are 49999^2 times a small one: both factors of their differences share a large prime,
    so that divisor lists would leave 32 bits and the per-lane divisor walk takes over."""
    S = S0 * 49999 ** 2
    r = wide.range(S, S + 1)
    rc, ost, olines, err = orc.search(S, S + 1)
    assert rc == 0 and ost["sets4"] > 0, err
    assert sorted(r.lines) == sorted(olines)
    assert_stats_equal(r.stats, ost)


@pytest.mark.parametrize("kernel,n", [("batched", 33), ("batched", 120000), ("persist", 4000)])
def test_many_divisor_walks_vs_single_calls(wide, kernel, n):
    """The same 4-sets for the per-lane walk, one item each: more than 32 per engine warp at 120000 (the walks
    of several rounds are gathered), of different items, each counted with its own."""
    S = [S0 * 49999 ** 2 for S0 in (4205, 5785, 6205)]
    alone = [wide.range(s, s + 1).stats for s in S]
    lo = [S[i * i % 7 % 3] for i in range(n)]
    with Search(1 << 44, kernel=kernel) as s:
        stats, r = s.batch(lo, [x + 1 for x in lo])
    assert not r.lines
    for x, st in zip(lo, stats):
        assert all(st[k] == alone[S.index(x)][k] for k in COUNTERS), x


@pytest.mark.parametrize("n", [1, 2, 31, 33, 4736, 4737, 9473])
@pytest.mark.parametrize("scale", [1, 65537 ** 2])
def test_triple_counts_and_scales_vs_oracle(wide, n, scale):
    """One triple per warp up to a full device, then several; scaled ones share a large prime (as above)."""
    abc = workloads.triples(n, seed=n, xmax=40 if scale > 1 else 2000) * scale
    got, state, st = wide.extend_triples(abc, 10 ** 15)
    assert not state.any() and st["triples"] == n
    check = range(n) if n < 100 else range(0, n, 97)
    for i in check:
        assert got[i] == orc.extend_triple(*(int(v) for v in abc[i]), 10 ** 15), i
