"""The work that users of this framework have it do, as measurable cases.

Every case goes through the package's public calls (``Search.range``, ``Search.batch``,
``Search.extend_triples``, ``serve.Server``) on an open context, takes host inputs and returns
host results, as a program that uses the package does.  ``prepare`` opens the context (and the
server), whose factor tables a program keeps between calls; ``run`` is one whole call with its
result lines.  A case's seed moves its interval, its items or its requests.
"""
from __future__ import annotations

import math
import sys
from itertools import combinations
from pathlib import Path

import numpy as np

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "pairwise-square-sums_b200"))

from ps4b200 import Search, workloads  # noqa: E402
from ps4b200.serve import Server  # noqa: E402

S_LIMIT = 1 << 44                     # the largest S a context can be opened for
FOUND = ("S_done", "pairs", "S_ge3", "triples", "sets4", "max_reps")
SEARCHED = ("sets5", "sets6", "multi", "ext_cand", "ext_sqrt", "max_divisors", "max_extensions")


def listed() -> list:
    return [
        # one narrow query on a wide context, as a service answers it: latency and launches
        {"name": "range 2e4 at 4e11", "kind": "range", "lo": 4 * 10**11, "width": 20011, "limit": 10**12 + 10**9,
         "verify": False, "noext": False},
        # a short check of an interval, as the smoke run does it
        {"name": "range 2e6 at 1e9", "kind": "range", "lo": 10**9, "width": 2 * 10**6, "limit": 2 * 10**9,
         "verify": False, "noext": False},
        # every S below a bound, as the drop-in CLI runs it: a first look, with the roots verified ...
        {"name": "bound 1e7 verified", "kind": "bound", "bound": 10**7, "verify": True, "noext": False},
        # ... the middle size, without the extension step (4-sets only) ...
        {"name": "bound 3e8 noext", "kind": "bound", "bound": 3 * 10**8, "verify": False, "noext": True},
        # ... and the headline search
        {"name": "bound 1e10", "kind": "bound", "bound": 10**10, "verify": False, "noext": False},
        # a block of the kind the block controller hands out
        {"name": "block 2e8 at 1e12", "kind": "range", "lo": 10**12, "width": 2 * 10**8, "limit": 2 * 10**12,
         "verify": False, "noext": False},
        # a block at the search's frontier, near the largest S supported
        {"name": "block 3e7 at 1.2e13", "kind": "range", "lo": 12 * 10**12, "width": 3 * 10**7 + 77,
         "limit": S_LIMIT, "verify": True, "noext": False},
        # uneven subranges in one call: wide ones ...
        {"name": "batch 64 uneven", "kind": "batch", "items": 64, "wmin": 10**5, "wmax": 10**8, "omax": 10**11,
         "limit": 2 * 10**11},
        # ... and many narrow ones
        {"name": "batch 300 narrow", "kind": "batch", "items": 300, "wmin": 10**3, "wmax": 6 * 10**5,
         "omax": 10**12, "limit": 2 * 10**12},
        # square-sum triples extended to 4-sets: a handful, and a large batch
        {"name": "triples 50", "kind": "triples", "n": 50, "xmax": 10**5, "dmax": 10**12, "limit": 2 * 10**12},
        {"name": "triples 1e5", "kind": "triples", "n": 10**5, "xmax": 10**5, "dmax": 10**12, "limit": 2 * 10**12},
        # the serving loop: a burst of mixed requests, every answer collected
        {"name": "serve 150 mixed", "kind": "serve", "n": 150, "wmin": 10**4, "wmax": 3 * 10**7, "omax": 10**12},
    ]


def _log(rng, a, b) -> int:
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng) -> dict:
    kind = rng.choice(["range", "range", "range", "bound", "bound", "batch", "batch", "triples", "triples", "serve"])
    flags = {"verify": rng.random() < 0.3, "noext": rng.random() < 0.15}
    if kind == "range":
        width = _log(rng, 10**4, 10**9)
        lo = _log(rng, 10**9, 13 * 10**12)
        # the densest S cost about three times S near 1e10
        width = min(width, 3 * 10**8 if lo > 10**12 else 10**9)
        limit = rng.choice([lo + width + 10**6, max(2 * 10**12, lo + width + 10**6), S_LIMIT])
        return {"kind": "range", "lo": lo, "width": width, "limit": limit, **flags}
    if kind == "bound":
        return {"kind": "bound", "bound": _log(rng, 10**6, 5 * 10**9), **flags}
    if kind == "batch":
        items = _log(rng, 8, 512)
        wmax = _log(rng, 3 * 10**5, max(4 * 10**5, min(10**9, 10**10 // items)))
        return {"kind": "batch", "items": items, "wmin": rng.choice([10**3, 10**4, 10**5]), "wmax": wmax,
                "omax": _log(rng, 10**10, 10**12), "limit": 2 * 10**12}
    if kind == "triples":
        return {"kind": "triples", "n": _log(rng, 1, 10**5), "xmax": _log(rng, 10**4, 3 * 10**5),
                "dmax": _log(rng, 10**9, 10**15), "limit": 2 * 10**12}
    return {"kind": "serve", "n": _log(rng, 20, 300), "wmin": 10**4, "wmax": _log(rng, 10**6, 5 * 10**7),
            "omax": 10**12}


# ------------------------------------------------------------------ inputs

def _interval(case: dict, seed: int):
    """[lo, hi) of a single search: the seed moves an interval, or lowers a bound a little."""
    rng = np.random.default_rng([seed, 17])
    if case["kind"] == "bound":
        return 1, case["bound"] - int(rng.integers(0, case["bound"] // 1000 + 1))
    lo = case["lo"] + int(rng.integers(0, 10**6))
    return lo, min(lo + case["width"], case["limit"])


def _limit(case: dict) -> int:
    if case["kind"] == "serve":
        return case["omax"] + 10**9 + 1
    return case["bound"] if case["kind"] == "bound" else case["limit"]


class _State:
    """An open context (and server), its inputs, and room for nothing else."""

    def __init__(self, case: dict, seed: int):
        kind = case["kind"]
        self.kind = kind
        self.search = Search(_limit(case), verify=case.get("verify", False), noext=case.get("noext", False))
        self.server = None
        # S of a pass, the same for every seed, for the sizes of its outputs
        if kind in ("range", "bound"):
            self.lo, self.hi = _interval(case, seed)
            self.width = case["bound"] if kind == "bound" else case["width"]
        elif kind == "batch":
            lo, hi = workloads.subranges(case["items"], seed, wmin=case["wmin"], wmax=case["wmax"], omax=case["omax"])
            self.lo, self.hi = lo.tolist(), np.minimum(hi, np.uint64(case["limit"])).tolist()
            self.width = case["items"] * case["wmax"] // 2
        elif kind == "triples":
            self.abc = workloads.triples(case["n"], seed, xmax=case["xmax"])
            self.dmax = case["dmax"]
        else:
            self.reqs = workloads.requests(case["n"], seed, rate=1000.0, wmin=case["wmin"], wmax=case["wmax"],
                                           omax=case["omax"])
            self.width = case["n"] * case["wmax"] // 2
            self.server = Server(self.search, hbm_budget=4 << 30)

    def __del__(self):
        if getattr(self, "server", None) is not None:
            self.server.close()
        if getattr(self, "search", None) is not None:
            self.search.close()


def prepare(case: dict, seed: int):
    return _State(case, seed)


# ------------------------------------------------------------------ one pass

def _counters(stats: dict) -> dict:
    hist = np.zeros(100, dtype=np.int64)
    for k, v in stats["hist5"].items():
        hist[k] = v
    return {"found": np.array([stats[k] for k in FOUND], dtype=np.int64),
            "searched": np.array([stats[k] for k in SEARCHED], dtype=np.int64), "hist5": hist}


def _padded(a: np.ndarray, room: int, fill: int = 0) -> np.ndarray:
    """The records at the front of an array whose size the case sets, whatever the seed finds."""
    if len(a) > room:
        raise ValueError(f"{len(a)} values, room for {room}")
    out = np.zeros(room, dtype=a.dtype) if fill == 0 else np.full(room, fill, dtype=a.dtype)
    out[:len(a)] = a
    return out


def _text(lines, width: float) -> np.ndarray:
    """The result lines of a pass over `width` S as bytes, zero behind the last one (a line has about
    100 bytes, and S yield one per 1e5 at most)."""
    return _padded(np.frombuffer("".join(lines).encode(), dtype=np.uint8), 65536 + int(1e-3 * width))


def run(state):
    s = state.search
    if state.kind in ("range", "bound"):
        r = s.range(state.lo, state.hi)
        return {**_counters(r.stats), "text": _text(r.lines + r.six_lines, state.width)}
    if state.kind == "batch":
        stats, r = s.batch(state.lo, state.hi)
        per = [_counters(x) for x in stats]
        return {**{k: np.stack([p[k] for p in per]) for k in per[0]}, "text": _text(r.lines + r.six_lines, state.width),
                "items": _padded(np.array(r.items, dtype=np.int64), 4096 + int(2e-5 * state.width), -1)}
    if state.kind == "triples":
        recs, bad, stats = s.extend_triples(state.abc, state.dmax, as_lists=False)
        room = 1024 + len(state.abc)
        return {"d": _padded(recs["d"].astype(np.int64), room),
                "item": _padded(recs["item"].astype(np.int64), room, -1), "state": bad,
                "searched": np.array([stats["ext_cand"], stats["ext_sqrt"]], dtype=np.int64)}
    # serving: everything submitted at once, answers taken as they finish
    srv, out = state.server, {}
    kinds = {q.rid: q.kind for q in state.reqs}
    for q in state.reqs:
        if q.kind == "range":
            srv.submit_range(q.rid, q.lo, q.hi)
        else:
            srv.submit_triple(q.rid, q.abc, q.dmax)
    while len(out) < len(state.reqs):
        for d in srv.progress(2000):
            rid = d["tag"]
            out[rid] = srv.take_range(rid) if kinds[rid] == "range" else srv.take_triple(rid)
    n = len(state.reqs)
    res = {"found": np.zeros((n, len(FOUND)), dtype=np.int64), "searched": np.zeros((n, len(SEARCHED)), dtype=np.int64),
           "hist5": np.zeros((n, 100), dtype=np.int64), "lines": np.zeros(n, dtype=np.int64),
           "triple": np.zeros((n, 4), dtype=np.int64)}
    text, ds = [], []
    for i, q in enumerate(state.reqs):
        a = out[q.rid]
        if q.kind == "range":
            for k, v in _counters(a.stats).items():
                res[k][i] = v
            res["lines"][i] = len(a.lines) + len(a.six_lines)
            text += a.lines + a.six_lines
        else:
            res["triple"][i] = (len(a[0]), a[1], a[2]["ext_cand"], a[2]["ext_sqrt"])
            ds += a[0]
    res["text"] = _text(text, state.width)
    res["d"] = _padded(np.array(ds, dtype=np.int64), 1024 + n)
    return res


# ------------------------------------------------------------------ the work of one pass

# Per S, what the search's own counters say at a few S (a straight line over log10 S between
# them): representations, representation triples, 4-sets, divisor-pair candidates, exact tests.
DENSITY = ((6, (0.39, 0.14, 0.023, 0.20, 0.05)), (9, (0.39, 0.60, 0.105, 2.18, 0.49)),
           (10, (0.39, 0.90, 0.14, 3.5, 0.85)), (11, (0.39, 1.28, 0.20, 5.9, 1.46)),
           (12, (0.39, 1.71, 0.272, 10.2, 2.64)), (13, (0.39, 2.2, 0.33, 14.5, 3.8)))
# 32-bit lane operations of one such event, at least
OPS = (5, 24, 80, 28, 80)


def _ops_per_S(S: float, noext: bool) -> float:
    x = min(max(math.log10(max(S, 1.0)), DENSITY[0][0]), DENSITY[-1][0])
    for (a, u), (b, v) in zip(DENSITY, DENSITY[1:]):
        if x <= b:
            d = [p + (q - p) * (x - a) / (b - a) for p, q in zip(u, v)]
            break
    return sum(o * n for o, n in zip(OPS[:2] if noext else OPS, d))


def work(case: dict) -> dict:
    """Bytes a pass takes in and gives back (intervals or triples, counter blocks, records and
    their lines), and its integer operations counted as flops."""
    kind = case["kind"]
    record, counters = 160.0, 113 * 8
    if kind == "bound":
        b = float(case["bound"])
        ops = b * _ops_per_S(b / 2, case["noext"])
        return {"bytes": 16 + counters + (0 if case["noext"] else 5.4e-6 * b * record), "flops": ops}
    if kind == "range":
        w = float(case["width"])
        return {"bytes": 16 + counters + (0 if case["noext"] else 2e-6 * w * record),
                "flops": w * _ops_per_S(case["lo"], case["noext"])}
    if kind == "triples":
        return {"bytes": case["n"] * 25.0, "flops": case["n"] * (300.0 + 11 * 28)}
    mean_w = (case["wmax"] - case["wmin"]) / math.log(case["wmax"] / case["wmin"])
    n = case["items"] if kind == "batch" else 0.7 * case["n"]
    tri = 0 if kind == "batch" else 0.3 * case["n"]
    return {"bytes": n * (16 + counters + 2e-6 * mean_w * record) + tri * 60.0,
            "flops": n * mean_w * _ops_per_S(case["omax"] / 2, False) + tri * 608.0}


# ------------------------------------------------------------------ exact values, in numpy

def _found(lo: int, hi: int) -> np.ndarray:
    """The FOUND counters of S in [lo, hi): representations S = p^2 + q^2 with 1 <= p <= q, the S
    with three or more (S not 2 mod 4), their triples, and the 4-sets of positive integers that
    the triples give: for p_x < p_y < p_z (P their squares), with c + d = P_x, b + d = P_y, and a + d =
    q_z^2 or p_z^2, the four members are positive integers in the first case when the p sum to an even
    number and P_z < P_x + P_y, in the second when the sum's parity is S's and P_z > S - P_x - P_y
    (and q_z != p_z)."""
    ss, ps = [], []
    q = np.arange(max(1, math.isqrt((lo + 1) // 2) - 1), math.isqrt(hi) + 1, dtype=np.int64)
    q2 = q * q
    p0 = np.sqrt(np.maximum(lo - q2, 1).astype(np.float64)).astype(np.int64) - 1
    p0 = np.maximum(p0, 1)
    p1 = np.minimum(q, np.sqrt(np.maximum(hi - q2, 0).astype(np.float64)).astype(np.int64) + 1)
    for step in range(int(np.max(p1 - p0)) + 1):
        p = p0 + step
        s = p * p + q2
        ok = (p <= p1) & (p <= q) & (s >= lo) & (s < hi)
        ss.append(s[ok])
        ps.append(p[ok])
        live = p <= p1
        if not live.all():
            q, q2, p0, p1 = q[live], q2[live], p0[live], p1[live]
        if not len(q):
            break
    ss, ps = np.concatenate(ss), np.concatenate(ps)
    order = np.lexsort((ps, ss))
    ss, ps = ss[order], ps[order]
    S, start, k = np.unique(ss, return_index=True, return_counts=True)
    sel = (k >= 3) & (S % 4 != 2)
    sets = 0
    for kk in np.unique(k[sel]):
        rows = sel & (k == kk)
        P = ps[start[rows][:, None] + np.arange(kk)[None, :]]
        Sv = S[rows]
        xyz = np.array(list(combinations(range(int(kk)), 3)))
        for part in np.array_split(np.arange(len(Sv)), max(1, len(Sv) * len(xyz) // 2_000_000)):
            a, b, c = (P[part][:, xyz[:, i]] for i in range(3))
            s = Sv[part][:, None]
            A, B, Z = a * a, b * b, c * c
            par = (a + b + c) & 1
            sets += int(((par == 0) & (Z < A + B)).sum())
            sets += int(((par == (s & 1)) & (2 * Z != s) & (Z > s - A - B)).sum())
    ks = k[sel].astype(object)
    return np.array([hi - lo, len(ss), int(sel.sum()), int(sum(x * (x - 1) * (x - 2) // 6 for x in ks)), sets,
                     int(k.max()) if len(k) else 0], dtype=np.int64)


def _extensions(abc, dmax: int):
    """Every (d, row) with 0 < d <= dmax, d not in the row, and d + a, d + b, d + c all squares."""
    ds, items = [], []
    for i, (a, b, c) in enumerate(sorted(int(v) for v in row) for row in abc):
        u = np.arange(math.isqrt(c) + 1, math.isqrt(dmax + c) + 1, dtype=np.int64)
        d = u * u - c
        for m in (a, b):
            w = np.rint(np.sqrt((d + m).astype(np.float64))).astype(np.int64)
            d = d[w * w == d + m]
        d = np.sort(d[(d <= dmax) & (d != a) & (d != b) & (d != c)])
        ds.append(d)
        items.append(np.full(len(d), i, dtype=np.int64))
    return np.concatenate(ds), np.concatenate(items)


def exact(case: dict, seed: int):
    """What the counters of the enumeration and the triples' extensions are, for sizes that numpy
    does in seconds; the rest has no value here."""
    if case["kind"] in ("range", "bound"):
        lo, hi = _interval(case, seed)
        if hi - lo > 10**7:
            return None
        return {"found": _found(lo, hi), "searched": None, "hist5": None, "text": None}
    if case["kind"] == "triples" and case["n"] * math.isqrt(case["dmax"]) <= 10**8:
        d, item = _extensions(workloads.triples(case["n"], seed, xmax=case["xmax"]), case["dmax"])
        room = 1024 + case["n"]
        return {"d": _padded(d, room), "item": _padded(item, room, -1), "state": None, "searched": None}
    return None
