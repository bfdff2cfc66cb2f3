"""Single steps of the search kernels, called directly on inputs that whole searches seldom or
never meet: the walk over representation pairs, and the roots of the hot paths -- the square test of the
extension engine and the triple kernel, the first p of the tile scan and the decoding of a pair number,
each a single-precision estimate and a correction.  (The exact roots behind the other paths:
test_gpu_roots.py.)

Bar: bit-exact against exact integer arithmetic on the host.
"""
from __future__ import annotations

import ctypes as C
import math
import random
from itertools import accumulate

import pytest

from ps4b200 import _abi

pytestmark = pytest.mark.gpu


# pairs per list, in order: lists of three representations have one pair (runs of them are what a window of
# 32 lists is least enough for), four have three, up to 288 representations
def pair_counts():
    yield [1]
    yield [1] * 31
    yield [1] * 32
    yield [1] * 33
    yield [1] * 1000
    for lead in (1, 2, 31, 32, 33, 63, 64, 65):       # a list that ends within, at and after a step's end
        yield [lead] + [1] * 97 + [3]
    yield [287 * 286 // 2, 1, 1, 287 * 286 // 2] + [1] * 40
    rng = random.Random(5)
    for share in (0.5, 0.9, 0.99):
        yield [1 if rng.random() < share else rng.choice((3, 6, 10, 21, 105, 1953)) for _ in range(600)]


@pytest.mark.parametrize("counts", list(pair_counts()), ids=lambda c: f"{len(c)}-lists-{sum(c)}-pairs")
def test_owner_of_every_pair(counts):
    first = list(accumulate(counts, initial=0))
    n, total = len(counts), first[-1]
    owner = (C.c_uint64 * total)()
    lib = _abi.load()
    assert lib.ps4_check_pair_owners(0, (C.c_uint32 * (n + 1))(*first), n, owner) == _abi.PS4_OK
    want = [first[i] << 32 | i for i in range(n) for _ in range(counts[i])]
    assert list(owner) == want


def test_pair_owner_arguments():
    lib = _abi.load()
    out = (C.c_uint64 * 4)()
    for first in ([1, 2], [0, 0], [0, 2, 2], [0, (1 << 24) + 1]):
        assert lib.ps4_check_pair_owners(0, (C.c_uint32 * len(first))(*first), len(first) - 1, out) == _abi.PS4_ERR_ARG


def fast_roots(which, pairs):
    lib = _abi.load()
    n = len(pairs)
    a = (C.c_uint64 * n)(*[x for x, _ in pairs])
    b = (C.c_uint64 * n)(*[y & (2 ** 64 - 1) for _, y in pairs])
    out = (C.c_uint64 * n)()
    assert lib.ps4_check_fast_roots(0, which, a, b, n, out) == _abi.PS4_OK
    return list(out)


LIM = 1 << 44                                     # u, |d| and S0 below it


def roots_near(top):
    """Numbers up to `top`: small ones, powers of two and their neighbours, random ones of each size."""
    rng = random.Random(11)
    vals = set(range(1, 40)) | {top, top - 1, top - 2}
    for b in range(1, top.bit_length() + 1):
        vals |= {(1 << b) + d for d in (-2, -1, 0, 1, 2)}
        vals |= {rng.getrandbits(b) for _ in range(60)}
    return sorted(v for v in vals if 1 <= v <= top)


def test_square_test_at_its_edges():
    """u^2 + d = s^2 - 1, s^2, s^2 + 1 for s from 1 to 2^44 and u as near and as far as |d| < 2^44 allows."""
    rng = random.Random(12)
    pairs = []
    for s in roots_near(LIM - 1):
        far = LIM // (2 * s + 2)
        us = {s, s - 1, s + 1, s - far, s + far, math.isqrt(max(s * s - LIM, 0)) + 1, math.isqrt(s * s + LIM - 2)}
        us |= {max(1, s + rng.randint(-far, far)) for _ in range(6)}
        pairs += [(u, s * s + e - u * u) for u in us if 1 <= u < LIM for e in (-1, 0, 1)
                  if abs(s * s + e - u * u) < LIM and s * s + e > 0]
    got = fast_roots(0, pairs)
    assert len(pairs) > 50000
    for (u, d), g in zip(pairs, got):
        n = u * u + d
        assert g == (math.isqrt(n) ** 2 == n), (u, d)


def test_first_representation_at_its_edges():
    """S0 - q^2 = r^2 - 1, r^2, r^2 + 1 for r up to q, and q about sqrt(S0/2) and sqrt(S0), to S0 near 2^44."""
    rng = random.Random(13)
    cases = set()
    for q in roots_near(math.isqrt(LIM)):
        for r in {0, 1, 2, q // 2, q - 2, q - 1, q, rng.randint(0, q), rng.randint(0, q), rng.randint(0, q)}:
            cases |= {(q * q + r * r + e, q) for e in (-1, 0, 1)}
    for S0 in [LIM - 1, LIM - 2, LIM - 4096] + [s * s + e for s in roots_near(math.isqrt(LIM - 1)) for e in (-1, 0, 1)]:
        least, top = math.isqrt((S0 + 1) // 2), math.isqrt(max(S0, 0))
        cases |= {(S0, least + k) for k in range(-1, 4)} | {(S0, top + k) for k in range(-2, 4)}
    cases = sorted((S0, q) for S0, q in cases if 1 <= S0 < LIM and q >= 1 and 2 * q * q >= S0 and q * q < S0 + (1 << 21))
    got = fast_roots(1, cases)
    assert len(cases) > 40000
    for (S0, q), g in zip(cases, got):
        m = S0 - q * q
        p = max(1, math.isqrt(m - 1) + 1) if m > 0 else 1
        assert (g & 0xFFFFFFFF, g >> 32) == (p, (p * p + q * q - S0) & 0xFFFFFFFF), (S0, q)


def test_pair_numbers():
    """The first, second and last pair of every y below 8192."""
    pairs = [(y * (y - 1) // 2 + x, 0) for y in range(1, 8192) for x in {0, 1, y - 1} if x < y]
    got = fast_roots(2, pairs)
    want = [y << 32 | x for y in range(1, 8192) for x in {0, 1, y - 1} if x < y]
    assert got == want


def test_fast_root_arguments():
    lib = _abi.load()
    one = (C.c_uint64 * 1)(1)
    assert lib.ps4_check_fast_roots(0, 3, one, one, 1, one) == _abi.PS4_ERR_ARG
    assert lib.ps4_check_fast_roots(0, 0, one, None, 1, one) == _abi.PS4_ERR_ARG
    assert lib.ps4_check_fast_roots(0, 0, None, None, 0, None) == _abi.PS4_OK
