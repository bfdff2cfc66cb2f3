"""Single steps of the search kernels, called directly on inputs that whole searches seldom or
never meet.

Bar: bit-exact against exact integer arithmetic on the host.
"""
from __future__ import annotations

import ctypes as C
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
