"""
The numbering of the precision form's ATM tasks: a task of any structure size
names a range of inner atoms, a tile of middle atoms and a chunk of outer atoms
that exist, and all of them are reached once.
"""

from __future__ import annotations

import ctypes
from functools import partial

import pytest

from conftest import package


@pytest.fixture(scope="module")
def task():
    fn = package()._lib.load().d4_selftest_atm_task

    def decode(n, s, t):
        out = (ctypes.c_int32 * 3)(-1, -1, -1)
        total = fn(n, s, t, out)
        return total, tuple(out)

    return decode


@pytest.mark.parametrize("n", [3, 10, 11, 18, 67, 131, 200])
@pytest.mark.parametrize("s", [1, 2, 4, 16])
def test_every_task_once(task, n, s):
    tiles = (n - 2 + 7) // 8
    total, _ = task(n, s, 0)
    got = [task(n, s, t)[1] for t in range(total)]
    # tile u from the top has u + 1 chunks and, g = tiles - 1 - u from below, g // s + 1 ranges
    want = {(ip, u, ch) for u in range(tiles) for ch in range(u + 1)
            for ip in range((tiles - 1 - u) // s + 1)}
    assert len(got) == len(want) and set(got) == want


@pytest.mark.parametrize("n", [47300, 60000, 90000])
def test_numbers_beyond_32_bits(task, n):
    s, tiles = 16, (n - 2 + 7) // 8
    decode = partial(task, n, s)
    total, first = decode(0)
    assert total > 2 ** 31 and first == (0, 0, 0)
    start, m, ip = 0, tiles, 0
    while m > 0:  # the first and the last task of every range of inner atoms
        count = m * (m + 1) // 2
        assert decode(start)[1] == (ip, 0, 0)
        assert decode(start + count - 1)[1] == (ip, m - 1, m - 1)
        start, m, ip = start + count, m - s, ip + 1
    assert start == total
