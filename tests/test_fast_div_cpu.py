"""Divisions by launch constants (the order of CTAs, the KV head, the part, the page, the row of a merge) are multiplications: every
quotient of 32-bit numbers must come out, also of the CTA numbers from 2^31 on that a grid of that many heads and rows has."""
import random

import pytest

from flash_attention_b200._lib import lib

TOP = 1 << 32


@pytest.mark.parametrize("lo,hi", [(1, 700), (2**16 - 40, 2**16 + 40), (2**31 - 40, 2**31 + 40), (TOP - 40, TOP)])
def test_every_quotient(lo, hi):
    rng, div = random.Random(lo), lib().fa_selftest_fast_div
    for d in range(lo, hi):
        near = [m * d + o for m in {0, 1, 2, 3, (2**31) // d, (TOP - 1) // d, rng.randrange(TOP // d + 1)} for o in (-1, 0, 1)]
        for n in near + [2**31 - 1, 2**31, TOP - 1, rng.randrange(TOP)]:
            if 0 <= n < TOP:
                assert div(n, d) == n // d, (n, d)


def test_random_pairs():
    rng, div = random.Random(5), lib().fa_selftest_fast_div
    for _ in range(30000):
        n, d = rng.getrandbits(rng.randrange(1, 33)), max(1, rng.getrandbits(rng.randrange(1, 33)))
        assert div(n, d) == n // d, (n, d)
