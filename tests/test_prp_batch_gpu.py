"""Small PRP batches: bases side by side and lanes per number, at the sizes where pick_batch changes layout."""
from __future__ import annotations

import random

import pytest

pytestmark = pytest.mark.gpu

PSEUDO = [2047, 3277, 4033, 4681, 8321, 15841, 29341, 3215031751, 3474749660383, 341550071728321]


def _mix(rng, bits, n):
    """Primes, odd composites, pseudoprimes to the first bases, tiny, even and zero values, shuffled."""
    import sympy
    if bits < 800:
        p = int(sympy.nextprime(rng.getrandbits(bits - 1) | (1 << (bits - 2))))
    else:
        p = 2 ** max(e for e in (607, 1279, 2203, 4253) if e <= bits) - 1
    q = int(sympy.nextprime(rng.getrandbits(min(bits // 2, 400) - 1)))
    fixed = [p, q, q * q, p - 2, 0, 1, 2, 3, 5, 7, 9, 47, 53, 54, 55, 2 ** 61 - 1] + PSEUDO
    nums = [fixed[i % len(fixed)] if i % 3 == 0 else rng.getrandbits(bits) | 1 for i in range(n)]
    rng.shuffle(nums)
    nums[0] = (1 << bits) - 1 if n > 1 else p  # the batch's width
    return nums


@pytest.mark.parametrize("words,n,rounds", [
    (1, 3, 16), (6, 40, 2), (16, 20, 16), (17, 1, 16), (22, 12, 16), (23, 9, 5), (23, 256, 2), (23, 257, 2),
    (24, 7, 16), (24, 97, 2), (32, 128, 3), (32, 129, 3), (47, 30, 16), (48, 10, 16), (48, 257, 2), (22, 1024, 2),
    (22, 1025, 2), (60, 148, 2), (60, 149, 2), (136, 6, 2), (22, 4096, 1), (22, 4097, 1), (28, 1793, 1),
    (65, 3072, 1), (65, 3073, 1), (80, 5, 16), (95, 148, 2), (95, 149, 2), (96, 2368, 1), (96, 2369, 1), (100, 6, 16),
    (135, 3, 16)])
def test_matches_the_oracle(ctx, oracle, words, n, rounds):
    rng = random.Random(words * 1000 + n)
    nums = _mix(rng, 32 * words, n)
    got = ctx.prp(nums, rounds=rounds)
    cut = range(n) if n <= 300 else sorted(rng.sample(range(n), 300))
    assert [int(got[i]) for i in cut] == [oracle.prp(nums[i], rounds) for i in cut]


@pytest.mark.parametrize("words", [64, 96])
def test_bases_at_the_width_of_the_lanes(ctx, oracle, words):
    """Operands with 7, 8 and 9 bits to spare in their lanes, and none: folded and multiplied bases side by side."""
    bits = 32 * words
    nums = []
    for spare in (0, 7, 8, 9):
        top = 1 << (bits - spare)
        nums += [top - 1, (top >> 1) + 1, top - 2 ** (bits // 3) + 1]
    for e in (1279, 2203):
        if e <= bits:
            nums += [2 ** e - 1, (2 ** e - 1) * ((1 << (bits - e - 8)) | 1)]
    got = ctx.prp(nums, rounds=16)
    assert [int(g) for g in got] == [oracle.prp(x, 16) for x in nums]
