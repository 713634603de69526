"""The search on tensor-core reductions: its error bounds in exact arithmetic (CPU), and its gaps against the
one-warp kernel's (which a draining submit still runs) at every operand size it is compiled for."""
from __future__ import annotations

import math
import random
from fractions import Fraction

import numpy as np
import pytest

SIZES = (12, 14, 15, 16, 18, 20, 22, 23, 24, 26, 28, 30, 32, 34, 36, 38, 40, 42, 44)


def _primorial(P: int) -> int:
    k = 1
    for q in range(2, P + 1):
        if all(q % r for r in range(2, int(q ** 0.5) + 1)):
            k *= q
    return k


def _size(k_log2: float, max_m: int) -> int:
    n = k_log2 + math.log2(max_m + 1)
    return next((L for L in SIZES if 32 * L >= n + 1.17), 0)


def _step(L, K, mu, mu_off, m, X, y, b):
    """One step as the kernel computes it (words, dropped columns and doubles included)."""
    h, mask = 32 * (L - 4), (1 << 32 * L) - 1
    T = y * y
    th, mub = (T >> h).to_bytes(4 * (L + 4), "little"), mu.to_bytes(4 * 48, "little")
    ncol = 4 + 4 * (L + 1)
    a, f = np.frombuffer(th, np.uint8).astype(np.int64), np.frombuffer(mub, np.uint8).astype(np.int64)
    prod = np.convolve(a, f)
    cols = [int(prod[mu_off + c]) if 0 <= mu_off + c < len(prod) else 0 for c in range(ncol)]
    assert max(cols) < 1 << 23
    q = sum(c << (8 * i) for i, c in enumerate(cols)) & ((1 << 32 * (L + 2)) - 1)
    frac, z = q & 0xffffffff, q >> 32
    words = [(z >> (32 * (L - 4 + k))) & 0xffffffff for k in range(5)]
    top = 0.0
    for w in reversed(words):
        top = top * 4294967296.0 + float(w)
    n = m * K + X
    nd = float(Fraction(n, 1 << 32 * (L - 4)))
    t = math.floor((-float(X) / nd) * top + (frac * 2.0 ** -32 - 1 / 16))
    z += t
    r = m * T - z * n
    assert 0 <= r * 100 <= 111 * n, r / n
    low = (m * ((T - (z % (1 << 32 * (L + 1))) * K) & mask) - X * z) & mask
    assert low == r
    return r << b


@pytest.mark.parametrize("L", SIZES)
def test_step_bounds_at_the_extremes(L):
    """r = m*T - z*n stays in [0, 1.11 n) for the smallest and largest K and m, and |X| up to the rule's limit."""
    rng = random.Random(L)
    for _ in range(40):
        X_log2 = rng.choice([2, 10, 14, 17, 22])
        m = rng.choice([1, 3, rng.randrange(1, 1 << 12), rng.randrange(1 << 20, 1 << 22), (1 << 30) - 1])
        if math.log2(m) + X_log2 > 44:
            m = 1 << 21
        top = 32 * L - 1.17 - math.log2(m + 1)          # largest log2 K
        low = 32 * (L - 4) + X_log2 + 9                 # smallest bits of K
        if low + 1 > top or 2 * math.log2(m) + top + 2.4 > 32 * (L + 1):
            continue
        kb = rng.choice([int(top), math.ceil(low), rng.randint(math.ceil(low), int(top))])
        K = rng.getrandbits(kb) | (1 << (kb - 1)) | 1
        X = 2 * rng.randrange(1, 1 << (X_log2 - 1)) * rng.choice([-1, 1])
        n = m * K + X
        t_log2 = 2 * (math.log2(K >> max(0, kb - 60)) + max(0, kb - 60) + math.log2(m + 1)) + 2.31
        h = 32 * (L - 4)
        cols = math.ceil((t_log2 + 8 - h) / 8)
        mu = (1 << (h + 8 * cols)) // K
        assert mu.bit_length() <= 32 * 48
        y = rng.choice([0, 1, n - 1, n // 3, 222 * n // 100, rng.randrange(2 * n)])
        for _ in range(6):
            y = _step(L, K, mu, cols - 4, m, X, y, rng.randrange(2))


CASES = [(P, d, m) for P, d, m in
         [(257, 210, 1_000_001), (281, 2310, 1_000_001), (307, 210, 5), (331, 2310, 1_000_001), (337, 2310, 10_000_001),
          (367, 210, 1_000_001), (401, 2190, 1_000_001), (433, 210, 1), (457, 210, 1_000_001), (491, 2310, 1_000_001),
          (503, 2190, 1_000_001), (503, 2190, (1 << 30) - 700), (523, 210, 999_999_001), (571, 210, 1_000_001),
          (601, 210, 1_000_001), (641, 210, 900_000_001), (677, 2310, 1_000_001), (719, 210, 1_000_001),
          (757, 2310, 1_000_001), (797, 210, 1_000_001), (839, 210, 1_000_001), (881, 210, 1_000_001),
          (907, 210, 1_000_001), (907, 210, 999_999_001), (947, 210, 1_000_001), (1009, 2310, 3)]]


def test_cases_cover_the_sizes():
    assert {_size(math.log2(_primorial(P) // d), m + 400) for P, d, m in CASES} >= set(SIZES)


@pytest.mark.gpu
@pytest.mark.parametrize("P,d,m_start", CASES)
def test_gaps_equal_the_one_warp_kernel(pg, P, d, m_start):
    with pg.Job(P, d, 3_000, 200_000, max_m_inc=400, max_m=m_start + 400) as job:
        a = job.search(m_start, 400)
        b = job.wait(job.submit(m_start, 400, flags=pg.PG_SUBMIT_DRAIN))
    assert len(a.ms) and np.array_equal(a.prev_gap, b.prev_gap) and np.array_equal(a.next_gap, b.next_gap)
    assert (a.next_gap > 0).all() and a.stats["prp_tests"] > 2 * len(a.ms)


@pytest.mark.gpu
@pytest.mark.parametrize("m_inc,cap", [(3, 0), (40, 1), (3_000, 2), (30_000, 0), (30_000, 6), (30_000, 14)])
def test_grids(pg, m_inc, cap):
    """Fewer candidates than a CTA holds, one CTA an SM and every CTA that fits, and each cap's grid."""
    with pg.Job(337, 2310, 5_000, 10_000_000, max_m_inc=m_inc, max_m=10_100_000) as job:
        a = job.wait(job.submit(10_000_001, m_inc, flags=pg.PG_SUBMIT_WARPS_PER_SM(cap)))
        b = job.wait(job.submit(10_000_001, m_inc, flags=pg.PG_SUBMIT_DRAIN))
    assert np.array_equal(a.prev_gap, b.prev_gap) and np.array_equal(a.next_gap, b.next_gap)


@pytest.mark.gpu
def test_short_sieve_and_extension(pg):
    """sl far below the gaps: candidates past sl, where factors shared by m and X appear, and continuations."""
    with pg.Job(503, 2190, 60, 10_000, max_m_inc=20_000, max_m=1_020_000, ext_window=3_000) as job:
        a = job.search(1_000_000, 20_000)
        b = job.wait(job.submit(1_000_000, 20_000, flags=pg.PG_SUBMIT_DRAIN))
    assert np.array_equal(a.prev_gap, b.prev_gap) and np.array_equal(a.next_gap, b.next_gap)


@pytest.mark.gpu
@pytest.mark.parametrize("m_inc", [2, 40, 400])
def test_lane_groups_few_sides(pg, m_inc):
    """Lane-group searches on grids of one warp per SM quarter and more, against every block with draining."""
    with pg.Job(337, 2310, 5_000, 10_000_000, max_m_inc=m_inc, max_m=10_100_000, tpi=8) as job:
        a = job.search(10_000_001, m_inc)
        b = job.wait(job.submit(10_000_001, m_inc, flags=pg.PG_SUBMIT_DRAIN))
    assert np.array_equal(a.prev_gap, b.prev_gap) and np.array_equal(a.next_gap, b.next_gap)


@pytest.mark.parametrize("P,d", [(257, 210), (337, 2310), (389, 210), (503, 2190), (811, 210)])
def test_start_from_the_leading_bits(P, d):
    """x * m^-1 for x = 2^e, e the exponent's leading bits, in exact arithmetic: the quotient words by the rounded
    reciprocal, the value and its bound, for candidates shorter than the CTA's longest too."""
    K, rng = _primorial(P) // d, random.Random(P)
    for m in [1, 2, 3, (1 << 30) - 1] + [rng.randrange(1, 1 << rng.randrange(2, 31)) for _ in range(60)]:
        X = 2 * rng.randrange(1, 1 << rng.randrange(1, 23)) * rng.choice([-1, 1])
        n = m * K + X
        if n % 2 == 0 or math.gcd(m, abs(X)) > 1:
            continue
        bmax = max(n.bit_length(), rng.choice([0, (((1 << 30) - 1) * K).bit_length()]))
        lead = (bmax - 32).bit_length() - 1
        e = n >> (bmax - lead)
        assert e == (n - 1) >> (bmax - lead) and 2 ** e < K
        inv, rem, q = ((1 << 64) - 1) // m, 0, 0
        for i in range(e >> 5, -1, -1):
            v = rem << 32 | ((1 << (e & 31)) if i == e >> 5 else 0)
            t = v * inv >> 64
            assert 0 <= v // m - t <= 2 and v // m < 1 << 32
            q, rem = q << 32 | v // m, v % m
        s = -pow(X, -1, m) * rem % m if m > 1 else 0
        assert (s * X + rem) % m == 0
        y = s * K + (s * X + rem) // m + q
        assert 0 <= 100 * y < 222 * n and (m * y - (1 << e)) % n == 0
