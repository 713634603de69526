"""Sieve rows of windows whose large primes are enumerated by their lattices, against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P,d,sl,limit,m_start,m_inc,small", [
    (337, 2310, 600, 3_000_000, 10_000_000, 400, 0),          # width below LAT_W, few m
    (337, 2310, 600, 3_000_000, 10_000_019, 1, 0),            # one m
    (211, 30, 8_191, 2_000_000, 1, 30, 1_000),                # width next to LAT_W, small primes stepped, m from 1
    (211, 30, 16_384, 5_000_000, 7, 60, 16_384),
    (503, 2190, 65_000, 20_000_000, 1_000_001, 60, 0),        # width eight times LAT_W
    (211, 2, 131_070, 8_000_000, 999_999, 12, 0),             # the widest rows
    (503, 2190, 3_000, 60_000_000, (1 << 30) - 900, 800, 0),  # m up to the rule's limit
    (503, 2190, 3_000, 60_000_000, (1 << 30) - 100, 800, 0),  # and across it
    (907, 210, 2_000, 4_400_000_000, 1_000_000, 40, 0),       # primes on both sides of 2^32
])
def test_rows_equal_the_oracle(pg, oracle, P, d, sl, limit, m_start, m_inc, small):
    with pg.Job(P, d, sl, limit, max_m_inc=max(m_inc, 2), max_m=m_start + m_inc, small_limit=small) as job:
        ms, rows = job.sieve_interval(m_start, m_inc)
    if not len(ms):
        pytest.skip("no m coprime to d")
    sel = np.arange(0, len(ms), 1 + len(ms) // 24)
    with oracle.Job(P, d, sl, limit) as oj:
        want = oj.sieve_m(ms[sel])
    assert np.array_equal(rows[sel], want)


def test_rows_do_not_depend_on_the_window(pg):
    """A window's rows equal those of its parts: primes change between search and lattice with its length."""
    with pg.Job(503, 2190, 10_000, 200_000_000, max_m_inc=60_000, max_m=1_100_000) as job:
        ms, rows = job.sieve_interval(1_000_000, 60_000)
        for inc in (20_000, 3_000, 100):
            part_ms, part = job.sieve_interval(1_000_000, inc)
            assert np.array_equal(part_ms, ms[:len(part_ms)]) and np.array_equal(part, rows[:len(part)])
