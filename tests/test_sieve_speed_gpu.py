"""The automatic choice between search and lattices is never the slower one by more than their launches."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P,d,sl,limit,m_inc", [
    (337, 2310, 2_000, 20_000_000, 4_000),      # a narrow strip: few primes left to the lattices
    (337, 2310, 2_000, 20_000_000, 10_000),
    (337, 2310, 600, 30_000_000, 40_000),
    (337, 2310, 600, 30_000_000, 4_000),        # all of them
    (337, 2310, 7_500, 100_000_000, 10_000),
    (337, 2310, 7_500, 100_000_000, 20_000),
    (337, 2310, 2_000, 300_000_000, 150_000),
    (503, 2190, 10_000, 300_000_000, 3_000),
    (503, 2190, 10_000, 1_000_000_000, 50_000),
    (907, 210, 18_000, 100_000_000, 3_000),
    (907, 210, 60_000, 300_000_000, 3_000),
])
def test_lattices_do_not_slow_the_sieve(pg, P, d, sl, limit, m_inc):
    """Sieve kernels' time, best of ten, against a job that forces the search: a tenth for the clocks, 10 us."""
    args = dict(p=P, d=d, sl=sl, max_prime=limit, max_m_inc=m_inc, max_m=12_000_000)
    with pg.Job(**args) as auto, pg.Job(**args, flags=pg.PG_JOB_LARGE_SEARCH) as forced:
        best = {}
        for name, job in (("auto", auto), ("search", forced)):
            runs = [job.search(10_000_000, m_inc) for _ in range(10)]
            best[name] = min(r.stats["sieve_ms"] for r in runs)
            assert all(r.stats["survivors"] == runs[0].stats["survivors"] for r in runs)
            best[name + " left"] = runs[0].stats["survivors"]
        assert best["auto left"] == best["search left"]
        assert best["auto"] <= 1.1 * best["search"] + 0.01


@pytest.mark.parametrize("P,d,sl,limit,m_inc", [(337, 2310, 600, 30_000_000, 4_000), (337, 2310, 40, 30_000_000, 60_000),
                                                (211, 30, 200, 60_000_000, 30_000), (211, 2, 2, 8_000_000, 4_000)])
def test_rows_of_narrow_strips(pg, P, d, sl, limit, m_inc):
    """Strips far narrower than the lattices' width and windows longer than their steps, row by row."""
    args = dict(p=P, d=d, sl=sl, max_prime=limit, max_m_inc=m_inc, max_m=12_000_000, small_limit=1_000)
    with pg.Job(**args) as auto, pg.Job(**args, flags=pg.PG_JOB_LARGE_SEARCH) as forced:
        for inc in (m_inc, m_inc // 7, 40):
            assert np.array_equal(auto.sieve_interval(10_000_000, inc)[1], forced.sieve_interval(10_000_000, inc)[1])
