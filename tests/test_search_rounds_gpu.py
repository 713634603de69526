"""Lane-group searches of few sides: the blocks that the rounds rule launches against every block that fits."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ms(pg, job, m_inc, flags):
    """Device time of the window's kernels, best of five."""
    runs = [job.wait(job.submit(1_000_001, m_inc, flags=flags)) for _ in range(5)]
    return min(r.stats["total_ms"] for r in runs), runs[0]


@pytest.mark.parametrize("P,d,tpi,m_inc", [(337, 2310, 16, 1_000), (337, 2310, 8, 1_400), (503, 2190, 8, 1_000),
                                           (503, 2190, 16, 600), (503, 2190, 4, 2_000), (907, 210, 8, 600),
                                           (1511, 210, 0, 300)])
def test_the_rule_is_not_slower_than_every_block(pg, P, d, tpi, m_inc):
    """A tenth for the rounds that fall one way or the other; the gaps are equal."""
    with pg.Job(P, d, 6_000 if P < 1_000 else 20_000, 10_000_000, max_m_inc=m_inc, max_m=2_000_000, tpi=tpi) as job:
        rule, a = _ms(pg, job, m_inc, 0)
        every, b = _ms(pg, job, m_inc, pg.PG_SUBMIT_WARPS_PER_SM(255))
    assert np.array_equal(a.prev_gap, b.prev_gap) and np.array_equal(a.next_gap, b.next_gap)
    assert rule <= 1.1 * every
