"""A flag that forces one large-prime method keeps the others out."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ARGS = dict(p=337, d=2310, sl=3_000, max_prime=100_000_000, max_m_inc=4_000, max_m=11_000_000)


def test_large_search_flag_forces_the_search(pg):
    """The window's large primes lie on both sides of one expected hit: a search and a lattice launch, or the search
    alone under the flag."""
    with pg.Job(**ARGS) as auto, pg.Job(**ARGS, flags=pg.PG_JOB_LARGE_SEARCH) as forced:
        a, b = auto.search(10_000_000, 4_000), forced.search(10_000_000, 4_000)
        assert np.array_equal(a.prev_gap, b.prev_gap) and np.array_equal(a.next_gap, b.next_gap)
        assert a.stats["survivors"] == b.stats["survivors"]
        assert np.array_equal(auto.sieve_interval(10_000_000, 300)[1], forced.sieve_interval(10_000_000, 300)[1])
        assert a.stats["kernel_launches"] - a.stats["relaunches"] * 2 == \
            b.stats["kernel_launches"] - b.stats["relaunches"] * 2 + 1


@pytest.mark.parametrize("flag", ["PG_JOB_LARGE_SEARCH", "PG_JOB_LARGE_STEP"])
def test_forced_methods_keep_no_lattices(pg, flag):
    with pg.Job(**ARGS, flags=getattr(pg, flag)) as forced:
        forced_bytes, primes = forced.info["device_bytes"], forced.info["num_primes"]
    assert primes > 1_000_000
    # 12 B of tables, at most 8 B of walk steps, the buffers of 4 000 m
    with pg.Job(**ARGS) as auto:
        buffers = auto.info["device_bytes"] - 28 * primes
    assert forced_bytes < buffers + 21 * primes
