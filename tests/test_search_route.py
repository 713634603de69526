"""Which search kernel runs: the tensor-core one wherever its sizes allow, as the job and the search report it."""
from __future__ import annotations

import math

import pytest

from test_tc_search import CASES, _primorial, _size

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P,d,m_start", CASES)
def test_the_tensor_core_search_runs_at_its_sizes(pg, P, d, m_start):
    with pg.Job(P, d, 3_000, 200_000, max_m_inc=60, max_m=m_start + 400) as job:
        assert job.info["tc_words"] == _size(math.log2(_primorial(P) // d), m_start + 400)
        assert job.search(m_start, 60).stats["tc_blocks"] > 0
        assert job.wait(job.submit(m_start, 60, flags=pg.PG_SUBMIT_DRAIN)).stats["tc_blocks"] == 0
        assert job.search(m_start, 60, pg.PG_SEARCH_PLAIN).stats["tc_blocks"] == 0


@pytest.mark.parametrize("P,d,max_m,tpi", [(503, 2190, 1 << 30, 0), (503, 2190, 2_000_000, 8), (211, 30, 2_000_000, 0),
                                           (1091, 210, 2_000_000, 0), (1511, 210, 2_000_000, 0)])
def test_refused_sizes_report_another_kernel(pg, P, d, max_m, tpi):
    with pg.Job(P, d, 3_000, 200_000, max_m_inc=60, max_m=max_m, tpi=tpi) as job:
        assert job.info["tc_words"] == 0
        assert job.search(1_000_001, 60).stats["tc_blocks"] == 0


@pytest.mark.parametrize("P,d", [(337, 2310), (503, 2190), (571, 210), (907, 210)])
def test_warp_caps_in_whole_blocks(pg, P, d):
    """A cap is rounded up to blocks of 4 warps, and one below what fits leaves a block's room."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    with pg.Job(P, d, 3_000, 200_000, max_m_inc=60, max_m=2_000_000) as job:
        def blocks(w):
            n, rest = divmod(job.wait(job.submit(1_000_001, 60, flags=pg.PG_SUBMIT_WARPS_PER_SM(w))).stats["tc_blocks"], sms)
            assert rest == 0
            return n
        most = blocks(255)
        assert 1 < most <= 4
        for w in range(1, 4 * most + 3):
            assert blocks(w) == (most if w >= 4 * most else min(-(-w // 4), most - 1))
